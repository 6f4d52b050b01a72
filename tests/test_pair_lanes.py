"""The two lanes of the two-site kernel's odd step on a periodic row of odd width,
on the CPU: the offsets that pair.cuh forms, compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tnl-lbm_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "pair.cuh"
using namespace lbm;
template <int CX>
int check(int X)
{
	int bad = 0;
	for (int x = 0; x < X; x += 2) {
		PairAt at = pair_at_of(nullptr, 4, 1024, 65536, 32, X, 4, 4, x, 1, 1, true, true);
		pair_ragged(at, x, X);
		int a, b;
		pair_lanes<CX>(at, a, b);
		bad += x + a != (x - CX + X) % X;  // the site the value streams from
		if (x + 1 < X)
			bad += x + b != (x + 1 - CX + X) % X;
		else  // the idle lane: the ghost site, which nobody writes, or what the first lane reads
			bad += x + b != X && b != a;
		if (bad)
			std::printf("X %d x %d CX %d: lanes read %d and %d\n", X, x, CX, x + a, x + b);
	}
	return bad;
}
int main(int, char** argv)
{
	const int X = std::atoi(argv[1]);
	return check<-1>(X) + check<0>(X) + check<1>(X) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-O0", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + CSRC,
                    str(d / "lanes.cu"), "-o", str(d / "lanes")], check=True)
    return str(d / "lanes")


@pytest.mark.parametrize("X", [1, 3, 5, 127, 255])
def test_lanes_of_an_odd_row(program, X):
    """Both lanes read the site that their direction streams from; the idle lane
    of the last pair reads nothing that another thread writes."""
    r = subprocess.run([program, str(X)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
