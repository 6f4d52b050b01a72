"""Host paths that a healthy GPU does not reach -- memory that runs out, a launch
that fails -- and the launches and copies that a call issues, on the CPU: the
library over the runtime of fake_cudart.cpp, in a process of its own."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")

PRELUDE = """
import ctypes, os, sys
import numpy as np
import pytnl_lbm as pl
lib = pl.library()
fake = ctypes.CDLL(os.environ["FAKE_CUDART"])
fake.fake_count.restype = ctypes.c_longlong
fake.fake_trace.restype = ctypes.c_char_p
fake.fake_in_use.restype = ctypes.c_size_t
fake.fake_last_copy_to.restype = ctypes.c_void_p
fake.fake_limit.argtypes = [ctypes.c_size_t]
fake.fake_fail_launch.argtypes = fake.fake_fail_new.argtypes = [ctypes.c_longlong]
fake.fake_pinned.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
def count(what): return fake.fake_count(what.encode())
def refused(f, *a, **k):
    try: f(*a, **k)
    except pl.LbmError as e: return e.code
    return 0
"""


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    (d / "versions").write_text("libcudart.so.12 { global: cuda*; __cuda*; fake_*; };\n")
    so = str(d / "libcudart.so.12")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CUDA, "-Wl,-soname,libcudart.so.12",
                    "-Wl,--version-script=" + str(d / "versions"), os.path.join(ROOT, "tests", "fake_cudart.cpp"),
                    "-o", so], check=True)
    env = dict(os.environ, LD_PRELOAD=so, FAKE_CUDART=so, PYTHONPATH=os.path.join(ROOT, "tnl-lbm_b200"))

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], capture_output=True, text=True, env=env, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_step_over_the_fake_runtime(child):
    """A step launches its kernel once, 16 steps go through a graph."""
    child("""
lat = pl.LBM(16, 8, 8, viscosity=0.01, periodic=True)
fake.fake_reset()
lat.step(3)
assert count("launches") == 3, fake.fake_trace()
lat.step(33)
assert (count("nodes"), count("graph launches")) == (16, 2)
assert lat.iteration == 36
""")


@pytest.mark.parametrize("room", ["checkpoints", "moments", "earlier moments", "all"])
def test_adjoint_forward_falls_back_to_checkpoints(child, room):
    """A forward pass runs wherever the checkpoints of all its steps and the
    final state fit: without room for the kept moments (an earlier run holds the
    checkpoints), with room for them but not for the checkpoints beside them, or
    with the moments of an earlier run in the way of a run that keeps none."""
    child("room = %r" % room + """
N, K, X, Y, Z = 400, 20, 512, 8, 8
lat = pl.LBM(X, Y, Z, viscosity=0.02, collision=pl.COLL_SRT, equilibrium=pl.EQ_SECOND_ORDER, periodic=True)
v = lat.device_view()
pop = v.sz * (Z + 2) * v.elem_size
enough = fake.fake_in_use() + 24 * X * Y * Z + 48 + (N // K + 1) * pop
def forward(n, every):
    fake.fake_reset()
    lat.adjoint_forward(np.zeros((3, Z, Y, X)), n, np.array([5]), np.zeros((1, 4)), checkpoint_every=every)
if room == "checkpoints":
    forward(N // K, 1)
if room == "earlier moments":
    forward(N, K)
fake.fake_limit(0 if room == "all" else enough)
n, every = (N // K, 1) if room == "earlier moments" else (N, K)
forward(n, every)
used = fake.fake_in_use()
assert (used > enough) == (room == "all")  # the moments do not fit beside the checkpoints
fake.fake_limit(0)
lat.adjoint_backward()
steps, recomputed = fake.fake_trace().count(b"adj_step_kernel"), fake.fake_trace().count(b"adj_primal_kernel") - n
assert steps == n and (recomputed < n if room == "all" else recomputed == n), (steps, recomputed)
lat.close()
""")


@pytest.mark.parametrize("shape", [(128, 0), (128, 1), (256, 3)])
def test_ensemble_blocks_of_steps(child, shape):
    """Several groups of members: a block of steps takes them one after the other,
    a single step (also the odd one ahead of a block) all in one launch."""
    child("shape = %r" % (shape,) + """
ens = pl.Ensemble([(64, 32, 32)] * 30, [0.01] * 30, cum_flags=3)  # 212 MB
ens.set_shape(*shape)
for n, launches in ((1, 1), (1, 1), (3, 12), (1, 1)):
    fake.fake_reset()
    ens.step(n)
    assert count("launches") == launches, (n, fake.fake_trace())
fake.fake_reset()
ens.step(1, sums=True)
assert count("launches") == 2, fake.fake_trace()  # the step and the finish of the sums
assert ens.iteration == 7
""")


def test_ensemble_graphs_are_bounded(child):
    """A graph of 16 steps has a node per step and group: ensembles of up to 64
    groups replay it, larger ones launch their (long) steps one by one."""
    child("""
for members, nodes, graph_launches, launches in ((30, 16 * 4, 2, 0), (620, 0, 0, 32 * 69)):
    ens = pl.Ensemble([(64, 32, 32)] * members, [0.01] * members, cum_flags=3)  # 7.1 MB each
    fake.fake_reset()
    ens.step(32)
    assert (count("nodes"), count("graph launches"), count("launches")) == (nodes, graph_launches, launches), \\
        (count("nodes"), count("graph launches"), count("launches"))
    assert ens.iteration == 32
    ens.close()
""")


@pytest.mark.parametrize("kind", ["lattice", "ensemble"])
def test_failed_launch_is_reported_once(child, kind):
    """The error of a step launch is that call's; the next call does not find it
    in the runtime and report it as its own."""
    child("kind = %r" % kind + """
if kind == "lattice":
    sim = pl.LBM(16, 8, 8, viscosity=0.01, periodic=True)
    read = sim.get_populations
else:
    sim = pl.Ensemble([(16, 8, 8)] * 2, [0.01] * 2)
    read = lambda: sim.get_populations(1)
fake.fake_fail_launch(1)
assert refused(sim.step, 1) == 3 and sim.iteration == 0
read()
sim.step(1)
assert sim.iteration == 1
""")


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("shape", [(128, 0), (256, 3)])
def test_failed_launch_leaves_no_members_apart(child, shape, graphs):
    """A block of steps whose launch fails part way has some groups ahead of the
    others: the ensemble refuses steps and read-out until it is initialised.  A
    launch that fails before any went out (or under capture) changes nothing."""
    child("shape, graphs = %r, %r" % (shape, graphs) + """
ens = pl.Ensemble([(64, 32, 32)] * 30, [0.01] * 30, cum_flags=3, use_graphs=graphs)  # 4 groups
ens.set_shape(*shape)
ens.init_taylor_green(0.05)
ens.step(2)
for n in (1, 3):
    fake.fake_fail_launch(1)
    assert refused(ens.step, n) == 3 and ens.iteration == 2
if graphs:
    fake.fake_fail_launch(9)
    assert refused(ens.step, 16) == 3 and ens.iteration == 2
    ens.step(16)
else:
    ens.step(16)
ens.get_populations(0)
fake.fake_fail_launch(6)
assert refused(ens.step, 3) == 3
for call in (lambda: ens.step(1), lambda: ens.step(3), ens.autotune, lambda: ens.get_populations(0)):
    assert refused(call) == 1
    assert "part way" in lib.lbm_last_error().decode()
ens.init_taylor_green(0.05)
ens.step(3)
ens.get_populations(29)
assert ens.iteration == 3
""")


FIELD = """
def field(storage, X, Y, Z):
    # a lattice whose macro field in device memory holds numbers of its own
    lat = pl.LBM(X, Y, Z, viscosity=0.01, periodic=True, storage=getattr(pl, "STORE_" + storage))
    lat.step(1, macro=True)
    n, t = 4 * X * Y * Z, np.float64 if storage == "F64" else np.float32
    a = np.random.default_rng(1).standard_normal(n).astype(t)
    ctypes.memmove(lat.device_view().macro, a.ctypes.data, a.nbytes)
    fake.fake_reset()
    return lat, a.astype(np.float64)
def read(lat, out):
    assert lib.lbm_get_macro(lat.h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
"""


@pytest.mark.parametrize("storage", ["F64", "F32"])
def test_field_copies_of_a_new_lattice(child, storage):
    """The first read-outs of a lattice pay for no staging: values that go as they
    are take one copy below 32 MB, values to be widened are copied into the
    caller's memory and widened there, until 16 MB have gone that way."""
    child(FIELD + "storage = %r" % storage + """
lat, want = field(storage, 33, 32, 31)  # 1 MB
for k in range(20):
    out = np.zeros_like(want)
    fake.fake_reset()
    read(lat, out)
    np.testing.assert_array_equal(out, want)
    if storage == "F32" and (k + 1) * out.nbytes >= 16 << 20:
        assert count("pinned") == 1 and count("host copies") > 1
        break
    assert (count("host copies"), count("pinned")) == (1, 0), k
assert k == 19 if storage == "F64" else k == (16 << 20) // out.nbytes
""")


@pytest.mark.parametrize("storage,shape,staged", [("F32", (33, 32, 31), 0), ("F32", (64, 64, 32), 1), ("F64", (64, 64, 32), 0)])
def test_field_copies_ahead_of_work(child, storage, shape, staged):
    """While the stream is at work, staging is made for 4 MB to be widened."""
    child(FIELD + "storage, shape, staged = %r, %r, %r" % (storage, shape, staged) + """
lat, want = field(storage, *shape)
fake.fake_busy(1)
out = np.zeros_like(want)
read(lat, out)
np.testing.assert_array_equal(out, want)
assert count("pinned") == staged and (count("host copies") > 1) == bool(staged)
fake.fake_busy(0)
read(lat, out)
np.testing.assert_array_equal(out, want)
assert count("pinned") == staged
lat.get_populations()  # and the query has left no error behind
""")


@pytest.mark.parametrize("storage,pinned", [("F64", 0), ("F64", 1), ("F32", 0)])
def test_large_field_copies(child, storage, pinned):
    """From 32 MB on (16 MB widened) a field is staged, but for values that go as
    they are into memory that the device reaches: those take one copy."""
    child(FIELD + "storage, pinned = %r, %r" % (storage, pinned) + """
lat, want = field(storage, 128, 128, 65 if storage == "F64" else 33)
out = np.zeros_like(want)
if pinned:
    fake.fake_pinned(out.ctypes.data, out.nbytes)
read(lat, out)
np.testing.assert_array_equal(out, want)
assert count("pinned") == 1 - pinned and (count("host copies") == 1) == bool(pinned)
assert (fake.fake_last_copy_to() == out.ctypes.data) == bool(pinned)
""")


@pytest.mark.parametrize("storage,shape", [("F64", (128, 128, 65)), ("F32", (128, 128, 33)), ("F32", (3, 1, 1))])
def test_field_copy_without_pinned_memory(child, storage, shape):
    """No pinned memory to be had: one pageable copy."""
    child(FIELD + "storage, shape = %r, %r" % (storage, shape) + """
lat, want = field(storage, *shape)
fake.fake_no_pinned(1)
out = np.zeros_like(want)
read(lat, out)
np.testing.assert_array_equal(out, want)
assert count("host copies") == 1
""")


@pytest.mark.parametrize("which", [1, 2, 3])
def test_field_copy_without_memory_for_a_thread(child, which):
    """No memory for the state of a helper thread: the caller takes its share."""
    child(FIELD + "which = %r" % which + """
lat, want = field("F32", 128, 64, 64)  # 16 MB to the caller: staged, four threads
out = np.zeros_like(want)
fake.fake_fail_new(which)
read(lat, out)
np.testing.assert_array_equal(out, want)
assert count("thrown") == 1
""")


@pytest.mark.parametrize("steps,every", [(64, 8), (400, 20), (100, 50), (9, 1)])
def test_bench_counts_the_adjoint_steps_that_run(child, steps, every):
    """The bench's traffic of a gradient: every primal step that runs moves its
    populations and force, every step's moments are written once."""
    child("steps, every = %d, %d" % (steps, every) + """
sys.path.insert(0, %r)""" % ROOT + """
import bench
X, Y, Z = 512, 8, 8
lat = pl.LBM(X, Y, Z, viscosity=0.02, collision=pl.COLL_SRT, equilibrium=pl.EQ_SECOND_ORDER, periodic=True)
v = lat.device_view()
fake.fake_reset()
lat.adjoint_forward(np.zeros((3, Z, Y, X)), steps, np.array([5]), np.zeros((1, 4)), checkpoint_every=every)
lat.adjoint_backward()
primal = fake.fake_trace().count(b"adj_primal_kernel")
recomputed, site_bytes = bench.adjoint_traffic(steps, every, v.sz * (Z + 2) * v.elem_size, X * Y * Z)
assert recomputed == primal - steps
assert abs(site_bytes - (240 * primal / steps + 16 + 520)) < 1e-9, site_bytes
""")
