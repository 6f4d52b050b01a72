// Discrete adjoint of the A-A step with the SRT collision and a per-site body
// force (the control), for gradients of an objective on the final state.
//
// One A-A step is a map of the population memory M_n -> M_{n+1} that is
// block-diagonal over sites: site x reads 27 locations R_q(x) and writes 27
// locations W_q(x), and {R_q(x)} = {W_q(x)} as sets (streaming_AA.h:12-116);
// locations no site touches (ghost slots nobody writes, GEO_NOTHING sites)
// map to themselves.  The adjoint step therefore has the same access pattern:
// each thread gathers the adjoint of its 27 outputs from W_q(x), applies the
// transposed Jacobian of its per-site update at the primal state M_n, and
// scatters the result to R_q(x), in place and race-free.  No linearisation
// error: the result is the exact gradient of the discrete FP update, up to
// rounding.
//
// Per-site update (GEO type from the map, bc.h:85-412) and its transpose:
//   FLUID, PERIODIC  rho = sum f, u = (sum c f + F/2) / rho (common.h:17-50),
//                    out = f + (feq - f)/tau + (1 - 1/(2 tau)) S feq with
//                    S_q = 3 (c_q - u).F / rho (col_srt.h:14-105)
//   WALL             out_q = f_opp(q) (full-way bounce-back, bc.h:201-221)
//   INFLOW           out = feq(1, u_inlet): no dependence on f or F
//   OUTFLOW_EQ       out = feq(1, u(f)) (bc.h:186-190)
//   SYM_*            mirror copy of one half of the directions (bc.h:222-293)
// With rho and u held fixed, the SRT transpose is the reference's adjoint
// collision (col_srt_adjoint.h:50-109, eq_adjoint.h:13-27): at rho = 1 and
// F = 0 both give f*_j + (sum_q f*_q w_q (feq_rho + feq_v)(q; c_j) - f*_j)/tau.
// The equilibrium is the second-order one (D3Q27_EQ, eq.h).
#pragma once

#include "aa_kernels.cuh"

namespace lbm {

// Resident blocks per SM of the adjoint step (register cap 65536 / (128 n)).  It
// moves 520 bytes a site (27 FP64 values in and out, 4 moments, the force, the
// force gradient in and out) and is bound by the latency of its gathers: 64 steps
// of a 160x48x48 channel backward take 2598 us at 4 blocks, 2520 at 5, 2490 at 6
// (80 registers, 44 bytes of spills in the odd step), against 6595 when each step
// read the 27 primal populations, summed direction by direction and ran on rows
// of 128 threads.
#ifndef ADJ_STEP_MINB
#define ADJ_STEP_MINB 6
#endif
// and of the primal step with a force field: the 64 steps forward (FP32, moments
// kept) take 1700 us at 4 blocks, 1740 at 5 (92-112 bytes of spills), 1850 at 6
// (2330 with checkpoints instead of moments); FP64 spills 330 bytes at 4 and runs 3
#ifndef ADJ_PRIMAL_MINB
#define ADJ_PRIMAL_MINB 4
#endif
template <typename R, bool ODD>
constexpr int adj_primal_minb()
{
	return sizeof(R) == 8 ? 3 : ADJ_PRIMAL_MINB;
}

template <typename T, typename R>
struct AdjArgs
{
	T* f;			   // primal populations (the step's input, or the state to observe)
	double* lam;	   // adjoint populations, FP64 whatever the storage, same layout (element strides) as f
	// density and velocity [4][Z][Y][X] of one step's sites before the collision
	// (density_velocity): written by the primal step (or null), read by the
	// adjoint step
	R* mom;
	long long sq;
	int sy, sz, x0;
	int X, Y, Z;
	FastDiv dx, dy;	 // division by X and by Y
	unsigned n;		 // sites
	int slot[27];	 // byte offsets of lam's 27 slot rows of a lattice row
	const uint8_t* map;	 // null: every site periodic
	const R* in_vx;		 // inlet profiles [Z][Y] (GEO_INFLOW) or null
	const R* in_vy;
	const R* in_vz;
	const double* force;  // per-site body force [3][Z][Y][X] or null (uniform p.fx..fz)
	double* grad;	  // d objective / d force, [3][Z][Y][X], accumulated
	CollParams<R> p;
};

// Sites are taken in linear order, 128 to a block, whatever the width of a row
// is: with one row per block column a channel of X = 160 kept 62 % of the lanes
// busy.  false past the last site.
template <typename T, typename R>
__device__ __forceinline__ bool adj_position(const AdjArgs<T, R>& a, long long& site, int& x, int& y, int& z)
{
	const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
	const unsigned row = fast_div(i, a.dx);
	x = (int) (i - row * (unsigned) a.X);
	z = (int) fast_div(row, a.dy);
	y = (int) (row - (unsigned) z * (unsigned) a.Y);
	site = i;
	return i < a.n;
}

// location of the value that direction q of a site reads (R_q) in the A-A
// step of the given parity
template <bool ODD, int q>
__device__ __forceinline__ long long aa_read_loc(long long sq, long long base, const Offsets& o)
{
	if constexpr (ODD)
		return opp(q) * sq + base + o.x[1 - cx(q)] + o.y[1 - cy(q)] + o.z[1 - cz(q)];
	else
		return q * sq + base;
}
// Addresses of a site's adjoint values: row pointers of the three z planes
// around it, the y and x steps from there, and the slots' offsets as constant
// operands (AdjArgs::slot), so that neither the gather nor the scatter
// multiplies (as PairAt of pair.cuh)
struct AdjAt
{
	char* P[3];		  // the site in planes z - 1, z, z + 1
	long long oy[3];  // byte offsets of rows y - 1, y, y + 1
	int ox[3];		  // and of sites x - 1, x, x + 1
};

template <typename T, typename R>
__device__ __forceinline__ AdjAt adj_at(const AdjArgs<T, R>& a, bool wrap, int x, int y, int z)
{
	constexpr int E = (int) sizeof(double);
	const int zm = wrap && z == 0 ? a.Z - 1 : z - 1, zp = wrap && z == a.Z - 1 ? 0 : z + 1;
	char* const row = reinterpret_cast<char*>(a.lam) + ((long long) (y + 1) * a.sy + a.x0 + x) * E;
	const long long plane = (long long) a.sz * E;
	AdjAt at;
	at.P[0] = row + (zm + 1) * plane;
	at.P[1] = row + (z + 1) * plane;
	at.P[2] = row + (zp + 1) * plane;
	at.oy[0] = (long long) (wrap && y == 0 ? a.Y - 1 : -1) * a.sy * E;
	at.oy[1] = 0;
	at.oy[2] = (long long) (wrap && y == a.Y - 1 ? -(a.Y - 1) : 1) * a.sy * E;
	at.ox[0] = (wrap && x == 0 ? a.X - 1 : -1) * E;
	at.ox[1] = 0;
	at.ox[2] = (wrap && x == a.X - 1 ? -(a.X - 1) : 1) * E;
	return at;
}

// where direction q of the site is written (its adjoint gathered) and read
// (its adjoint scattered)
template <bool ODD, int q>
__device__ __forceinline__ double* adj_write_at(const AdjAt& at, const int (&slot)[27])
{
	if constexpr (ODD)
		return reinterpret_cast<double*>(at.P[1 + cz(q)] + at.oy[1 + cy(q)] + at.ox[1 + cx(q)] + slot[q]);
	else
		return reinterpret_cast<double*>(at.P[1] + slot[opp(q)]);
}
template <bool ODD, int q>
__device__ __forceinline__ double* adj_read_at(const AdjAt& at, const int (&slot)[27])
{
	if constexpr (ODD)
		return reinterpret_cast<double*>(at.P[1 - cz(q)] + at.oy[1 - cy(q)] + at.ox[1 - cx(q)] + slot[opp(q)]);
	else
		return reinterpret_cast<double*>(at.P[1] + slot[q]);
}

// collision constants of one site: the per-site force replaces the uniform one
template <typename T, typename R>
__device__ __forceinline__ CollParams<R> site_params(const AdjArgs<T, R>& a, long long site, long long nsites)
{
	CollParams<R> p = a.p;
	if (a.force) {
		p.fx = (R) a.force[site];
		p.fy = (R) a.force[nsites + site];
		p.fz = (R) a.force[2 * nsites + site];
		p.hfx = R(0.5) * p.fx;
		p.hfy = R(0.5) * p.fy;
		p.hfz = R(0.5) * p.fz;
	}
	return p;
}

// d feq_q(rho, u) / d u_a of the second-order equilibrium, contracted with a
// per-direction weight: adds l_q * d feq_q / d u to (bx, by, bz)
template <int q, typename R>
__device__ __forceinline__ void add_dfeq_du(R lq, R rho, R vx, R vy, R vz, R& bx, R& by, R& bz)
{
	const R cu = R(cx(q)) * vx + R(cy(q)) * vy + R(cz(q)) * vz;
	const R s = lq * R(weight(q)) * rho;
	const R g = R(3) + R(9) * cu;
	bx += s * (g * R(cx(q)) - R(3) * vx);
	by += s * (g * R(cy(q)) - R(3) * vy);
	bz += s * (g * R(cz(q)) - R(3) * vz);
}

// 8-byte asynchronous copy global -> shared (cp.async, cached in L1)
__device__ __forceinline__ void copy8_async(double* dst, const double* src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned) __cvta_generic_to_shared(dst)), "l"(src)
				 : "memory");
}

// primal moments and collision constants of one site, in FP64: the
// transpose is evaluated in FP64 at the primal's values (the FP32 primal's
// moments and constants converted exactly), so that the adjoint carries no
// FP32 rounding whatever the storage
struct AdjSite
{
	double rho, ir, vx, vy, vz;
	double fx, fy, fz;		  // the site's body force
	double inv_tau, srt_force;  // 1/tau, 1 - 1/(2 tau)
};

template <typename R>
__device__ __forceinline__ AdjSite adj_site(R rho, R vx, R vy, R vz, const CollParams<R>& p)
{
	AdjSite m;
	m.rho = (double) rho;
	m.ir = rho == R(0) ? 1.0 : (double) rcp(rho);
	m.vx = (double) vx;
	m.vy = (double) vy;
	m.vz = (double) vz;
	m.fx = (double) p.fx;
	m.fy = (double) p.fy;
	m.fz = (double) p.fz;
	m.inv_tau = (double) p.inv_tau;
	m.srt_force = (double) p.srt_force;
	return m;
}

// Transpose of the SRT update with body force at one site: l <- J^T l, and the
// force gradient dF += (d out / d F)^T l.  With g_q = w_q l_q every sum over the
// directions is one of the moments T_abc = sum_q g_q cx^a cy^b cz^c of order
// <= 3 (c^3 = c), and the weights factorise over the axes (2/3 and 1/6), so the
// 27 values are reduced line by line (three operations a line, 1/6 of each axis
// left to the end) and the rest is algebra on 17 numbers: about 240 FP64
// operations a site instead of about 1000 direction by direction.  The new
// value of direction j goes to put(j, value).
template <typename Put>
__device__ __forceinline__ void srt_vjp(const AdjSite& m, const double* l, double* dF, Put&& put)
{
	const double rho = m.rho, ir = m.ir;
	const double vx = m.vx, vy = m.vy, vz = m.vz;
	const double it = m.inv_tau, k = m.srt_force;
	// moments, the powers of cx, cy and cz in turn
	double M[27];
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int q = decltype(Qc)::value;
			M[ci(cx(q) + 1, cy(q) + 1, cz(q) + 1)] = l[q];
		}
	);
	auto line = [](double& a, double& b, double& c)
	{
		const double s = c + a, d = c - a;
		a = s + 4.0 * b;
		b = d;
		c = s;
	};
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int i = 0; i < 3; i++)
			line(M[ci(0, j, i)], M[ci(1, j, i)], M[ci(2, j, i)]);
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int i = 0; i < 3; i++)
			line(M[ci(j, 0, i)], M[ci(j, 1, i)], M[ci(j, 2, i)]);
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int i = 0; i < 3; i++)
			line(M[ci(j, i, 0)], M[ci(j, i, 1)], M[ci(j, i, 2)]);
	const double w = 1.0 / 216.0;
	const double T000 = w * M[ci(0, 0, 0)], T100 = w * M[ci(1, 0, 0)], T010 = w * M[ci(0, 1, 0)], T001 = w * M[ci(0, 0, 1)];
	const double T200 = w * M[ci(2, 0, 0)], T020 = w * M[ci(0, 2, 0)], T002 = w * M[ci(0, 0, 2)];
	const double T110 = w * M[ci(1, 1, 0)], T101 = w * M[ci(1, 0, 1)], T011 = w * M[ci(0, 1, 1)];
	const double T210 = w * M[ci(2, 1, 0)], T201 = w * M[ci(2, 0, 1)], T120 = w * M[ci(1, 2, 0)], T021 = w * M[ci(0, 2, 1)];
	const double T102 = w * M[ci(1, 0, 2)], T012 = w * M[ci(0, 1, 2)], T111 = w * M[ci(1, 1, 1)];
	// second moments contracted with u, and third moments contracted with u once
	const double ux = vx * T200 + vy * T110 + vz * T101;
	const double uy = vx * T110 + vy * T020 + vz * T011;
	const double uz = vx * T101 + vy * T011 + vz * T002;
	const double U200 = vx * T100 + vy * T210 + vz * T201, U020 = vx * T120 + vy * T010 + vz * T021;
	const double U002 = vx * T102 + vy * T012 + vz * T001, U110 = vx * T210 + vy * T120 + vz * T111;
	const double U101 = vx * T201 + vy * T111 + vz * T102, U011 = vx * T111 + vy * T021 + vz * T012;
	const double e0 = 1.0 - 1.5 * (vx * vx + vy * vy + vz * vz);
	// sum_q l_q feq_q and sum_q l_q feq_q (c_q - u)
	const double u1 = vx * T100 + vy * T010 + vz * T001;
	const double sum_lf = rho * (e0 * T000 + 3.0 * u1 + 4.5 * (vx * ux + vy * uy + vz * uz));
	const double hx = rho * (e0 * T100 + 3.0 * ux + 4.5 * (vx * U200 + vy * U110 + vz * U101)) - vx * sum_lf;
	const double hy = rho * (e0 * T010 + 3.0 * uy + 4.5 * (vx * U110 + vy * U020 + vz * U011)) - vy * sum_lf;
	const double hz = rho * (e0 * T001 + 3.0 * uz + 4.5 * (vx * U101 + vy * U011 + vz * U002)) - vz * sum_lf;
	// sum_q l_q (1/tau + k S_q) d feq_q / du, S_q = 3 (c_q - u).F / rho and
	// d feq_q / du = w_q rho ((3 + 9 c.u) c - 3 u), less the part of dS/du
	const double t = 3.0 * k * ir;
	const double gx = t * m.fx, gy = t * m.fy, gz = t * m.fz;
	const double al = it - (gx * vx + gy * vy + gz * vz);
	const double g1 = al * T000 + (gx * T100 + gy * T010 + gz * T001);
	const double bx = rho * (3.0 * (al * T100 + (gx * T200 + gy * T110 + gz * T101) - vx * g1)
							 + 9.0 * (al * ux + gx * U200 + gy * U110 + gz * U101)) - sum_lf * gx;
	const double by = rho * (3.0 * (al * T010 + (gx * T110 + gy * T020 + gz * T011) - vy * g1)
							 + 9.0 * (al * uy + gx * U110 + gy * U020 + gz * U011)) - sum_lf * gy;
	const double bz = rho * (3.0 * (al * T001 + (gx * T101 + gy * T011 + gz * T002) - vz * g1)
							 + 9.0 * (al * uz + gx * U101 + gy * U011 + gz * U002)) - sum_lf * gz;
	// the second pass reads l from memory again: held since the first it would
	// take 54 registers
	asm volatile("" ::: "memory");
	const double omit = 1.0 - it;
	const double Bx = bx * ir, By = by * ir, Bz = bz * ir;
	const double A = it * sum_lf * ir - (Bx * vx + By * vy + Bz * vz);
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int j = decltype(Qc)::value;
			put(Qc, omit * l[j] + (A + cx(j) * Bx + cy(j) * By + cz(j) * Bz));
		}
	);
	// d out / d F: through u (du/dF = 1 / (2 rho)) and through S directly
	dF[0] += 0.5 * Bx + t * hx;
	dF[1] += 0.5 * By + t * hy;
	dF[2] += 0.5 * Bz + t * hz;
}

// transpose of out = feq(1, u(f)) (GEO_OUTFLOW_EQ), in place
__device__ __forceinline__ void outflow_eq_vjp(const AdjSite& m, double* l, double* dF)
{
	const double ir = m.ir, vx = m.vx, vy = m.vy, vz = m.vz;
	double bx = 0, by = 0, bz = 0;
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int q = decltype(Qc)::value;
			add_dfeq_du<q>(l[q], 1.0, vx, vy, vz, bx, by, bz);
		}
	);
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int j = decltype(Qc)::value;
			l[j] = (bx * (cx(j) - vx) + by * (cy(j) - vy) + bz * (cz(j) - vz)) * ir;
		}
	);
	const double half_ir = 0.5 * ir;
	dF[0] += bx * half_ir;
	dF[1] += by * half_ir;
	dF[2] += bz * half_ir;
}

// transpose of the mirror copy of a symmetry plane (see symmetry(),
// aa_kernels.cuh), in place: the directions whose component along the normal
// equals `side` hand their adjoint to their mirror image (which is never one
// of them) and become zero
__device__ __forceinline__ void symmetry_vjp(double* l, int axis, int side)
{
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int q = decltype(Qc)::value;
			if constexpr (cx(q) != 0) {
				constexpr int m = dir(-cx(q), cy(q), cz(q));
				if (axis == 0 && cx(q) == side) {
					l[m] += l[q];
					l[q] = 0.0;
				}
			}
			if constexpr (cy(q) != 0) {
				constexpr int m = dir(cx(q), -cy(q), cz(q));
				if (axis == 1 && cy(q) == side) {
					l[m] += l[q];
					l[q] = 0.0;
				}
			}
			if constexpr (cz(q) != 0) {
				constexpr int m = dir(cx(q), cy(q), -cz(q));
				if (axis == 2 && cz(q) == side) {
					l[m] += l[q];
					l[q] = 0.0;
				}
			}
		}
	);
}

// Primal A-A step with SRT collision and a per-site force: the per-site code
// of aa_step_kernel (GENERAL, COLL_SRT) with the site's force in place of the
// uniform one.  With a uniform force field it is the production SRT step.
// With a.mom the sites' density and velocity before the collision are kept:
// all that the adjoint of the step needs of its primal input (16 bytes a site in
// FP32 where the populations are 108).
template <typename S, bool ODD>
__global__ void __launch_bounds__(128, adj_primal_minb<typename S::R, ODD>())
	adj_primal_kernel(const AdjArgs<typename S::T, typename S::R> a)
{
	using R = typename S::R;
	int x, y, z;
	long long site;
	if (!adj_position(a, site, x, y, z))
		return;
	const long long nsites = a.n;
	const uint8_t geo = a.map ? a.map[site] : (uint8_t) GEO_PERIODIC;
	if (geo == GEO_NOTHING)
		return;
	StepArgs<typename S::T, R> sa{};
	sa.Y = a.Y;
	sa.in_vx = a.in_vx;
	sa.in_vy = a.in_vy;
	sa.in_vz = a.in_vz;
	sa.p = site_params(a, site, nsites);
	const long long base = (long long) (z + 1) * a.sz + (long long) (y + 1) * a.sy + a.x0 + x;
	const Offsets o = neighbour_offsets(geo == GEO_PERIODIC, x, y, z, a.X, a.Y, a.Z, a.sy, a.sz);
	Site<R> s;
	aa_read<S, ODD>(a.f, a.sq, base, o, s.f);
	R rho_in = R(1);
	if (geo == GEO_OUTFLOW_EQ) {  // apply_boundary replaces the density
		density_velocity(s, sa.p);
		rho_in = s.rho;
	}
	const bool coll = apply_boundary(s, geo, sa, z, y);
	if (a.mom) {
		a.mom[site] = geo == GEO_OUTFLOW_EQ ? rho_in : s.rho;
		a.mom[nsites + site] = s.vx;
		a.mom[2 * nsites + site] = s.vy;
		a.mom[3 * nsites + site] = s.vz;
	}
	if (coll)
		collide<R, COLL_SRT, 0>(s, sa.p);
	aa_write<S, ODD>(a.f, a.sq, base, o, s.f);
}

// Adjoint of one A-A step: lam (adjoint of the step's output) is replaced in
// place by the adjoint of its input, with mom the moments of the step's primal
// input; grad accumulates the force gradient of this step.  The adjoint values
// of a site are gathered from its write locations, transformed in FP64 and
// scattered to its read locations.  Blocks of 128 threads (the shared array
// has one row per thread).
template <typename T, typename R, bool ODD>
__global__ void __launch_bounds__(128, ADJ_STEP_MINB) adj_step_kernel(const AdjArgs<T, R> a)
{
	int x, y, z;
	long long site;
	if (!adj_position(a, site, x, y, z))
		return;
	const long long nsites = a.n;
	const uint8_t geo = a.map ? a.map[site] : (uint8_t) GEO_PERIODIC;
	if (geo == GEO_NOTHING)
		return;
	// the site's 27 adjoint values live in shared memory (27 doubles per
	// thread, an odd stride: no bank conflicts beyond the two wavefronts of a
	// 64-bit access), not in registers: 54 registers fewer per thread and so
	// more resident warps for this memory-bound step
	__shared__ double lsh[128 * 27];
	double* const l = lsh + threadIdx.x * 27;
	const bool fluid = geo == GEO_FLUID || geo == GEO_PERIODIC;
	R mom[4] = {R(1), R(0), R(0), R(0)};
	AdjAt at = adj_at(a, geo == GEO_PERIODIC, x, y, z);
	// the adjoint values go straight to shared memory (asynchronous copies,
	// no registers), and the moments' loads are in flight with them
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int q = decltype(Qc)::value;
			copy8_async(l + q, adj_write_at<ODD, q>(at, a.slot));
		}
	);
	asm volatile("cp.async.commit_group;" ::: "memory");
	if (fluid || geo == GEO_OUTFLOW_EQ)
#pragma unroll
		for (int i = 0; i < 4; i++)
			mom[i] = a.mom[i * nsites + site];
	const CollParams<R> p = site_params(a, site, nsites);
	// each thread reads only its own row of lsh: the wait makes this
	// thread's copies visible to it, no block barrier is needed
	asm volatile("cp.async.wait_group 0;" ::: "memory");
	// the scatter's 27 addresses are formed anew from here, not kept since the
	// gather
#pragma unroll
	for (int i = 0; i < 3; i++)
		asm volatile("" : "+l"(at.P[i]));
	double dF[3] = {0, 0, 0};
	auto put = [&](auto Qc, double v) { *adj_read_at<ODD, decltype(Qc)::value>(at, a.slot) = v; };
	const AdjSite m = adj_site(mom[0], mom[1], mom[2], mom[3], p);
	if (fluid)
		srt_vjp(m, l, dF, put);
	else {
		if (geo == GEO_WALL)
			// full-way bounce-back swaps opposite directions: its transpose too
			static_for<13>(
				[&](auto Qc)
				{
					constexpr int q = 2 * decltype(Qc)::value + 1;
					const double t = l[q];
					l[q] = l[opp(q)];
					l[opp(q)] = t;
				}
			);
		else if (geo == GEO_INFLOW)
			static_for<27>(
				[&](auto Qc)
				{
					constexpr int q = decltype(Qc)::value;
					l[q] = 0.0;
				}
			);
		else if (geo >= GEO_SYM_TOP && geo <= GEO_SYM_FRONT) {
			const int axis = geo <= GEO_SYM_BOTTOM ? 2 : (geo <= GEO_SYM_RIGHT ? 0 : 1);
			const int side = (geo == GEO_SYM_TOP || geo == GEO_SYM_RIGHT || geo == GEO_SYM_FRONT) ? -1 : 1;
			symmetry_vjp(l, axis, side);
		}
		else
			outflow_eq_vjp(m, l, dF);
		static_for<27>([&](auto Qc) { put(Qc, l[decltype(Qc)::value]); });
	}
	if (a.grad && a.force && (dF[0] != 0.0 || dF[1] != 0.0 || dF[2] != 0.0)) {
		a.grad[site] += dF[0];
		a.grad[nsites + site] += dF[1];
		a.grad[2 * nsites + site] += dF[2];
	}
}

// Objective on the state f (the input of a step of the given parity):
// J = sum_i 1/2 [w_rho (rho_i - rho*_i)^2 + |u_i - u*_i|^2] at the sample
// sites, with rho and u the moments that step computes (density_velocity).
// Writes the per-sample terms to loss[i]; with lam set, adds seed * dJ/df to
// lam at the read locations and seed * dJ/dF to grad.  Sample sites are
// distinct fluid sites.
template <typename S, bool ODD>
__global__ void adj_objective_kernel(const AdjArgs<typename S::T, typename S::R> a, const long long* __restrict__ samples,
									 const double* __restrict__ target, int nsamples, double w_rho, double seed,
									 double* __restrict__ loss)
{
	using R = typename S::R;
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nsamples)
		return;
	const long long site = samples[i];
	const long long nsites = (long long) a.X * a.Y * a.Z;
	const int x = (int) (site % a.X);
	const int y = (int) ((site / a.X) % a.Y);
	const int z = (int) (site / ((long long) a.X * a.Y));
	const uint8_t geo = a.map ? a.map[site] : (uint8_t) GEO_PERIODIC;
	const CollParams<R> p = site_params(a, site, nsites);
	const long long base = (long long) (z + 1) * a.sz + (long long) (y + 1) * a.sy + a.x0 + x;
	const Offsets o = neighbour_offsets(geo == GEO_PERIODIC, x, y, z, a.X, a.Y, a.Z, a.sy, a.sz);
	Site<R> s;
	aa_read<S, ODD>(a.f, a.sq, base, o, s.f);
	density_velocity(s, p);
	const double drho = (double) s.rho - target[4 * i + 0];
	const double dvx = (double) s.vx - target[4 * i + 1];
	const double dvy = (double) s.vy - target[4 * i + 2];
	const double dvz = (double) s.vz - target[4 * i + 3];
	loss[i] = 0.5 * (w_rho * drho * drho + dvx * dvx + dvy * dvy + dvz * dvz);
	if (!a.lam)
		return;
	const double ir = (double) s.ir, vx = (double) s.vx, vy = (double) s.vy, vz = (double) s.vz;
	const double ex = seed * dvx, ey = seed * dvy, ez = seed * dvz, er = seed * w_rho * drho;
	static_for<27>(
		[&](auto Qc)
		{
			constexpr int q = decltype(Qc)::value;
			const double d = er + (ex * (cx(q) - vx) + ey * (cy(q) - vy) + ez * (cz(q) - vz)) * ir;
			a.lam[aa_read_loc<ODD, q>(a.sq, base, o)] += d;
		}
	);
	if (a.grad && a.force) {
		const double h = 0.5 / (double) s.rho;
		a.grad[site] += seed * dvx * h;
		a.grad[nsites + site] += seed * dvy * h;
		a.grad[2 * nsites + site] += seed * dvz * h;
	}
}

}  // namespace lbm
