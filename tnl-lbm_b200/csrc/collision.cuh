// Per-site operators of the D3Q27 hot path for the sm_100a kernels: moments,
// equilibria and the collision operators that share TNL-LBM's COLL slot
// (cumulant, SRT, BGK, MRT-LES).  All routines work on a register-resident
// site (27 populations plus rho and u) and are fully unrolled, so every array
// index below is a compile-time constant.
//
// Per-viscosity quantities (omega1, the Geier 2017 rates omega3..5, A, B and
// their products) are computed once per lattice on the host
// (lbm_abi.cu: make_coll_params) instead of per site as the reference does in
// col_cum.h:195-228.
#pragma once

#include <type_traits>
#include <utility>

#include "d3q27.cuh"

namespace lbm {

template <typename R>
struct Site
{
	R f[27];
	R rho, ir, vx, vy, vz;	// ir = 1 / rho
};

// collision-slot identifiers (runtime values of lbm_desc.collision)
enum Coll : int
{
	COLL_CUM = 0,
	COLL_SRT = 1,
	COLL_BGK = 2,
	COLL_MRT = 3
};
// cumulant variant bits (USE_GEIER_CUM_2017 / USE_GEIER_CUM_ANTIALIAS, defs.h:312-315)
enum : int
{
	CUM_2017 = 1,
	CUM_ANTIALIAS = 2
};
// equilibrium identifiers: D3Q27_EQ (eq.h) and D3Q27_EQ_INV_CUM (eq_inv_cum.h)
enum : int
{
	EQ_SECOND_ORDER = 0,
	EQ_INV_CUM = 1
};

// Per-lattice constants of the collision slot, in the compute type.  w1_3, w3 ..
// w5, c43 and cB are left for the collisions of plugins: the built-in ones read
// what is folded from them (l3 .. l5, kA, k45, kB).
template <typename R>
struct CollParams
{
	R nu;
	R fx, fy, fz;
	R hfx, hfy, hfz;  // half force for the velocity shift (common.h:40-48)
	// cumulant
	R w1, one_m_w1;
	R k33;			  // 3 (1 - omega1/2)
	R hw1, w1_3h, w1_3;	 // omega1/2, 3 omega1/2, 3 omega1
	R w3, w4, w5;	  // Geier 2017 third/fourth-order rates
	R c43, c45, cB;	  // (2/3) g A, -(4/3) g A, -(1/3) g B with g = 1/omega1 - 1/2
	R l3, l4, l5;	  // lambda (1 - omega3) / 2, lambda (1 - omega4) / 2, lambda (1 - omega5), lambda = 0.01
	R kA, k45, kB;	  // c43 omega1 / 2, c45 omega1 / 2, -3 omega1 cB
	// SRT / BGK / MRT
	R inv_tau, srt_force;  // 1/tau, 1 - 1/(2 tau)
	R bgk_force;		   // 1 - omega1/2
	R tau, tau2;		   // MRT-LES: tau and tau^2
	int eq;				   // equilibrium used by SRT and by equilibrium BCs
};

template <typename R>
__device__ __forceinline__ R rcp(R x)
{
	return R(1) / x;
}
template <>
__device__ __forceinline__ float rcp<float>(float x)
{
	return __frcp_rn(x);
}
// division where a few ulp do not matter (limiter weights)
template <typename R>
__device__ __forceinline__ R div_approx(R a, R b)
{
	return a / b;
}
template <>
__device__ __forceinline__ float div_approx<float>(float a, float b)
{
	return __fdividef(a, b);
}

// a b + c: the compiler contracts it for scalars, the packed type has its own
template <typename R>
__device__ __forceinline__ R fmadd(R a, R b, R c)
{
	return a * b + c;
}

// density and velocity with the half-force shift; pairwise summation order of
// common.h:31-49 (Geier 2015 Appendix J)
template <typename R>
__device__ __forceinline__ void density_velocity(Site<R>& s, const CollParams<R>& p)
{
	const R* f = s.f;
	s.rho = ((((f[PPP] + f[MMM]) + (f[PMP] + f[MPM])) + ((f[PPM] + f[MMP]) + (f[MPP] + f[PMM])))
			 + (((f[ZPP] + f[ZMM]) + (f[ZPM] + f[ZMP])) + ((f[PZP] + f[MZM]) + (f[PZM] + f[MZP]))
				+ ((f[PPZ] + f[MMZ]) + (f[PMZ] + f[MPZ])))
			 + ((f[PZZ] + f[MZZ]) + (f[ZPZ] + f[ZMZ]) + (f[ZZP] + f[ZZM])))
		  + f[ZZZ];
	s.ir = rcp(s.rho);
	s.vz = ((((f[PPP] - f[MMM]) + (f[MPP] - f[PMM])) + ((f[PMP] - f[MPM]) + (f[MMP] - f[PPM])))
			+ (((f[ZPP] - f[ZMM]) + (f[ZMP] - f[ZPM])) + ((f[PZP] - f[MZM]) + (f[MZP] - f[PZM]))) + (f[ZZP] - f[ZZM]) + p.hfz)
		 * s.ir;
	s.vx = ((((f[PPP] - f[MMM]) + (f[PMP] - f[MPM])) + ((f[PPM] - f[MMP]) + (f[PMM] - f[MPP])))
			+ (((f[PZP] - f[MZM]) + (f[PZM] - f[MZP])) + ((f[PPZ] - f[MMZ]) + (f[PMZ] - f[MPZ]))) + (f[PZZ] - f[MZZ]) + p.hfx)
		 * s.ir;
	s.vy = ((((f[PPP] - f[MMM]) + (f[PPM] - f[MMP])) + ((f[MPP] - f[PMM]) + (f[MPM] - f[PMP])))
			+ (((f[PPZ] - f[MMZ]) + (f[MPZ] - f[PMZ])) + ((f[ZPP] - f[ZMM]) + (f[ZPM] - f[ZMP]))) + (f[ZPZ] - f[ZMZ]) + p.hfy)
		 * s.ir;
}

// ---------------------------------------------------------------------------
// equilibria, direction by direction
// ---------------------------------------------------------------------------

// second-order equilibrium w_q rho (1 + 3 c.u + 4.5 (c.u)^2 - 1.5 u^2) (eq.h:13-130)
template <int Q, typename R>
__device__ __forceinline__ R eq_second(R rho, R vx, R vy, R vz, R usq)
{
	const R cu = R(cx(Q)) * vx + R(cy(Q)) * vy + R(cz(Q)) * vz;
	return R(weight(Q)) * rho * ((R(1) - R(1.5) * usq + R(3) * cu) + R(4.5) * cu * cu);
}

// per-axis factor of the factorised equilibrium (eq_inv_cum.h:24-136)
template <int C, typename R>
__device__ __forceinline__ R inv_cum_axis(R v, R v3v)	// v3v = 3 v^2
{
	return C == 0 ? v3v - R(2) : (C > 0 ? v3v + R(3) * v + R(1) : v3v - R(3) * v + R(1));
}
template <int Q>
__host__ __device__ constexpr double inv_cum_coef()
{
	return nnz(Q) == 0 ? -1.0 / 27.0 : nnz(Q) == 1 ? 1.0 / 54.0 : nnz(Q) == 2 ? -1.0 / 108.0 : 1.0 / 216.0;
}
template <int Q, typename R>
__device__ __forceinline__ R eq_inv_cum(R rho, R vx, R vy, R vz, R vx3, R vy3, R vz3)
{
	return R(inv_cum_coef<Q>()) * rho
		 * (inv_cum_axis<cx(Q)>(vx, vx3) * inv_cum_axis<cy(Q)>(vy, vy3) * inv_cum_axis<cz(Q)>(vz, vz3));
}

template <typename R>
__device__ __forceinline__ void set_equilibrium(R* f, int eq, R rho, R vx, R vy, R vz)
{
	if (eq == EQ_INV_CUM) {
		const R vx3 = R(3) * vx * vx, vy3 = R(3) * vy * vy, vz3 = R(3) * vz * vz;
#pragma unroll
		for (int q = 0; q < 27; q++) {
			// explicit instantiation per direction
			switch (q) {
#define LBM_EQ_CASE(Q) \
	case Q: f[Q] = eq_inv_cum<Q>(rho, vx, vy, vz, vx3, vy3, vz3); break;
				LBM_EQ_CASE(0) LBM_EQ_CASE(1) LBM_EQ_CASE(2) LBM_EQ_CASE(3) LBM_EQ_CASE(4) LBM_EQ_CASE(5)
				LBM_EQ_CASE(6) LBM_EQ_CASE(7) LBM_EQ_CASE(8) LBM_EQ_CASE(9) LBM_EQ_CASE(10) LBM_EQ_CASE(11)
				LBM_EQ_CASE(12) LBM_EQ_CASE(13) LBM_EQ_CASE(14) LBM_EQ_CASE(15) LBM_EQ_CASE(16) LBM_EQ_CASE(17)
				LBM_EQ_CASE(18) LBM_EQ_CASE(19) LBM_EQ_CASE(20) LBM_EQ_CASE(21) LBM_EQ_CASE(22) LBM_EQ_CASE(23)
				LBM_EQ_CASE(24) LBM_EQ_CASE(25) LBM_EQ_CASE(26)
#undef LBM_EQ_CASE
			}
		}
	}
	else {
		const R usq = vx * vx + vy * vy + vz * vz;
#pragma unroll
		for (int q = 0; q < 27; q++) {
			switch (q) {
#define LBM_EQ_CASE(Q) \
	case Q: f[Q] = eq_second<Q>(rho, vx, vy, vz, usq); break;
				LBM_EQ_CASE(0) LBM_EQ_CASE(1) LBM_EQ_CASE(2) LBM_EQ_CASE(3) LBM_EQ_CASE(4) LBM_EQ_CASE(5)
				LBM_EQ_CASE(6) LBM_EQ_CASE(7) LBM_EQ_CASE(8) LBM_EQ_CASE(9) LBM_EQ_CASE(10) LBM_EQ_CASE(11)
				LBM_EQ_CASE(12) LBM_EQ_CASE(13) LBM_EQ_CASE(14) LBM_EQ_CASE(15) LBM_EQ_CASE(16) LBM_EQ_CASE(17)
				LBM_EQ_CASE(18) LBM_EQ_CASE(19) LBM_EQ_CASE(20) LBM_EQ_CASE(21) LBM_EQ_CASE(22) LBM_EQ_CASE(23)
				LBM_EQ_CASE(24) LBM_EQ_CASE(25) LBM_EQ_CASE(26)
#undef LBM_EQ_CASE
			}
		}
	}
}

// ---------------------------------------------------------------------------
// cumulant collision (col_cum.h:13-511; Geier 2015 / Geier 2017)
// ---------------------------------------------------------------------------

// cube index of a direction or of a moment triple (orders or positions 0..2)
__host__ __device__ constexpr int ci(int i, int j, int k)
{
	return i * 9 + j * 3 + k;
}

// forward chimera transform of a line (m, z, p) about velocity u (Eqs 6-14)
template <typename R>
__device__ __forceinline__ void chim_fwd(R& m, R& z, R& p, R u, R u2)
{
	const R s = p + m, d = p - m;
	const R k0 = s + z;
	const R k1 = d - u * k0;
	const R k2 = s - R(2) * u * d + u2 * k0;
	m = k0;
	z = k1;
	p = k2;
}

// backward chimera transform (Eqs 88-96 of Geier 2015), written through the
// sum s = v+ + v- = k0 u^2 + 2 u k1 + k2 and the difference d = v+ - v- =
// u k0 + k1 of the outer values: v0 = k0 - s, v+- = (s +- d) / 2.  The three
// values then add up to k0 and their first moment is d up to one rounding
// each, the mass and momentum the line carries, where the term-by-term form
// of the paper rounds every term separately.
template <typename R>
__device__ __forceinline__ void chim_bwd(R& a, R& b, R& c, R u, R u2)
{
	const R k0 = a, k1 = b, k2 = c;
	const R s = k0 * u2 + (R(2) * u * k1 + k2);
	const R hd = R(0.5) * (u * k0 + k1);
	a = s * R(0.5) - hd;
	b = k0 - s;
	c = s * R(0.5) + hd;
}

// backward transforms of lines with vanishing moments (the default cumulant's odd
// moments of order three and five)
template <typename R>
__device__ __forceinline__ void chim_bwd_no_k1(R& a, R& b, R& c, R u, R u2)
{
	const R k0 = a;
	const R s = fmadd(k0, u2, c), hd = (R(0.5) * u) * k0;
	a = fmadd(s, R(0.5), -hd);
	b = k0 - s;
	c = fmadd(s, R(0.5), hd);
}
template <typename R>
__device__ __forceinline__ void chim_bwd_only_k1(R& a, R& b, R& c, R u)
{
	const R k1 = b;
	a = (u - R(0.5)) * k1;
	b = (R(-2) * u) * k1;
	c = (u + R(0.5)) * k1;
}

// The cumulant collision, with as few operations as the algebra leaves: it runs
// on the FP32 (or FP64) pipes, which bound every 16-bit step and every lattice
// that L2 holds.  Against the formulas term by term, some 190 of them packed
// operations a pair between the transforms (75 in the default variant), now
// about 105 (45):
//   * products with 1/rho are formed once per cumulant and enter one multiply-add;
//   * the two other normal stresses follow from the first and the differences
//     that are relaxed: (e34 + e35 - 2 e33) / 3 = (e33 + e34 + e35) / 3 - e33;
//   * a limited rate w + (1 - w) |C| / (lambda rho + |C|) leaves the factor
//     1 - rate = (1 - w) lambda rho / (lambda rho + |C|), without the cancellation;
//   * the fourth-order equilibria are those of the stress differences, the
//     viscosity's constants folded on the host (kA, k45, kB; rho / rho = 1);
//   * terms that vanish in the default variant are not formed (an addition of
//     0 x is not the compiler's to drop).
// B200, us a step: duct 512x128x128 FP16 (default) 224.5 -> 212.6, Taylor-Green
// vortex (Geier 2017) 256^3 FP16 475 -> 462, 64^3 FP32 (in L2) 10.1 -> 9.4; steps that
// HBM bounds stay.  Errors against FP64 are unchanged (FP32, 400 steps: 5e-7 of the
// populations, 2e-5 of the velocity).
template <typename R, int FLAGS>
__device__ __forceinline__ void collide_cumulant(Site<R>& s, const CollParams<R>& p)
{
	constexpr bool v2017 = (FLAGS & CUM_2017) != 0;
	constexpr bool antialias = (FLAGS & CUM_ANTIALIAS) != 0;
	const R rho = s.rho, ir = s.ir, vx = s.vx, vy = s.vy, vz = s.vz;
	const R vx2 = vx * vx, vy2 = vy * vy, vz2 = vz * vz;

	R M[27];
#pragma unroll
	for (int q = 0; q < 27; q++)
		M[ci(cx(q) + 1, cy(q) + 1, cz(q) + 1)] = s.f[q];
#pragma unroll
	for (int i = 0; i < 3; i++)
#pragma unroll
		for (int j = 0; j < 3; j++)
			chim_fwd(M[ci(i, j, 0)], M[ci(i, j, 1)], M[ci(i, j, 2)], vz, vz2);
#pragma unroll
	for (int i = 0; i < 3; i++)
#pragma unroll
		for (int k = 0; k < 3; k++)
			chim_fwd(M[ci(i, 0, k)], M[ci(i, 1, k)], M[ci(i, 2, k)], vy, vy2);
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int k = 0; k < 3; k++)
			chim_fwd(M[ci(0, j, k)], M[ci(1, j, k)], M[ci(2, j, k)], vx, vx2);

	// central moments M[ci(a,b,c)] = k_abc; cumulants of order <= 3 equal them
	const R k000 = M[ci(0, 0, 0)];
	const R C110 = M[ci(1, 1, 0)], C101 = M[ci(1, 0, 1)], C011 = M[ci(0, 1, 1)];
	const R C200 = M[ci(2, 0, 0)], C020 = M[ci(0, 2, 0)], C002 = M[ci(0, 0, 2)];

	// second order (col_cum.h:231-259), omega2 = 1, with the velocity
	// derivatives of the anti-aliasing terms (col_cum.h:234-250)
	const R d1 = C200 - C020, d2 = C200 - C002;
	const R Cs110 = p.one_m_w1 * C110;
	const R Cs101 = p.one_m_w1 * C101;
	const R Cs011 = p.one_m_w1 * C011;
	R e33 = p.one_m_w1 * d1, e34 = p.one_m_w1 * d2, e35 = k000;
	R Dxu = 0;
	if constexpr (antialias) {
		const R trace = ((C200 + C020) + C002) - (rho - R(1));
		Dxu = -ir * fmadd(p.hw1, d1 + d2, R(0.5) * trace);
		const R wir = p.w1_3h * ir;
		const R Dyv = fmadd(wir, d1, Dxu), Dzw = fmadd(wir, d2, Dxu);
		const R x = vx2 * Dxu, y = vy2 * Dyv, z = vz2 * Dzw;
		const R kr = p.k33 * rho;
		e33 = fmadd(kr, y - x, e33);
		e34 = fmadd(kr, z - x, e34);
		e35 = fmadd(R(-1.5) * rho, (x + y) + z, k000);
	}
	const R Cs200 = R(1.0 / 3.0) * ((e33 + e34) + e35);
	const R Cs020 = Cs200 - e33;
	const R Cs002 = Cs200 - e34;

	// products with 1/rho (normal stresses) and 2/rho (shear stresses)
	const R ir2 = ir + ir;
	const R P = Cs200 * ir, Q = Cs020 * ir, S = Cs002 * ir;
	const R A2 = Cs110 * ir2, B2 = Cs101 * ir2, C2 = Cs011 * ir2;

	// fourth-order cumulants to central moments (Eqs 81-84 of Geier 2015)
	R ks211, ks121, ks112, ks220, ks022, ks202;
	R odd = 0;	// third-order part of k222, times rho / 2
	if constexpr (v2017) {
		// third order (Eqs 117-122, 42) with limited rates (col_cum.h:203-216);
		// fifth- and sixth-order cumulants relax fully (col_cum.h:294-297)
		const R C120 = M[ci(1, 2, 0)], C102 = M[ci(1, 0, 2)], C210 = M[ci(2, 1, 0)];
		const R C012 = M[ci(0, 1, 2)], C201 = M[ci(2, 0, 1)], C021 = M[ci(0, 2, 1)];
		const R C111 = M[ci(1, 1, 1)];
		const R lam_rho = R(0.01) * rho;
		const R n3 = p.l3 * rho, n4 = p.l4 * rho, n5 = p.l5 * rho;
		auto limited = [&](R n, R c) { return c * div_approx(n, lam_rho + fabs(c)); };
		const R e117 = limited(n3, C120 + C102), e120 = limited(n4, C120 - C102);
		const R e118 = limited(n3, C210 + C012), e121 = limited(n4, C210 - C012);
		const R e119 = limited(n3, C201 + C021), e122 = limited(n4, C201 - C021);
		const R Cs120 = e117 + e120, Cs102 = e117 - e120;
		const R Cs210 = e118 + e121, Cs012 = e118 - e121;
		const R Cs201 = e119 + e122, Cs021 = e119 - e122;
		const R Cs111 = limited(n5, C111), two111 = Cs111 + Cs111;
		// fourth order (Eqs 43-48), omega6 = omega7 = omega8 = 1
		const R a = d1 + d2;
		const R e45 = fmadd(p.c45 * rho, Dxu, p.k45 * a);
		const R Cs220 = fmadd(-p.kA, a, e45);
		const R Cs202 = fmadd(-p.kA, fmadd(R(-2), d1, d2), e45);
		const R Cs022 = fmadd(-p.kA, fmadd(R(-2), d2, d1), e45);
		ks211 = fmadd(P, Cs011, fmadd(B2, Cs110, p.kB * C011));
		ks121 = fmadd(Q, Cs101, fmadd(A2, Cs011, p.kB * C101));
		ks112 = fmadd(S, Cs110, fmadd(C2, Cs101, p.kB * C110));
		ks220 = fmadd(Q, Cs200, fmadd(A2, Cs110, Cs220));
		ks022 = fmadd(S, Cs020, fmadd(C2, Cs011, Cs022));
		ks202 = fmadd(P, Cs002, fmadd(B2, Cs101, Cs202));
		// Cs221, Cs212, Cs122, Cs222 = 0
		M[ci(1, 2, 2)] = fmadd(Q, Cs102, fmadd(S, Cs120, fmadd(C2, two111, fmadd(A2, Cs012, B2 * Cs021))));
		M[ci(2, 1, 2)] = fmadd(S, Cs210, fmadd(P, Cs012, fmadd(B2, two111, fmadd(C2, Cs201, A2 * Cs102))));
		M[ci(2, 2, 1)] = fmadd(P, Cs021, fmadd(Q, Cs201, fmadd(A2, two111, fmadd(B2, Cs120, C2 * Cs210))));
		odd = fmadd(Cs111, two111, fmadd(Cs120, Cs102, fmadd(Cs210, Cs012, Cs201 * Cs021)));
		M[ci(1, 2, 0)] = Cs120;
		M[ci(1, 0, 2)] = Cs102;
		M[ci(2, 1, 0)] = Cs210;
		M[ci(0, 1, 2)] = Cs012;
		M[ci(2, 0, 1)] = Cs201;
		M[ci(0, 2, 1)] = Cs021;
		M[ci(1, 1, 1)] = Cs111;
	}
	else {
		// default variant (col_cum.h:330-366)
		ks211 = fmadd(P, Cs011, B2 * Cs110);
		ks121 = fmadd(Q, Cs101, A2 * Cs011);
		ks112 = fmadd(S, Cs110, C2 * Cs101);
		ks220 = fmadd(Q, Cs200, A2 * Cs110);
		ks022 = fmadd(S, Cs020, C2 * Cs011);
		ks202 = fmadd(P, Cs002, B2 * Cs101);
	}
	R ks222 = fmadd(P, ks022, fmadd(Q, ks202, S * ks220));
	ks222 = fmadd(R(2), fmadd(C2, ks211, fmadd(B2, ks121, A2 * ks112)), ks222);
	if constexpr (v2017)
		ks222 = fmadd(ir2, odd, ks222);
	{
		R t = R(4) * ((A2 * B2) * Cs011);
		t = fmadd(B2 * B2, Cs020, t);
		t = fmadd(C2 * C2, Cs200, t);
		t = fmadd(A2 * A2, Cs002, t);
		t = fmadd(P + P, Q * Cs002, t);
		ks222 = ks222 - t;
	}

	// post-collision central moments; first moments flipped (col_cum.h:369-373)
	M[ci(1, 0, 0)] = -M[ci(1, 0, 0)];
	M[ci(0, 1, 0)] = -M[ci(0, 1, 0)];
	M[ci(0, 0, 1)] = -M[ci(0, 0, 1)];
	M[ci(1, 1, 0)] = Cs110;
	M[ci(1, 0, 1)] = Cs101;
	M[ci(0, 1, 1)] = Cs011;
	M[ci(2, 0, 0)] = Cs200;
	M[ci(0, 2, 0)] = Cs020;
	M[ci(0, 0, 2)] = Cs002;
	M[ci(2, 1, 1)] = ks211;
	M[ci(1, 2, 1)] = ks121;
	M[ci(1, 1, 2)] = ks112;
	M[ci(2, 2, 0)] = ks220;
	M[ci(0, 2, 2)] = ks022;
	M[ci(2, 0, 2)] = ks202;
	M[ci(2, 2, 2)] = ks222;

	if constexpr (v2017) {
#pragma unroll
		for (int j = 0; j < 3; j++)
#pragma unroll
			for (int k = 0; k < 3; k++)
				chim_bwd(M[ci(0, j, k)], M[ci(1, j, k)], M[ci(2, j, k)], vx, vx2);
	}
	else {
		// the odd moments of order three and five are zero
		M[ci(2, 0, 1)] = M[ci(2, 1, 0)] = R(0);
		chim_bwd(M[ci(0, 0, 0)], M[ci(1, 0, 0)], M[ci(2, 0, 0)], vx, vx2);
		chim_bwd(M[ci(0, 0, 1)], M[ci(1, 0, 1)], M[ci(2, 0, 1)], vx, vx2);
		chim_bwd(M[ci(0, 1, 0)], M[ci(1, 1, 0)], M[ci(2, 1, 0)], vx, vx2);
		chim_bwd_no_k1(M[ci(0, 0, 2)], M[ci(1, 0, 2)], M[ci(2, 0, 2)], vx, vx2);
		chim_bwd_no_k1(M[ci(0, 1, 1)], M[ci(1, 1, 1)], M[ci(2, 1, 1)], vx, vx2);
		chim_bwd_no_k1(M[ci(0, 2, 0)], M[ci(1, 2, 0)], M[ci(2, 2, 0)], vx, vx2);
		chim_bwd_no_k1(M[ci(0, 2, 2)], M[ci(1, 2, 2)], M[ci(2, 2, 2)], vx, vx2);
		chim_bwd_only_k1(M[ci(0, 1, 2)], M[ci(1, 1, 2)], M[ci(2, 1, 2)], vx);
		chim_bwd_only_k1(M[ci(0, 2, 1)], M[ci(1, 2, 1)], M[ci(2, 2, 1)], vx);
	}
#pragma unroll
	for (int i = 0; i < 3; i++)
#pragma unroll
		for (int k = 0; k < 3; k++)
			chim_bwd(M[ci(i, 0, k)], M[ci(i, 1, k)], M[ci(i, 2, k)], vy, vy2);
#pragma unroll
	for (int i = 0; i < 3; i++)
#pragma unroll
		for (int j = 0; j < 3; j++)
			chim_bwd(M[ci(i, j, 0)], M[ci(i, j, 1)], M[ci(i, j, 2)], vz, vz2);
#pragma unroll
	for (int q = 0; q < 27; q++)
		s.f[q] = M[ci(cx(q) + 1, cy(q) + 1, cz(q) + 1)];
}

// ---------------------------------------------------------------------------
// SRT, BGK, MRT-LES through the same slot
// ---------------------------------------------------------------------------

// calls f with std::integral_constant q for every direction, or for one of every
// two opposite ones
template <int... Is, typename F>
__device__ __forceinline__ void each_direction_of(std::integer_sequence<int, Is...>, F&& f)
{
	(f(std::integral_constant<int, Is>{}), ...);
}
template <typename F>
__device__ __forceinline__ void each_direction(F&& f)
{
	each_direction_of(std::make_integer_sequence<int, 27>{}, f);
}
template <typename F>
__device__ __forceinline__ void each_pair(F&& f)
{
	each_direction_of(std::integer_sequence<int, 1, 3, 5, 7, 9, 11, 13, 15, 17, 19, 21, 23, 25>{}, f);
}
// c_q . v without the components that are zero
template <int Q, typename R>
__device__ __forceinline__ R along(R x, R y, R z)
{
	const R sx = cx(Q) > 0 ? x : -x, sy = cy(Q) > 0 ? y : -y, sz = cz(Q) > 0 ? z : -z;
	if constexpr (cx(Q) != 0 && cy(Q) != 0 && cz(Q) != 0)
		return (sx + sy) + sz;
	else if constexpr (cx(Q) != 0 && cy(Q) != 0)
		return sx + sy;
	else if constexpr (cx(Q) != 0 && cz(Q) != 0)
		return sx + sz;
	else if constexpr (cy(Q) != 0 && cz(Q) != 0)
		return sy + sz;
	else if constexpr (cx(Q) != 0)
		return sx;
	else if constexpr (cy(Q) != 0)
		return sy;
	else if constexpr (cz(Q) != 0)
		return sz;
	else
		return R(0);
}

// 1 / rho for the SRT forcing, 1 where rho = 0 (col_srt.h:19, the ADE case)
template <typename R>
__device__ __forceinline__ R inv_rho_or_one(const Site<R>& s)
{
	return s.rho == R(0) ? R(1) : s.ir;
}

// Guo-like forcing term S_q = 3 (c_q - u).F / rho (col_srt.h:22-48)
template <int Q, typename R>
__device__ __forceinline__ R force_term(const Site<R>& s, const CollParams<R>& p, R irho)
{
	return R(3) * ((R(cx(Q)) - s.vx) * p.fx + (R(cy(Q)) - s.vy) * p.fy + (R(cz(Q)) - s.vz) * p.fz) * irho;
}

// relaxation and forcing of one direction; the population is rounded once
template <typename R>
__device__ __forceinline__ void relax(R& f, R feq, R rate, R k)
{
	f = f + fmadd(feq - f, rate, feq * k);
}

// Textbook BGK (col_srt.h:14-105).  FP64 and the packed pairs form the equilibrium
// of a direction where it is used, the second-order one for two opposite
// directions together (its even and odd part; each direction's product with the
// weight is rounded by itself, or the density errors of a pair would add up), and
// the forcing 3 (c - u).F / rho feq as linear in c, its factor k0 + c.k: with the 27
// equilibria in an array first the packed kernel spilled 56-170 bytes.  B200, us a
// step: duct 512x128x128 FP32 on the two-site kernel 318 -> 289, 256x96x96 FP64
// 171 -> 159.  One site in FP32 keeps the reference's order of operations: nothing
// spills there, and the adjoint's objective in FP32 is nearer to FP64 with it.
template <typename R>
__device__ __forceinline__ void collide_srt(Site<R>& s, const CollParams<R>& p)
{
	if constexpr (std::is_same<R, float>::value) {
		R feq[27];
		set_equilibrium(feq, p.eq, s.rho, s.vx, s.vy, s.vz);
		const R irho = inv_rho_or_one(s);
		each_direction(
			[&](auto Qc)
			{
				constexpr int q = decltype(Qc)::value;
				s.f[q] += (feq[q] - s.f[q]) * p.inv_tau + p.srt_force * force_term<q>(s, p, irho) * feq[q];
			}
		);
	}
	else {
		const R rho = s.rho, vx = s.vx, vy = s.vy, vz = s.vz;
		const R g = R(3) * (p.srt_force * inv_rho_or_one(s));
		const R kx = g * p.fx, ky = g * p.fy, kz = g * p.fz;
		const R k0 = -fmadd(vx, kx, fmadd(vy, ky, vz * kz));
		if (p.eq == EQ_INV_CUM) {
			const R vx3 = R(3) * vx * vx, vy3 = R(3) * vy * vy, vz3 = R(3) * vz * vz;
			each_direction(
				[&](auto Qc)
				{
					constexpr int q = decltype(Qc)::value;
					relax(s.f[q], eq_inv_cum<q>(rho, vx, vy, vz, vx3, vy3, vz3), p.inv_tau, along<q>(kx, ky, kz) + k0);
				}
			);
		}
		else {
			const R base = fmadd(R(-1.5), fmadd(vx, vx, fmadd(vy, vy, vz * vz)), R(1));
			relax(s.f[ZZZ], (R(weight(ZZZ)) * rho) * base, p.inv_tau, k0);
			each_pair(
				[&](auto Qc)
				{
					constexpr int q = decltype(Qc)::value, m = opp(q);
					const R wr = R(weight(q)) * rho;
					const R cu = along<q>(vx, vy, vz), ck = along<q>(kx, ky, kz);
					const R even = fmadd(R(4.5) * cu, cu, base), odd = R(3) * cu;
					relax(s.f[q], wr * (even + odd), p.inv_tau, k0 + ck);
					relax(s.f[m], wr * (even - odd), p.inv_tau, k0 - ck);
				}
			);
		}
	}
}

// Geier's improved BGK with factorised equilibrium (col_bgk.h:18-144)
template <typename R>
__device__ __forceinline__ void collide_bgk(Site<R>& s, const CollParams<R>& p)
{
	const R third = R(1.0 / 3.0);
	const R Xz = third - R(1) + s.vx * s.vx, Xp = R(-0.5) * (Xz + R(1) + s.vx), Xm = Xp + s.vx;
	const R Yz = third - R(1) + s.vy * s.vy, Yp = R(-0.5) * (Yz + R(1) + s.vy), Ym = Yp + s.vy;
	const R Zz = third - R(1) + s.vz * s.vz, Zp = R(-0.5) * (Zz + R(1) + s.vz), Zm = Zp + s.vz;
	// the forcing as collide_srt's
	const R g = R(3) * (p.bgk_force * s.ir);
	const R kx = g * p.fx, ky = g * p.fy, kz = g * p.fz;
	const R k0 = -fmadd(s.vx, kx, fmadd(s.vy, ky, s.vz * kz));
	each_direction([&](auto Qc) {
		constexpr int q = decltype(Qc)::value;
		const R X = cx(q) == 0 ? Xz : (cx(q) > 0 ? Xp : Xm);
		const R Y = cy(q) == 0 ? Yz : (cy(q) > 0 ? Yp : Ym);
		const R Z = cz(q) == 0 ? Zz : (cz(q) > 0 ? Zp : Zm);
		relax(s.f[q], -s.rho * X * Y * Z, p.w1, along<q>(kx, ky, kz) + k0);
	});
}

// MRT-LES: Smagorinsky-relaxed second moments, populations rebuilt from
// rho, u and the relaxed tensor (col_mrt.h:14-141)
template <typename R>
__device__ __forceinline__ void collide_mrt(Site<R>& s, const CollParams<R>& p)
{
	R Pxx = 0, Pyy = 0, Pzz = 0, Pxy = 0, Pxz = 0, Pyz = 0;
#pragma unroll
	for (int q = 0; q < 27; q++) {
		const R v = s.f[q];
		if (cx(q) != 0)
			Pxx += v;
		if (cy(q) != 0)
			Pyy += v;
		if (cz(q) != 0)
			Pzz += v;
		if (cx(q) * cy(q) != 0)
			Pxy += R(cx(q) * cy(q)) * v;
		if (cx(q) * cz(q) != 0)
			Pxz += R(cx(q) * cz(q)) * v;
		if (cy(q) * cz(q) != 0)
			Pyz += R(cy(q) * cz(q)) * v;
	}
	const R rho = s.rho, vx = s.vx, vy = s.vy, vz = s.vz;
	const R third = R(1.0 / 3.0);
	const R Pnxx = Pxx - rho * (third + vx * vx);
	const R Pnyy = Pyy - rho * (third + vy * vy);
	const R Pnzz = Pzz - rho * (third + vz * vz);
	const R Pnxz = Pxz - rho * vx * vz;
	const R Pnxy = Pxy - rho * vx * vy;
	const R Pnyz = Pyz - rho * vy * vz;
	const R Q = R(2) * (Pnxx * Pnxx + Pnyy * Pnyy + Pnzz * Pnzz + R(2) * (Pnxy * Pnxy + Pnxz * Pnxz + Pnyz * Pnyz));
	const R omega = R(2) / (sqrt(p.tau2 + R(2 * 0.0342 * 9.0) * sqrt(Q) * s.ir) + p.tau);
	Pxx -= omega * Pnxx;
	Pyy -= omega * Pnyy;
	Pzz -= omega * Pnzz;
	Pxy -= omega * Pnxy;
	Pxz -= omega * Pnxz;
	Pyz -= omega * Pnyz;
	const R P2 = Pxx + Pyy + Pzz;
#pragma unroll
	for (int q = 0; q < 27; q++) {
		const R cu = vx * R(cx(q)) + vy * R(cy(q)) + vz * R(cz(q));
		const R cc = Pxx * R(cx(q) * cx(q)) + Pyy * R(cy(q) * cy(q)) + Pzz * R(cz(q) * cz(q))
				   + R(2) * (Pxy * R(cx(q) * cy(q)) + Pxz * R(cx(q) * cz(q)) + Pyz * R(cy(q) * cz(q)));
		s.f[q] = R(weight(q)) * (rho * ((R(2.5) - R(1.5) * R(nnz(q))) + R(3) * cu) + R(4.5) * cc - R(1.5) * P2);
	}
}

template <typename R, int COLL, int CUMF>
__device__ __forceinline__ void collide(Site<R>& s, const CollParams<R>& p)
{
	if constexpr (COLL == COLL_CUM)
		collide_cumulant<R, CUMF>(s, p);
	else if constexpr (COLL == COLL_SRT)
		collide_srt(s, p);
	else if constexpr (COLL == COLL_BGK)
		collide_bgk(s, p);
	else
		collide_mrt(s, p);
}

}  // namespace lbm
