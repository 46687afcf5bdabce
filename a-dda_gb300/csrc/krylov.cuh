// krylov.cuh - what the Krylov vector kernels (solver.cu) and the matvec's last kernel share: block sums, the state of a
// right-hand side, and the scalar steps of the recurrences, which run in the last block of the kernel whose sums they
// need.
//
// GB300 issues an FP64 instruction every 76 cycles per warp scheduler, so FP64 work that every thread or every block
// repeats costs more than the vectors' traffic on small particles. Hence:
//   - sums over a warp are taken in 64-bit fixed point relative to the warp's largest value: 32 values rounded to a unit of
//     2^-57 to 2^-56 of it, so below 2^-52 of it together and as often up as down (5 FP64 additions: 5 * 2^-53 of the sum);
//     54 integer instructions a sum against 380 cycles;
//   - a kernel's scalar coefficients are converted to double-float once per block by one warp (Coefs), not by every
//     thread;
//   - the scalar steps are not launches of their own: the last block to finish (last_block) sums the partial sums in a
//     fixed order and updates the state.
// Measured: mixed QMR_CS at grid 128^3, 2 RHS 207 -> 182 us an iteration; FP64 QMR_CS at 32^3 85 -> 67 us; adjoint solve
// of a 32^3 cube 31.5 -> 23.8 ms (the scalar kernels alone took 29 us of an iteration, the square root, division and
// complex division chain of the second one 15).
#pragma once

#include "common.cuh"
#include "fft_lines2.cuh"

namespace adda {

// ---------------------------------------------------------------------------------------------------------------
// sums

constexpr int SUM_TOP = 57; // 32 values below 2^57

// key of |v| whose largest over the warp fixes the exponent, and v in fixed point for that exponent
__device__ __forceinline__ int sum_key(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ bool sum_finite(double, int key) { return key < 0x7ff00000; }
__device__ __forceinline__ int sum_emax(double, int key) { return max(1, key >> 20); }
__device__ __forceinline__ int sum_exp(double, int emax) { return emax - 1075 - (SUM_TOP - 53); }
__device__ __forceinline__ long long sum_fx(double v, int emax)
{
	const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff, sh = emax - max(ex, 1);
	long long m = ((long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(v);
	// rounded: cutting off would take up to 31 units off a sum of squares
	m = sh > 62 ? 0 : (((m << (SUM_TOP - 52)) >> sh) + 1) >> 1;
	return hi < 0 ? -m : m;
}
__device__ __forceinline__ int sum_key(DF v) { return __float_as_int(v.h) & 0x7fffffff; }
__device__ __forceinline__ bool sum_finite(DF, int key) { return key < 0x7f800000; }
__device__ __forceinline__ int sum_emax(DF, int key) { return max(1, key >> 23); }
__device__ __forceinline__ int sum_exp(DF, int emax) { return emax - 150 - (SUM_TOP - 24); }
__device__ __forceinline__ long long sum_fx(float v, int emax)
{
	const int b = __float_as_int(v), ex = (b >> 23) & 0xff, sh = emax - max(ex, 1);
	const long long m = (long long)((b & 0x7fffff) | (ex ? 0x800000 : 0)) << (SUM_TOP - 24);
	// cut off: only below 2^-33 of the warp's largest value, or in a double-float's low part, which has either sign; a
	// double-float itself ends at 2^-48
	const long long q = sh > 62 ? 0 : m >> sh;
	return b < 0 ? -q : q;
}
__device__ __forceinline__ long long sum_fx(DF v, int emax) { return sum_fx(v.h, emax) + sum_fx(v.l, emax); }

// sum over a full warp (lane 0); a non-finite value makes it the plain FP64 sum (infinity or NaN)
template <typename T> __device__ __forceinline__ double warp_total(T v)
{
	const int key = __reduce_max_sync(0xffffffffu, sum_key(v));
	if (!sum_finite(v, key)) {
		double s = acc_val(v);
		for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
		return s;
	}
	const int emax = sum_emax(v, key);
	long long q = sum_fx(v, emax);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) q += __shfl_down_sync(0xffffffffu, q, o);
	return fx_to_double(q, sum_exp(v, emax));
}

// sums of NV values over the block; out is valid in thread 0. Every thread calls it (a full block of whole warps).
template <int NV, typename T> __device__ __forceinline__ void block_totals(const T *v, double *out)
{
	__shared__ double sh[NV][32];
	__shared__ double tot[NV];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
	__syncthreads();
#pragma unroll
	for (int j = 0; j < NV; j++) {
		const double s = warp_total(v[j]);
		if (lane == 0) sh[j][wid] = s;
	}
	__syncthreads();
	for (int j = wid; j < NV; j += nw) {
		const double s = warp_total(lane < nw ? sh[j][lane] : 0.0);
		if (lane == 0) tot[j] = s;
	}
	__syncthreads();
#pragma unroll
	for (int j = 0; j < NV; j++) out[j] = tot[j];
}

// whether this block is the last of nblk to get here (cnt: a counter at zero, left at zero); every thread calls it after
// the block's partial sums are written by thread 0
__device__ __forceinline__ bool last_block(unsigned *cnt, unsigned nblk)
{
	__shared__ int last;
	if (threadIdx.x == 0) {
		__threadfence();
		last = atomicAdd(cnt, 1u) == nblk - 1;
		if (last) {
			*cnt = 0;
			__threadfence();
		}
	}
	__syncthreads();
	return last != 0;
}

// sums of the nblk partial sums of RHS r, 4 doubles each (fixed order); valid in thread 0
template <int NV> __device__ __forceinline__ void sum_parts(const double *part, size_t nblk, int r, double *out)
{
	double v[NV];
#pragma unroll
	for (int j = 0; j < NV; j++) v[j] = 0;
	for (size_t b = threadIdx.x; b < nblk; b += blockDim.x)
#pragma unroll
		for (int j = 0; j < NV; j++) v[j] += __ldcg(part + ((size_t)r * nblk + b) * 4 + j);
	block_totals<NV>(v, out);
}

// ---------------------------------------------------------------------------------------------------------------
// scalars of a right-hand side

struct RhsState {
	double inprodR, inprodRp1, epsB, resid_scale;
	int niter, counter, done, status, half, mc, maxiter, x0zero;
	int it0;  // niter when the current Krylov run started (role parity of the swapped QMR_CS / CSYM buffers)
	double prev_err; // last reported relative residual (ProgressReport's prev_err, kept in checkpoints)
	int full; // BiCGStab: no half-step exit
	// QMR_CS
	double c_old, c_new, om_old, om_new;
	double2 beta, tautilda, s_old, s_new, alpha, theta, eta, zetat;
	// BiCGStab, BiCG_CS (ro, balpha), CGNR (real parts of ro, balpha)
	double2 ro_old, ro_new, omega, balpha;
	// CSYM: beta_(k+1) = |w| (real); tau, c, s, theta, eta share the QMR_CS fields, gamma is kept in zetat
	double cs_beta;
	// QMR_CS_2: ro_k, theta_(k-1), c_(k-1); eps_(k-1), eta_(k-1), beta_k; delta_k = v_k.v_k
	double q2_ro, q2_theta, q2_c;
	double2 q2_eps, q2_eta, q2_beta, q2_delta;
	// BCGS2: rho_0, rho_1, alpha; the convex-combination coefficients y0[1], y0[2]
	double2 b2_rho0, b2_rho1, b2_alpha, b2_y1, b2_y2;
	// coefficients for the vector kernels
	double2 k0, k1, k2, k3, kib, kr;
	double d0;
	double temp; // |b|^2
};

__device__ __forceinline__ double2 dc(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ double2 dmul(double2 a, double2 b) { return dc(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 dadd(double2 a, double2 b) { return dc(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 dsub(double2 a, double2 b) { return dc(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 dscal(double2 a, double s) { return dc(a.x * s, a.y * s); }
__device__ __forceinline__ double2 dneg(double2 a) { return dc(-a.x, -a.y); }
__device__ __forceinline__ double2 dconj(double2 a) { return dc(a.x, -a.y); }
__device__ __forceinline__ double dabs(double2 a) { return hypot(a.x, a.y); }
__device__ __forceinline__ double2 ddiv(double2 a, double2 b)
{
	// a/b with scaling against overflow (Smith's method)
	if (fabs(b.x) >= fabs(b.y)) {
		const double r = b.y / b.x, d = b.x + b.y * r;
		return dc((a.x + a.y * r) / d, (a.y - a.x * r) / d);
	}
	const double r = b.x / b.y, d = b.x * r + b.y;
	return dc((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}
__device__ __forceinline__ double2 dinv(double2 b) { return ddiv(dc(1, 0), b); }
__device__ __forceinline__ double2 dsqrt(double2 z)
{
	const double a = z.x, b = z.y;
	const double t = sqrt(0.5 * (hypot(a, b) + fabs(a)));
	if (t == 0) return dc(0, 0);
	if (a >= 0) return dc(t, b / (2 * t));
	return dc(fabs(b) / (2 * t), copysign(t, b));
}

// ---------------------------------------------------------------------------------------------------------------
// scalar steps: one thread, on the sums of the kernel before

// QMR_CS after v.Av (iterative.c:956-982)
__device__ __forceinline__ void qmr_after_matvec(RhsState &S, int *done, const double *s)
{
	if (S.om_new * S.om_new > 1e10) { // 1/omega^2 < 1e-10, iterative.c:958-960
		S.status = ADDA_GB300_EBREAKDOWN;
		S.done = 1;
		*done = 1;
		return;
	}
	const double2 alpha = dc(s[1], s[2]);
	S.alpha = alpha;
	S.theta = dscal(dmul(dconj(S.s_old), S.beta), S.om_old);
	S.eta = dadd(dscal(S.beta, S.c_old * S.c_new * S.om_old), dscal(dmul(alpha, dconj(S.s_new)), S.om_new));
	S.zetat = dsub(dscal(alpha, S.c_new * S.om_new), dscal(dmul(S.s_new, S.beta), S.c_old * S.om_old));
	S.k0 = (S.niter == 1) ? dc(0, 0) : dc(-S.beta.x, -S.beta.y);
	S.k1 = dc(-alpha.x, -alpha.y);
	S.om_old = S.om_new;
}

// QMR_CS after v~ (sums re^2, im^2, re*im; iterative.c:986-1012). With z = v~.v~ and h = |z|: beta = sqrt(z),
// |beta| = sqrt(h), 1/beta = conj(beta)/h; zeta = zetat*(zabs/zt), 1/zeta = conj(zetat)/(zt*zabs). One warp: an FP64
// square root or division is ten dependent instructions of 76 cycles, so the lanes take the independent ones together
// (two rounds of roots, one of divisions). s valid in lane 0.
__device__ __forceinline__ void qmr_after_v1(RhsState &S, const double *s)
{
	const int lane = threadIdx.x & 31;
	const double s0 = __shfl_sync(0xffffffffu, s[0], 0), s1 = __shfl_sync(0xffffffffu, s[1], 0),
				 s2 = __shfl_sync(0xffffffffu, s[2], 0);
	const double nrm = s0 + s1, za = s0 - s1, zb = 2 * s2;
	const double2 zetat = S.zetat;
	// h without over- or underflow: (za, zb) scaled by a power of two
	const int ex = max(1, (max(__double2hiint(za) & 0x7fffffff, __double2hiint(zb) & 0x7fffffff)) >> 20);
	const double dn = __hiloint2double((2046 - min(ex, 2045)) << 20, 0), up = __hiloint2double(min(ex, 2045) << 20, 0);
	const double zs = za * dn, zt_ = zb * dn;
	const double zt2 = zetat.x * zetat.x + zetat.y * zetat.y;
	const double r1 = sqrt(lane == 0 ? zs * zs + zt_ * zt_ : lane == 1 ? zt2 + nrm : lane == 2 ? zt2 : nrm);
	const double h = __shfl_sync(0xffffffffu, r1, 0) * up, zabs = __shfl_sync(0xffffffffu, r1, 1),
				 zt = __shfl_sync(0xffffffffu, r1, 2), snrm = __shfl_sync(0xffffffffu, r1, 3);
	const double r2 = sqrt(lane == 0 ? 0.5 * (h + fabs(za)) : h);
	const double t = __shfl_sync(0xffffffffu, r2, 0), sh = __shfl_sync(0xffffffffu, r2, 1);
	const bool tiny = zt < 1e-40;
	const double num = lane == 0 ? zb : lane == 1 ? snrm : lane == 4 ? zt : lane == 5 ? zt * sh : 1.0;
	const double den = lane == 0 ? 2 * t : lane == 1 ? sh : lane == 2 ? h : lane == 3 ? (tiny ? zabs : zt * zabs)
		: lane == 4 ? zabs : zabs * snrm;
	const double q = num / den;
	const double u = t == 0 ? 0 : __shfl_sync(0xffffffffu, q, 0), om_new = __shfl_sync(0xffffffffu, q, 1),
				 hi = __shfl_sync(0xffffffffu, q, 2), zi = __shfl_sync(0xffffffffu, q, 3), c_new = __shfl_sync(0xffffffffu, q, 4),
				 co = __shfl_sync(0xffffffffu, q, 5); // c_new / om_new
	if (lane) return;
	const double2 beta = za >= 0 ? dc(t, u) : dc(fabs(u), copysign(t, zb));
	const double2 t4 = tiny ? dc(zi, 0) : dc(zetat.x * zi, -zetat.y * zi); // 1/zeta
	const double2 s_new = dscal(dmul(beta, t4), om_new);
	const double2 tau = S.tautilda, tt = dmul(dneg(s_new), tau);
	const int it = S.niter;
	S.k0 = it <= 2 ? dc(0, 0) : dmul(dneg(S.theta), t4);
	S.k1 = it == 1 ? dc(0, 0) : dmul(dneg(S.eta), t4);
	S.k2 = t4;
	S.k3 = dscal(tau, c_new);
	S.kib = dc(beta.x * hi, -beta.y * hi);
	S.kr = dscal(tt, co);
	S.d0 = s_new.x * s_new.x + s_new.y * s_new.y;
	S.c_old = S.c_new;
	S.c_new = c_new;
	S.s_old = S.s_new;
	S.s_new = s_new;
	S.beta = beta;
	S.om_new = om_new;
	S.tautilda = tt;
}

// BiCGStab: alpha = ro_new / (v.r~*) (iterative.c:694-698)
__device__ __forceinline__ void bs_after_v(RhsState &S, int *done, const double *s)
{
	const double2 t = dc(s[1], s[2]);
	if (dabs(t) / dabs(S.ro_new) < 1e-10) { // iterative.c:695-697
		S.status = ADDA_GB300_EBREAKDOWN;
		S.done = 1;
		*done = 1;
		return;
	}
	S.balpha = ddiv(S.ro_new, t);
	S.k0 = dc(-S.balpha.x, -S.balpha.y);
}
// BiCGStab: the half step's residual (iterative.c:703-707)
__device__ __forceinline__ void bs_after_s(RhsState &S, const double *s)
{
	S.inprodRp1 = s[0];
	S.half = (S.inprodRp1 < S.epsB && !S.full) ? 1 : 0; // converged at the half step
}
// BiCGStab: omega = s.t* / |t|^2
__device__ __forceinline__ void bs_after_t(RhsState &S, const double *s)
{
	if (!S.half) S.omega = dscal(dc(s[1], s[2]), 1 / s[0]);
}

// ProgressReport (iterative.c:282-306) + loop condition (iterative.c:1467); s[0] = |r|^2 unless half
// mode 0: |r|^2 from the sums; 1: BiCGStab (also the next ro, half-step exit); 2: inprodRp1 already set by the
// method's scalar step (CSYM's |tau|^2)
__device__ __forceinline__ void progress(RhsState &S, int *done, const double *s, double *hist, int hist_cap, int mode)
{
	const bool bcgs = mode == 1;
	if (!S.half && mode != 2) S.inprodRp1 = s[0];
	if (bcgs && !S.half) S.ro_old = S.ro_new; // the next bs_s0 sums the r.r~* partials of bs_v3 itself
	if (S.inprodRp1 <= S.inprodR) {
		S.inprodR = S.inprodRp1;
		S.counter = 0;
	}
	else S.counter++;
	S.prev_err = sqrt(S.resid_scale * S.inprodRp1);
	if (S.niter < hist_cap) hist[S.niter] = S.prev_err;
	S.niter++;
	S.done = !(S.inprodR > S.epsB && S.niter <= S.maxiter && S.counter <= S.mc);
	*done = S.done;
}

// the scalar step after a matvec, in the last block of its gather kernel (MvEpi::tail)
enum MvTail { TAIL_NONE = 0, TAIL_QMR = 1, TAIL_BS_V = 2, TAIL_BS_T = 3 };
static __device__ __noinline__ void matvec_tail(int tail, RhsState *st, int *done, const double *part, size_t nblk, int r)
{
	double s[3];
	sum_parts<3>(part, nblk, r, s);
	if (threadIdx.x) return;
	RhsState &S = st[r];
	if (tail == TAIL_QMR) qmr_after_matvec(S, done + r, s);
	else if (tail == TAIL_BS_V) bs_after_v(S, done + r, s);
	else bs_after_t(S, s);
}

} // namespace adda
