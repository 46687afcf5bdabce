// matvec_lines2.cuh - the matvec's stages (K1, K2a, K2b, K2c, K3 of matvec_kernels.cuh) on the two-pass transforms of
// fft_lines2.cuh: the FP64 matvec in 64-bit fixed point where all three axes have plans for it (use_fx), and the FP32
// matvec of axis lengths without compile-time kernels. Data flow, buffers and their layouts are the same (fixed point: 16-byte complex integers in the place of
// double2).
//
// Fixed point: the data between two kernels are integers with an exponent per producing block (FxExp below), so that
// no kernel converts to or from floating point but K1 (S.x) and K3 (S.X). A consumer shifts what it loads to one common
// exponent, the one that puts the largest value of its input just below 2^FX_TOP; the largest value comes from the
// bits OR-ed together by the producers, not from a worst case, so the growth of a transform costs no bits.
//
// Measured (one matvec): FP64 at grid 256^3, 2 RHS 19.21 ms with FP64 instructions (97 % of the FP64 pipe's rate) ->
// 4.95 ms; FP32 at 192x154x112, 8 RHS 1.409 -> 0.82 ms, at 96^3 with per-dipole polarisabilities, 2 RHS 0.154 -> 0.081
// ms, at 32^3, 1 RHS 36 -> 20.7 us (against the multi-pass transforms in shared memory with a run-time plan and plain
// launches). Error against 64 bits unchanged (FP64 1.6e-16).
// The fixed-point kernels have 128 registers and 14-15 warps an SM, issue on 19-38 % of the cycles and wait for instruction
// fetch (no instruction 2.0-2.3 per issue), global loads and, in the z transforms, the barrier between the passes. ptxas
// reports 520 to 1480 bytes of spill stores for them, over the butterflies of all radices up to 16 that one kernel holds; of
// the instructions a launch executes 0.04 to 0.9 % are spills.
#pragma once

#include "fft_lines2.cuh"
#include "matvec_kernels.cuh"

namespace adda {
namespace mv {

// exponents of the fixed-point data (value = integer * 2^e); "top": |value| < 2^top
struct FxExp {
	int *ex;    // after K1: [R][bZ][ny1] e of a K1 block (W1 y-lines, all kx and components)
	int *ez;    // after K2a: [R][gX][3][ny2] e of a K2a block (W2 y-lines, all kz)
	int *ezr;   // the same of the reflected transform (particle near a substrate)
	int *ey;    // after K2b: [R][gX][gZ] e of a column (all y and components)
	int *ex2;   // after K2c: [R][gX][3][ny2] e of a K2c block
	int *topx;  // [R][ny2] top of all K1 blocks of W2 y-lines; K3 puts it back to FX_LOW for the next matvec
	int *topz;  // [R][gX] top of all K2a blocks of a kx (of both transforms)
	int *topy;  // [R][gX] top of all columns of a kx
	int *topx2; // [R] top of all K2c blocks
	const fx2 *D;  // interaction matrix, components scaled to 2^60 per row, as split halves (see fx_split)
	const int *eD; // [gX][DsZ] exponents of its rows
	const fx2 *Rm; // reflected interaction, likewise
	const int *eR; // [gX][gZ]
	int ny1, ny2;
};

template <class A> struct Lines2 {
	Plan2 px, py, pz;
	const typename A::Tw *tx, *tz; // W_n^(j*q) at [q*r2 + j] (fixed point: times 2^(64 - shift))
	const typename A::Tw *ty, *tyi; // the same of the y axis, and at [j*r1 + q] for its inverse transform
	int shx, shy, shz;
	FxExp f;
};

// the largest of v over the block, in every thread (s: one shared int, holding FX_LOW before the call's first barrier)
__device__ __forceinline__ int block_max(int v, int *s)
{
	v = __reduce_max_sync(0xffffffffu, v);
	if ((threadIdx.x & 31) == 0) atomicMax(s, v);
	__syncthreads();
	return *s;
}
// OR over the block, in every thread (s: one shared word, zero before the call's first barrier)
__device__ __forceinline__ unsigned block_or(unsigned v, unsigned *s)
{
	v = __reduce_or_sync(0xffffffffu, v);
	if ((threadIdx.x & 31) == 0) atomicOr(s, v);
	__syncthreads();
	return *s;
}
// cached in L2 only; streaming (Xf, see XF_LD)
__device__ __forceinline__ float2 ld_cg(const float2 *p) { return __ldcg(p); }
__device__ __forceinline__ fx2 ld_cg(const fx2 *p)
{
	const longlong2 v = __ldcg(reinterpret_cast<const longlong2 *>(p));
	return fx2{v.x, v.y};
}
__device__ __forceinline__ float2 ld_cs(const float2 *p) { return __ldcs(p); }
__device__ __forceinline__ fx2 ld_cs(const fx2 *p)
{
	const longlong2 v = __ldcs(reinterpret_cast<const longlong2 *>(p));
	return fx2{v.x, v.y};
}
__device__ __forceinline__ void st_cs(float2 *p, float2 v) { __stcs(p, v); }
__device__ __forceinline__ void st_cs(fx2 *p, fx2 v) { __stcs(reinterpret_cast<longlong2 *>(p), make_longlong2(v.x, v.y)); }
// elements of the dipole tile's type (K1's input, K3's output): complex float or double
template <class A> using TileC = typename CxT<typename A::T>::type;

// K1: S.x of W x-lines (one z) into a tile, then the x transform of its 3W lines
template <class A, typename V, int W, int W2, int RC>
__global__ void __launch_bounds__(32 * ((3 * W * radix_max(RC) + 31) / 32), A::FX && RC == RC_SMALL ? 512 / (3 * W * RADIX_MAX) : 1)
	l2_scatter_x(MvP<typename A::T, V> p, Lines2<A> q)
{
	chain_entry(p.early);
	typedef typename A::C C;
	typedef TileC<A> TC;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	if (rhs_done(p, blockIdx.z)) return; // blockIdx.z = RHS
	__shared__ int smax;
	__shared__ unsigned sor;
	constexpr int NL = 3 * W, LS = tile_ls(3 * W);
	TC *a = reinterpret_cast<TC *>(smem_raw); // bX x LS
	C *xb = reinterpret_cast<C *>(smem_raw + (((size_t)p.bX * LS * sizeof(TC) + 15) & ~(size_t)15));
	const int r = blockIdx.z, z = blockIdx.y, y0 = blockIdx.x * W;
	const size_t lq = (size_t)(r / p.rpp); // the lattice of RHS r's particle
	const uint32_t *lstart = p.line_start + lq * ((size_t)p.bZ * p.bY + 1), *lxy = p.xy + lq * p.lat_stride;
	const uint8_t *lmat = p.mat + lq * p.lat_stride;
	const int wy = min(W, p.bY - y0);
	for (int t = threadIdx.x; t < p.bX * LS; t += blockDim.x) a[t] = cx<TC>(0, 0);
	if constexpr (A::FX) {
		if (threadIdx.x == 0) {
			smax = 0;
			sor = 0;
		}
		// the tops that later kernels of this matvec collect start below everything
		const int nb = gridDim.x * gridDim.y, b = blockIdx.y * gridDim.x + blockIdx.x;
		for (int t = b * blockDim.x + threadIdx.x; t < p.gX; t += nb * blockDim.x) {
			q.f.topz[(size_t)r * p.gX + t] = FX_LOW;
			q.f.topy[(size_t)r * p.gX + t] = FX_LOW;
			if (t == 0) q.f.topx2[r] = FX_LOW;
		}
	}
	__syncthreads();
	const size_t line = (size_t)z * p.bY + y0;
	const uint32_t i0 = lstart[line], i1 = lstart[line + wy];
	const V *arg = p.arg + (size_t)r * p.N * 3;
	int hmax = 0;
#pragma unroll 2
	for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
		const uint32_t xy = lxy[i];
		const int x = xy & 0xffff, y = xy >> 16;
		const uint8_t m = lmat[i];
#pragma unroll
		for (int comp = 0; comp < 3; comp++) {
			TC v = cvt<TC>(arg[(size_t)i * 3 + comp]);
			if (p.her) v = cconj(v);
			v = cmul(ccs_of(p.ccs, p.per_dip, p.nmat, p.N, r, i, m, comp), v);
			a[x * LS + comp * W + (y - y0)] = v;
			if constexpr (A::FX)
				hmax = max(hmax, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
		}
	}
	int emax = 0;
	if constexpr (A::FX) {
		hmax = block_max(hmax, &smax);
		emax = max(1, hmax >> 20);
	}
	else __syncthreads();
	const int l = threadIdx.x % NL, j = threadIdx.x / NL, comp = l / W, yy = l - comp * W;
	const int r1 = q.px.r1, r2 = q.px.r2, ks = xch_ks(NL, r2), bX = p.bX;
	if (j < r2) {
		auto ld = [&](int, int i) {
			if (i >= bX) return cx<C>(0, 0);
			const TC v = a[i * LS + l];
			if constexpr (A::FX) return fx2{fx_from_double(v.x, emax), fx_from_double(v.y, emax)};
			else return v;
		};
		ADDA_RADIX_SWITCH(r1, (pass_first<A, RR, false, true>(ld, xb, ks, j * NL + l, j, r2, q.tx, q.shx)))
	}
	__syncthreads();
	const size_t plane = (size_t)p.bZ * p.bY;
	unsigned acc = 0;
	if (j < r1 && yy < wy) {
		C *dst = reinterpret_cast<C *>(p.Xf) + (size_t)r * p.gX * 3 * plane + (size_t)comp * plane + (size_t)z * p.bY + y0 +
			yy;
		auto ld = [&](int t) { return xb[j * ks + t * NL + l]; };
		auto st = [&](int, int kx, C v) {
			st_cs(dst + (size_t)kx * 3 * plane, v);
			if constexpr (A::FX) {
				fx_or(acc, v.x);
				fx_or(acc, v.y);
			}
		};
		ADDA_RADIX_SWITCH(r2, (pass_second<A, RR, false, false>(ld, st, j, r1)))
	}
	if constexpr (A::FX) {
		acc = block_or(acc, &sor);
		if (threadIdx.x == 0) {
			const int e = emax - 1075 - (FX_TOP - 53) + q.shx;
			q.f.ex[((size_t)r * p.bZ + z) * q.f.ny1 + blockIdx.x] = e;
			atomicMax(q.f.topx + (size_t)r * q.f.ny2 + y0 / W2, hmax >= 0x7ff00000 ? FX_BAD : e + fx_bits(acc));
		}
	}
}

// K2a (MODE 0), K2c (MODE 1) and K2a of the reflected transform (MODE 2: the inverse sign into TzR): the z
// transform of W y-lines of one (RHS, kx, component)
template <class A, int W, int MODE, int W1, int RC>
__global__ void __launch_bounds__(W * radix_max(RC), A::FX && RC == RC_SMALL ? 512 / (W * RADIX_MAX) : 1) l2_fftz(MvGeom<typename A::T> p, Lines2<A> q)
{
	chain_entry(p.early);
	typedef typename A::C C;
	constexpr bool INV = MODE == 1, SGN = MODE != 0;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	if (rhs_done(p, blockIdx.z)) return; // blockIdx.z = RHS
	__shared__ unsigned sor;
	C *xb = reinterpret_cast<C *>(smem_raw);
	const int r = blockIdx.z, kxl = blockIdx.y / 3, comp = blockIdx.y % 3, kx = p.kx0 + kxl;
	const int y0 = blockIdx.x * W, wy = min(W, p.bY - y0), gZ = p.gZ, bZ = p.bZ;
	const size_t plane = (size_t)bZ * p.bY;
	C *xf = reinterpret_cast<C *>(p.Xf) + (((size_t)r * p.gX + kx) * 3 + comp) * plane + y0;
	C *tz = reinterpret_cast<C *>(MODE == 2 ? p.TzR : p.Tz) + (((size_t)r * p.CK + kxl) * 3 + comp) * (size_t)gZ * p.bY + y0;
	const int l = threadIdx.x % W, j = threadIdx.x / W;
	const bool yok = l < wy;
	const int r1 = q.pz.r1, r2 = q.pz.r2, ks = xch_ks(W, r2);
	int et = 0, top = 0;
	const int *ex = nullptr, *ey = nullptr;
	if constexpr (A::FX) {
		if (threadIdx.x == 0) sor = 0;
		if constexpr (INV) {
			top = q.f.topy[(size_t)r * p.gX + kx];
			ey = q.f.ey + ((size_t)r * p.gX + kx) * gZ;
		}
		else {
			top = q.f.topx[(size_t)r * q.f.ny2 + blockIdx.x];
			ex = q.f.ex + (size_t)r * bZ * q.f.ny1 + (y0 + l) / W1;
		}
		et = top - FX_TOP;
	}
	if (j < r2) {
		auto ld = [&](int, int z) {
			if (!yok || (!INV && z >= bZ)) return cx<C>(0, 0);
			if constexpr (INV) {
				C v = ld_cg(tz + (size_t)z * p.bY + l);
				if constexpr (A::FX) {
					const int d = ey[z] - et;
					v = fx_shift(v, d);
				}
				return v;
			}
			else {
				C v = ld_cs(xf + (size_t)z * p.bY + l);
				if constexpr (A::FX) {
					const int d = ex[(size_t)z * q.f.ny1] - et;
					v = fx_shift(v, d);
				}
				return v;
			}
		};
		ADDA_RADIX_SWITCH(r1, (pass_first<A, RR, SGN, !INV>(ld, xb, ks, j * W + l, j, r2, q.tz, q.shz)))
	}
	__syncthreads();
	unsigned acc = 0;
	if (j < r1 && yok) {
		auto ld = [&](int t) { return xb[j * ks + t * W + l]; };
		auto st = [&](int, int z, C v) {
			if (INV && z >= bZ) return;
			if constexpr (INV) st_cs(xf + (size_t)z * p.bY + l, v);
			else tz[(size_t)z * p.bY + l] = v;
			if constexpr (A::FX) {
				fx_or(acc, v.x);
				fx_or(acc, v.y);
			}
		};
		ADDA_RADIX_SWITCH(r2, (pass_second<A, RR, SGN, INV>(ld, st, j, r1)))
	}
	if constexpr (A::FX) {
		acc = block_or(acc, &sor);
		if (threadIdx.x == 0) {
			const int e = et + q.shz;
			const int t = top >= FX_BAD / 2 ? FX_BAD : e + fx_bits(acc);
			(INV ? q.f.ex2 : MODE == 2 ? q.f.ezr : q.f.ez)[(((size_t)r * p.gX + kx) * 3 + comp) * q.f.ny2 + blockIdx.x] = e;
			atomicMax(INV ? q.f.topx2 + r : q.f.topz + (size_t)r * p.gX + kx, t);
		}
	}
}

// D~.v in fixed point: D's entries as split halves (re low, re high, im low, im high), results r = sum * 2^(k - 64).
// |v| < 2^60.5 and |D| components < 2^60 keep the sums of partial products below 2^63.
__device__ __forceinline__ int4 fx_neg4(int4 a) { return make_int4(-a.x, -a.y, -a.z, -a.w); }
struct FxV {
	int xh, xl, yh, yl;
};
__device__ __forceinline__ FxV fx_vsplit(fx2 v)
{
	FxV s;
	fx_split(v.x, s.xh, s.xl);
	fx_split(v.y, s.yh, s.yl);
	return s;
}
__device__ __forceinline__ long long fx_take(long long hi, long long t, int k)
{
	// (hi*2^64 + t*2^32 ...) >> (64 - k): hi + (t >> 32) and the k upper bits of t's low word
	hi += t >> 32;
	const unsigned lo = (unsigned)t;
	const unsigned w0 = __funnelshift_l(lo, (unsigned)hi, k), w1 = __funnelshift_l((unsigned)hi, (unsigned)(hi >> 32), k);
	return ((long long)(int)w1 << 32) | w0;
}
__device__ __forceinline__ fx2 fx_dot3(int4 a, int4 b, int4 c, const FxV &u, const FxV &v, const FxV &w, int k)
{
	long long t = 0, s = 0, hr = 0, hi = 0;
#define ADDA_FX_TERM(m, q)                                                                                           \
	t = (long long)q.xh * m.x + t;                                                                                  \
	t = (long long)q.xl * m.y + t;                                                                                  \
	t = (long long)q.yh * -m.z + t;                                                                                 \
	t = (long long)q.yl * -m.w + t;                                                                                 \
	s = (long long)q.xh * m.z + s;                                                                                  \
	s = (long long)q.xl * m.w + s;                                                                                  \
	s = (long long)q.yh * m.x + s;                                                                                  \
	s = (long long)q.yl * m.y + s;                                                                                  \
	hr = (long long)q.xh * m.y + hr;                                                                                \
	hr = (long long)q.yh * -m.w + hr;                                                                               \
	hi = (long long)q.xh * m.w + hi;                                                                                \
	hi = (long long)q.yh * m.y + hi;
	ADDA_FX_TERM(a, u)
	ADDA_FX_TERM(b, v)
	ADDA_FX_TERM(c, w)
#undef ADDA_FX_TERM
	return fx2{fx_take(hr, t, k), fx_take(hi, s, k)};
}

// K2b: y transforms, D product (matvec.c:271-305 incl. the reduced-FFT signs) and inverse y transforms of G columns
// (kz, RHS), RHS fastest, with 3*P threads each (P = max(r1, r2)): one group of P per component line, which lives in a
// shared slot. Pass 1 leaves Y[q][j] in row q; from there thread q works in its own row (second pass, first inverse
// pass), and the second inverse pass reads columns. The D product takes the three components of row q's elements
// c, c+3, ... (c the thread's component). Rows are r2|1 long: every phase is free of bank conflicts.
// SURF (particle near a substrate): three more slots hold the lines of TzR; the product adds R~ times their spectra
// (M21 = M12, M31 = -M13, M32 = -M23, cReflMatrVec cmplx.h:391-401; R reduced in y only).
template <class A, int W2, int RC, bool SURF>
__global__ void __launch_bounds__(A::FX ? 128 : 384, RC == RC_BIG ? (A::FX ? 2 : 1) : (A::FX ? 4 : 2))
	l2_fft_y(MvGeom<typename A::T> p, Lines2<A> q, int G, int P)
{
	chain_entry(p.early);
	typedef typename A::C C;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned sor[3][8];
	if (all_done(p)) return;
	const int gc = threadIdx.x / P, g = gc / 3, c = gc - 3 * g, j = threadIdx.x - gc * P;
	const int r1 = q.py.r1, r2 = q.py.r2, pitch = r2 | 1, slot = r1 * pitch;
	const int unit = blockIdx.x * G + g;
	const int r = unit % p.R, kz = unit / p.R;
	const bool live = g < G && kz < p.gZ && !rhs_done(p, r);
	const int kxl = blockIdx.y, kx = p.kx0 + kxl, bY = p.bY, gY = p.gY;
	constexpr int NS = SURF ? 2 : 1; // sets of three slots
	C *buf = reinterpret_cast<C *>(smem_raw) + (size_t)g * 3 * NS * slot; // the column's slots
	C *line = buf + c * slot;                                        // the thread's own line
	const size_t at = ((((size_t)r * p.CK + kxl) * 3 + c) * p.gZ + kz) * (size_t)bY;
	C *col = reinterpret_cast<C *>(p.Tz) + at;
	int et = 0, top = 0;
	size_t eat = 0;
	if constexpr (A::FX) {
		if (threadIdx.x < 24) sor[threadIdx.x / 8][threadIdx.x % 8] = 0;
		if (live) {
			top = q.f.topz[(size_t)r * p.gX + kx];
			eat = (((size_t)r * p.gX + kx) * 3 + c) * q.f.ny2;
		}
		et = top - FX_TOP;
	}
	if (live && j < r2) {
#pragma unroll 1
		for (int h = 0; h < NS; h++) {
			const C *src = h ? reinterpret_cast<const C *>(p.TzR) + at : col;
			const int *ez = (h ? q.f.ezr : q.f.ez) + eat;
			auto ld = [&](int, int y) {
				if (y >= bY) return cx<C>(0, 0);
				C v = ld_cg(src + y);
				if constexpr (A::FX) {
					const int d = ez[y / W2] - et;
					v = fx_shift(v, d);
				}
				return v;
			};
			ADDA_RADIX_SWITCH(r1, (pass_first<A, RR, false, true>(ld, line + 3 * h * slot, pitch, j, j, r2, q.ty, q.shy)))
		}
	}
	__syncthreads();
	const bool rz = kz >= p.DsZ;
	const int zz = rz ? p.gZ - kz : kz;
	const bool act = live && j < r1;
	unsigned acc = 0;
	C *own = line + j * pitch;
	if (act) {
#pragma unroll 1
		for (int h = 0; h < NS; h++) {
			C *o = own + 3 * h * slot;
			auto ld = [&](int t) { return o[t]; };
			auto st = [&](int t, int, C v) {
				o[t] = v;
				if constexpr (A::FX) {
					fx_or(acc, v.x);
					fx_or(acc, v.y);
				}
			};
			ADDA_RADIX_SWITCH(r2, (pass_second<A, RR, false, false>(ld, st, j, r1)))
		}
	}
	if constexpr (A::FX)
		if (act) atomicOr(&sor[0][g], acc);
	__syncthreads();
	constexpr int k = 3;
	int eo = 0, ed = 0, shv = 0, dD = 0, dR = 0;
	if constexpr (A::FX) {
		// the components of v are brought just below 2^60: the products leave out the lowest partial product, 2^-60 of
		// the largest v and D; |sum of three| < 3 * 2^60.5 * 2^60.5, so 3 more bits than the upper 64 fit
		shv = fx_bits(sor[0][g & 7]) - 60;
		if (live) ed = q.f.eD[(size_t)kx * p.DsZ + zz];
		if constexpr (SURF)
			if (live) { // the row's two products at the larger of the two exponents
				const int er = q.f.eR[(size_t)kx * p.gZ + kz];
				dD = max(0, er - ed);
				dR = max(0, ed - er);
				ed = max(ed, er);
			}
		eo = et + q.shy + shv + ed + 64 - k;
		acc = 0;
	}
	if (act) {
		C *row = buf + j * pitch;
		const size_t drow = ((size_t)kx * p.DsZ + zz) * p.DsY;
#pragma unroll(A::FX ? 1 : 2)
		for (int t = c; t < r2; t += 3) {
			const int ky = j + r1 * t;
			const bool ry = ky >= p.DsY;
			const int yy = ry ? gY - ky : ky;
			if constexpr (A::FX) {
				const int4 *f = reinterpret_cast<const int4 *>(q.f.D) + (drow + yy) * 6;
				int4 m0 = __ldg(f), m1 = __ldg(f + 1), m2 = __ldg(f + 2), m3 = __ldg(f + 3), m4 = __ldg(f + 4),
					 m5 = __ldg(f + 5);
				if (ry) m1 = fx_neg4(m1);
				if (ry != rz) m4 = fx_neg4(m4);
				if (rz) m2 = fx_neg4(m2);
				fx2 w0 = row[t], w1 = row[slot + t], w2 = row[2 * slot + t];
				if (shv <= 0) {
					w0 = fx2{w0.x << -shv, w0.y << -shv};
					w1 = fx2{w1.x << -shv, w1.y << -shv};
					w2 = fx2{w2.x << -shv, w2.y << -shv};
				}
				else {
					w0 = fx_shift(w0, -shv);
					w1 = fx_shift(w1, -shv);
					w2 = fx_shift(w2, -shv);
				}
				const FxV v0 = fx_vsplit(w0), v1 = fx_vsplit(w1), v2 = fx_vsplit(w2);
				fx2 o0 = fx_dot3(m0, m1, m2, v0, v1, v2, k), o1 = fx_dot3(m1, m3, m4, v0, v1, v2, k),
					o2 = fx_dot3(m2, m4, m5, v0, v1, v2, k);
				if constexpr (SURF) {
					const bool qy = ky > gY / 2;
					const int4 *fr = reinterpret_cast<const int4 *>(q.f.Rm) + (((size_t)kx * p.gZ + kz) * p.RsY + (qy ? gY - ky : ky)) * 6;
					m0 = __ldg(fr), m1 = __ldg(fr + 1), m2 = __ldg(fr + 2), m3 = __ldg(fr + 3), m4 = __ldg(fr + 4), m5 = __ldg(fr + 5);
					if (qy) {
						m1 = fx_neg4(m1);
						m4 = fx_neg4(m4);
					}
					const C *ur = row + 3 * slot;
					FxV u[3];
#pragma unroll
					for (int i = 0; i < 3; i++) {
						const fx2 w = ur[i * slot + t];
						u[i] = fx_vsplit(fx_shift(w, -shv));
					}
					const auto add = [&](fx2 a, fx2 b) {
						return cadd(fx_shift(a, -dD), fx_shift(b, -dR));
					};
					o0 = add(o0, fx_dot3(m0, m1, m2, u[0], u[1], u[2], k));
					o1 = add(o1, fx_dot3(m1, m3, m4, u[0], u[1], u[2], k));
					o2 = add(o2, fx_dot3(fx_neg4(m2), fx_neg4(m4), m5, u[0], u[1], u[2], k));
				}
				fx_or(acc, o0.x);
				fx_or(acc, o0.y);
				fx_or(acc, o1.x);
				fx_or(acc, o1.y);
				fx_or(acc, o2.x);
				fx_or(acc, o2.y);
				row[t] = o0;
				row[slot + t] = o1;
				row[2 * slot + t] = o2;
			}
			else {
				const float4 *f = reinterpret_cast<const float4 *>(p.D) + (drow + yy) * 3;
				const float4 d0 = __ldg(f), d1 = __ldg(f + 1), d2 = __ldg(f + 2);
				C m0 = make_float2(d0.x, d0.y), m1 = make_float2(d0.z, d0.w), m2 = make_float2(d1.x, d1.y);
				C m3 = make_float2(d1.z, d1.w), m4 = make_float2(d2.x, d2.y), m5 = make_float2(d2.z, d2.w);
				if (ry) m1 = cneg(m1);
				if (ry != rz) m4 = cneg(m4);
				if (rz) m2 = cneg(m2);
				const C v0 = row[t], v1 = row[slot + t], v2 = row[2 * slot + t];
				C o0 = cfma(m0, v0, cfma(m1, v1, cmul(m2, v2))), o1 = cfma(m1, v0, cfma(m3, v1, cmul(m4, v2))),
				  o2 = cfma(m2, v0, cfma(m4, v1, cmul(m5, v2)));
				if constexpr (SURF) {
					const bool qy = ky > gY / 2;
					const float4 *fr = reinterpret_cast<const float4 *>(p.Rm) + (((size_t)kx * p.gZ + kz) * p.RsY + (qy ? gY - ky : ky)) * 3;
					const float4 e0 = __ldg(fr), e1 = __ldg(fr + 1), e2 = __ldg(fr + 2);
					m0 = make_float2(e0.x, e0.y), m1 = make_float2(e0.z, e0.w), m2 = make_float2(e1.x, e1.y);
					m3 = make_float2(e1.z, e1.w), m4 = make_float2(e2.x, e2.y), m5 = make_float2(e2.z, e2.w);
					if (qy) {
						m1 = cneg(m1);
						m4 = cneg(m4);
					}
					const C *ur = row + 3 * slot;
					const C u0 = ur[t], u1 = ur[slot + t], u2 = ur[2 * slot + t];
					o0 = cfma(m0, u0, cfma(m1, u1, cfma(m2, u2, o0)));
					o1 = cfma(m1, u0, cfma(m3, u1, cfma(m4, u2, o1)));
					o2 = cfma(cneg(m2), u0, cfma(cneg(m4), u1, cfma(m5, u2, o2)));
				}
				row[t] = o0;
				row[slot + t] = o1;
				row[2 * slot + t] = o2;
			}
		}
	}
	if constexpr (A::FX)
		if (act) atomicOr(&sor[1][g], acc);
	__syncthreads();
	int sh = 0;
	if constexpr (A::FX) {
		sh = max(0, fx_bits(sor[1][g & 7]) - FX_TOP);
		eo += sh + q.shy;
		acc = 0;
	}
	// the inverse transform has the radices in the other order: thread q's row holds elements q + r1*t
	if (act) {
		auto ld = [&](int t, int) {
			C v = own[t];
			if constexpr (A::FX)
				if (sh) v = fx2{fx_rshift(v.x, sh), fx_rshift(v.y, sh)};
			return v;
		};
		ADDA_RADIX_SWITCH(r2, (pass_first<A, RR, true, false>(ld, own, 1, 0, j, r1, q.tyi, q.shy)))
	}
	__syncthreads();
	if (live && j < r2) {
		const C *cb = line + j;
		auto ld = [&](int t) { return cb[t * pitch]; };
		auto st = [&](int, int y, C v) {
			if (y >= bY) return;
			col[y] = v;
			if constexpr (A::FX) {
				fx_or(acc, v.x);
				fx_or(acc, v.y);
			}
		};
		ADDA_RADIX_SWITCH(r1, (pass_second<A, RR, true, true>(ld, st, j, r2)))
	}
	if constexpr (A::FX) {
		if (live && j < r2) atomicOr(&sor[2][g], acc);
		__syncthreads();
		if (live && j == 0 && c == 0) {
			const int t = top >= FX_BAD / 2 || ed >= FX_BAD / 2 ? FX_BAD : eo + fx_bits(sor[2][g]);
			q.f.ey[((size_t)r * p.gX + kx) * p.gZ + kz] = eo;
			atomicMax(q.f.topy + (size_t)r * p.gX + kx, t);
		}
	}
}

// K3: inverse x transform of W y-lines (one z), then y = x + S.X for their dipoles with the epilogue reductions
template <class A, typename V, int W, int W2, int RC>
__global__ void __launch_bounds__(32 * ((3 * W * radix_max(RC) + 31) / 32), A::FX && RC == RC_SMALL ? 512 / (3 * W * RADIX_MAX) : 1)
	l2_gather_x(MvP<typename A::T, V> p, Lines2<A> q, MvEpi e)
{
	chain_entry(p.early);
	typedef typename A::C C;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	if (rhs_done(p, blockIdx.z)) return; // blockIdx.z = RHS
	constexpr int NL = 3 * W, LS = tile_ls(3 * W);
	C *a = reinterpret_cast<C *>(smem_raw); // bX x LS
	C *xb = reinterpret_cast<C *>(smem_raw + (((size_t)p.bX * LS * sizeof(C) + 15) & ~(size_t)15));
	const int r = blockIdx.z, z = blockIdx.y, y0 = blockIdx.x * W;
	const int wy = min(W, p.bY - y0), bX = p.bX;
	const size_t plane = (size_t)p.bZ * p.bY;
	const int l = threadIdx.x % NL, j = threadIdx.x / NL, comp = l / W, yy = l - comp * W;
	const int r1 = q.px.r1, r2 = q.px.r2, ks = xch_ks(NL, r2);
	const bool ok = yy < wy;
	int et = 0, top = 0;
	const int *ex = nullptr;
	if constexpr (A::FX) {
		top = q.f.topx2[r];
		et = top - FX_TOP;
		if (z == 0 && threadIdx.x == 0 && y0 % W2 == 0) q.f.topx[(size_t)r * q.f.ny2 + y0 / W2] = FX_LOW;
		ex = q.f.ex2 + ((size_t)r * p.gX * 3 + comp) * q.f.ny2 + (y0 + yy) / W2;
	}
	if (j < r2) {
		const C *src = reinterpret_cast<const C *>(p.Xf) + (size_t)r * p.gX * 3 * plane + (size_t)comp * plane +
			(size_t)z * p.bY + y0 + yy;
		auto ld = [&](int, int kx) {
			if (!ok) return cx<C>(0, 0);
			C v = ld_cs(src + (size_t)kx * 3 * plane);
			if constexpr (A::FX) {
				const int d = ex[(size_t)kx * 3 * q.f.ny2] - et;
				v = fx_shift(v, d);
			}
			return v;
		};
		ADDA_RADIX_SWITCH(r1, (pass_first<A, RR, true, false>(ld, xb, ks, j * NL + l, j, r2, q.tx, q.shx)))
	}
	__syncthreads();
	const int eo = et + q.shx;
	if (j < r1) {
		auto ld = [&](int t) { return xb[j * ks + t * NL + l]; };
		auto st = [&](int, int x, C v) {
			if (x < bX) a[x * LS + l] = v;
		};
		ADDA_RADIX_SWITCH(r2, (pass_second<A, RR, true, true>(ld, st, j, r1)))
	}
	__syncthreads();
	auto get = [&](int i) {
		const C v = a[i];
		if constexpr (A::FX) {
			if (top >= FX_BAD / 2) return make_double2(__hiloint2double(0x7ff80000, 0), __hiloint2double(0x7ff80000, 0));
			return make_double2(fx_to_double(v.x, eo), fx_to_double(v.y, eo));
		}
		else return v;
	};
	gather_lines<typename A::T, V, W>(p, e, get, LS, r, z, y0, wy, blockDim.x);
}

// ---------------------------------------------------------------------------------------------------------------
// host side

// shared memory of the kernels
template <class A> inline size_t l2_xtile_smem(int bX, const Plan2 &p, int w)
{
	return ((sizeof(TileC<A>) * (size_t)bX * tile_ls(3 * w) + 15) & ~(size_t)15) +
		sizeof(typename A::C) * (size_t)p.r1 * xch_ks(3 * w, p.r2);
}
template <class A> inline size_t l2_z_smem(const Plan2 &p, int w)
{
	return sizeof(typename A::C) * (size_t)p.r1 * xch_ks(w, p.r2);
}
template <class A> inline size_t l2_y_smem(const Plan2 &p, int g, bool surf)
{
	return sizeof(typename A::C) * (size_t)g * (surf ? 6 : 3) * p.r1 * (p.r2 | 1);
}
// the exponent tables inside fx_exps
inline FxExp fx_tables(const adda_gb300_ctx *c, size_t *ints = nullptr)
{
	FxExp f;
	const size_t R = c->Rmax, gX = c->gX;
	f.ny1 = (c->bY + FX_W1 - 1) / FX_W1;
	f.ny2 = (c->bY + FX_W2 - 1) / FX_W2;
	int *at = c->fx_exps;
	f.ex = at;
	at += R * c->bZ * f.ny1;
	f.ez = at;
	at += R * gX * 3 * f.ny2;
	f.ezr = at;
	if (c->surface) at += R * gX * 3 * f.ny2;
	f.ey = at;
	at += R * gX * c->gZ;
	f.ex2 = at;
	at += R * gX * 3 * f.ny2;
	f.topx = at;
	at += R * f.ny2;
	f.topz = at;
	at += R * gX;
	f.topy = at;
	at += R * gX;
	f.topx2 = at;
	at += R;
	if (ints) *ints = (size_t)(at - c->fx_exps);
	f.D = (const fx2 *)c->Dfx;
	f.eD = c->fx_eD;
	f.Rm = (const fx2 *)c->Rfx;
	f.eR = c->fx_eD + (size_t)c->gX * c->DsZ;
	return f;
}
template <class A> inline Lines2<A> make_lines2(const adda_gb300_ctx *c)
{
	Lines2<A> q;
	const Plan2 *p = A::FX ? c->p2x : c->p2;
	q.px = p[0];
	q.py = p[1];
	q.pz = p[2];
	if constexpr (A::FX) {
		q.tx = c->tw2x[0];
		q.ty = c->tw2x[1];
		q.tz = c->tw2x[2];
		q.tyi = c->tw2x[3];
		q.shx = fx_shift(c->gX);
		q.shy = fx_shift(c->gY);
		q.shz = fx_shift(c->gZ);
		q.f = fx_tables(c);
	}
	else {
		q.tx = c->tw2f[0];
		q.ty = c->tw2f[1];
		q.tz = c->tw2f[2];
		q.tyi = c->tw2f[3];
	}
	return q;
}
// once per kernel and device: its code on the device (load), or shared memory up to SMEM_CAP where it wants more than near
// the default limit (48 KB with the static part)
template <auto KERN> inline int l2_opt_in(const adda_gb300_ctx *c, bool load)
{
	static std::atomic<unsigned long long> done[2]{};
	const unsigned long long bit = 1ull << (c->device & 63);
	if (done[load].load(std::memory_order_acquire) & bit) return ADDA_GB300_OK;
	cudaFuncAttributes a;
	if (load) ADDA_CUDA(cudaFuncGetAttributes(&a, KERN));
	else ADDA_CUDA(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_CAP));
	done[load].fetch_or(bit, std::memory_order_release);
	return ADDA_GB300_OK;
}
// launch of a kernel; a grid without blocks (no RHS) only loads and opts it in, at the context's creation (prepare_f64, matvec_setup_f32)
template <auto KERN, typename... Ar>
inline int l2_launch(const adda_gb300_ctx *c, dim3 g, int nt, size_t sm, cudaStream_t st, const Ar &...args)
{
	const bool none = !(g.x && g.z);
	int rc = none ? l2_opt_in<KERN>(c, true) : ADDA_GB300_OK;
	if (!rc && sm > 32 * 1024) rc = l2_opt_in<KERN>(c, false);
	if (rc || none) return rc;
	launch_next(KERN, g, dim3(nt), sm, st, args...);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}
inline int l2_threads(int lines, const Plan2 &p) { return (lines * std::max(p.r1, p.r2) + 31) / 32 * 32; }

// columns per block of the y kernel: as asked for in FP32, 128 threads in fixed point
template <class A> inline int l2_columns(const Plan2 &p, int pairs)
{
	const int t = 3 * std::max(p.r1, p.r2);
	return std::max(1, std::min(A::FX ? 8 : pairs, (A::FX ? 128 : 384) / t));
}

template <class A, int W, int MODE, int W1, int RC>
inline int l2_z(adda_gb300_ctx *c, const MvGeom<typename A::T> &p, int ck, cudaStream_t st)
{
	const Lines2<A> q = make_lines2<A>(c);
	const dim3 g((c->bY + W - 1) / W, 3 * ck, p.R);
	return l2_launch<l2_fftz<A, W, MODE, W1, RC>>(c, g, l2_threads(W, q.pz), l2_z_smem<A>(q.pz, W), st, p, q);
}
template <class A, int W2, int RC>
inline int l2_y(adda_gb300_ctx *c, const MvGeom<typename A::T> &p, int ck, int pairs, cudaStream_t st)
{
	const Lines2<A> q = make_lines2<A>(c);
	// a column near a substrate has twice the lines: half the columns
	const int P = std::max(q.py.r1, q.py.r2), G = l2_columns<A>(q.py, c->surface ? std::max(1, pairs / 2) : pairs);
	const dim3 g((c->gZ * p.R + G - 1) / G, ck);
	const int nt = (3 * G * P + 31) / 32 * 32;
	if (c->surface) return l2_launch<l2_fft_y<A, W2, RC, true>>(c, g, nt, l2_y_smem<A>(q.py, G, true), st, p, q, G, P);
	return l2_launch<l2_fft_y<A, W2, RC, false>>(c, g, nt, l2_y_smem<A>(q.py, G, false), st, p, q, G, P);
}
template <class A, typename V, int W, int W2, int RC>
inline int l2_k1(adda_gb300_ctx *c, const MvP<typename A::T, V> &p, cudaStream_t st)
{
	const Lines2<A> q = make_lines2<A>(c);
	const dim3 g((c->bY + W - 1) / W, c->bZ, p.R);
	return l2_launch<l2_scatter_x<A, V, W, W2, RC>>(c, g, l2_threads(3 * W, q.px), l2_xtile_smem<A>(c->bX, q.px, W), st, p, q);
}
template <class A, typename V, int W, int W2, int RC>
inline int l2_k3(adda_gb300_ctx *c, const MvP<typename A::T, V> &p, const MvEpi &e, cudaStream_t st)
{
	const Lines2<A> q = make_lines2<A>(c);
	const dim3 g((c->bY + W - 1) / W, c->bZ, p.R);
	return l2_launch<l2_gather_x<A, V, W, W2, RC>>(c, g, l2_threads(3 * W, q.px), l2_xtile_smem<A>(c->bX, q.px, W), st, p, q, e);
}

} // namespace mv
} // namespace adda
