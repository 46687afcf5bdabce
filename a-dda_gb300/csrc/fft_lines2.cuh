// fft_lines2.cuh - two-pass transforms of lines whose length is a product of two register radices.
//
// A line of n = r1*r2 elements (radices up to 32 of the prime factors 2, 3, 5, 7, 11, 13) is transformed as: element i = j + r2*t; thread j < r2 does DFT_r1 over t in registers, multiplies
// by W_n^(j*q) and leaves Y[q][j] in shared memory; thread q < r1 does DFT_r2 over j and holds X[q + r1*p]. One
// exchange, whatever the radices; they are run-time numbers (block-uniform switches), so one kernel serves all sizes. Of the
// even lengths up to 512 that fftFit gives, FP32 has a plan for all but 490, fixed point, which has fewer radices above 16
// (radix_built), for all but 242, 286, 294, 308, 330, 338, 364, 378, 390, 392, 396, 420, 440, 462, 468, 484, 486, 490 and 504:
// one axis of those lengths, or above 512, leaves the FP64 matvec to FP64 instructions.
//
// Two arithmetics:
//   Ar32  complex float.
//   ArFx  64-bit fixed point with a common exponent per block of lines, the arithmetic of the FP64 matvec. GB300 issues
//         an FP64 instruction every 76 cycles per warp scheduler (1.68 per clock and SM, measured) but a 32x32+64-bit
//         multiply-add or a 64-bit add every 2, so a complex product costs 30 cycles here against 304 in FP64 and a
//         complex sum 4 against 152.
//         Range: |component| < 2^FX_TOP on entry, so a sum of n terms stays below n*sqrt(2)*2^FX_TOP; the twiddles
//         between the passes carry a factor 2^-fx_shift(n), which keeps the results below 2^62.5 and everything that
//         is multiplied (at most half of a pass's terms; two thirds in a radix-3 butterfly, whose products are real and
//         have room for that) below 2^61.5, the bound of the products. Error: one unit is 2^-56 of the block's largest
//         value on entry and 2^-(56 - fx_shift(n)) after the first pass (2^-54 up to 256 elements, 2^-53 up to 512), where
//         the signal has grown by sqrt(r1), 4 and more there: no more than the rounding of an FP64 transform (1.6e-16 a
//         matvec of a 128^3 sphere, both).
#pragma once

#include "common.cuh"

#include <type_traits>

namespace adda {

// ---------------------------------------------------------------------------------------------------------------
// 64-bit fixed point

struct __align__(16) fx2 {
	long long x, y;
};
constexpr int FX_TOP = 56;
// power of two the twiddles between the two passes scale by (result = product / 2^shift)
__host__ __device__ constexpr int fx_shift(int n)
{
	int s = 2;
	while ((256 << (s - 2)) < n) s++;
	return s;
}

// a = h*2^32 + l with l signed
__device__ __forceinline__ void fx_split(long long a, int &h, int &l)
{
	l = (int)a;
	h = (int)(a >> 32) + (int)((unsigned)l >> 31);
}
// a*k / 2^64 rounded, k a 64-bit fixed-point constant (|a| < 2^61.5): the three upper partial products
__device__ __forceinline__ long long fx_mulhi(long long a, long long k)
{
	int ah, al;
	fx_split(a, ah, al);
	const int kl = (int)k, kh = (int)(k >> 32) + (int)((unsigned)kl >> 31);
	const long long t = (long long)ah * kl + ((long long)al * kh + 0x80000000ll);
	return (long long)ah * kh + (t >> 32);
}
// v * c for a compile-time constant |c| < 1 (scale 2^63: the product comes out halved and is doubled)
__device__ __forceinline__ long long fx_mulc(long long v, double c)
{
	const long long r = fx_mulhi(v, (long long)(c * 9223372036854775808.0));
	return r + r;
}
// v * (c + i s), compile-time constants; |c| == |s| (odd multiples of pi/4) takes two real products
__device__ __forceinline__ fx2 crot(fx2 v, double c, double s)
{
	if (c == 0) return s > 0 ? fx2{-v.y, v.x} : fx2{v.y, -v.x}; // a quarter turn: 1 is no constant of the products
	if (c == s) return fx2{fx_mulc(v.x - v.y, c), fx_mulc(v.x + v.y, c)};
	if (c == -s) return fx2{fx_mulc(v.x + v.y, c), fx_mulc(v.y - v.x, c)};
	const long long kc = (long long)(c * 9223372036854775808.0), ks = (long long)(s * 9223372036854775808.0);
	const int cl = (int)kc, ch = (int)(kc >> 32) + (int)((unsigned)cl >> 31);
	const int sl = (int)ks, sh = (int)(ks >> 32) + (int)((unsigned)sl >> 31);
	int xh, xl, yh, yl;
	fx_split(v.x, xh, xl);
	fx_split(v.y, yh, yl);
	long long t = (long long)xh * cl + ((long long)xl * ch + 0x80000000ll);
	t = (long long)yh * -sl + t;
	t = (long long)yl * -sh + t;
	long long u = (long long)xh * sl + ((long long)xl * sh + 0x80000000ll);
	u = (long long)yh * cl + u;
	u = (long long)yl * ch + u;
	const long long re = (long long)xh * ch + ((long long)yh * -sh + (t >> 32));
	const long long im = (long long)xh * sh + ((long long)yh * ch + (u >> 32));
	return fx2{re + re, im + im};
}
// v * w / 2^64, w = {c, s} as signed 32-bit halves (c high, c low, s high, s low); conj: times the conjugate.
// |v| < 2^61.5 in modulus and |w| <= 2^62: the sums of partial products stay below 2^63
__device__ __forceinline__ fx2 fx_cmul(fx2 v, int4 w, bool conj)
{
	int xh, xl, yh, yl;
	fx_split(v.x, xh, xl);
	fx_split(v.y, yh, yl);
	const int ph = conj ? -w.z : w.z, pl = conj ? -w.w : w.w, mh = conj ? w.z : -w.z, ml = conj ? w.w : -w.w;
	long long t = (long long)xh * w.y + ((long long)xl * w.x + 0x80000000ll);
	t = (long long)yh * ml + t;
	t = (long long)yl * mh + t;
	long long u = (long long)xh * pl + ((long long)xl * ph + 0x80000000ll);
	u = (long long)yh * w.y + u;
	u = (long long)yl * w.x + u;
	return fx2{(long long)xh * w.x + ((long long)yh * mh + (t >> 32)), (long long)xh * ph + ((long long)yh * w.x + (u >> 32))};
}
// v / 2^s rounded
__device__ __forceinline__ long long fx_rshift(long long v, int s) { return (v + (1ll << (s - 1))) >> s; }
// v * 2^d rounded, d of either sign (the caller's range makes a left shift safe); d is mostly the same for a whole warp,
// so the two directions are separate paths
__device__ __forceinline__ fx2 fx_shift(fx2 v, int d)
{
	if (d >= 0) return fx2{v.x << d, v.y << d};
	const int s = min(-d, 62);
	const long long half = 1ll << (s - 1);
	return fx2{(v.x + half) >> s, (v.y + half) >> s};
}
// bits that v and the values OR-ed into the same accumulator need: their common magnitude is below
// 2^(64 - clz(acc)) (the accumulator holds high words of |v| or |v|-1)
__device__ __forceinline__ void fx_or(unsigned &acc, long long v)
{
	const int h = (int)(v >> 32);
	acc |= (unsigned)(h ^ (h >> 31));
}
// number m with |v| < 2^m for every v that went into acc; 32 when only low words are set (or nothing is)
__device__ __forceinline__ int fx_bits(unsigned acc) { return 64 - __clz((int)acc); }

// A block of values v with one exponent e: value = v * 2^e, |value| < 2^top. top = FX_BAD: an infinity or NaN went in
// (everything computed from it is NaN, as it would be in an FP64 transform); FX_LOW: below every top.
constexpr int FX_BAD = 1 << 20, FX_LOW = -(1 << 20);

// double -> fixed point with the exponent field emax of the block's largest value (>= 1): |v| < 2^FX_TOP, and
// value = v * 2^(emax - 1075 - (FX_TOP - 53))
__device__ __forceinline__ long long fx_from_double(double d, int emax)
{
	const int hi = __double2hiint(d);
	const int ex = (hi >> 20) & 0x7ff;
	long long m = ((long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(d);
	const int sh = emax - max(ex, 1);
	m <<= FX_TOP - 53;
	m = sh > 60 ? 0 : sh ? fx_rshift(m, sh) : m;
	return hi < 0 ? -m : m;
}
// fixed point -> double, v * 2^e rounded, in integer arithmetic (a conversion instruction costs FP64 issue time)
__device__ __forceinline__ double fx_to_double(long long v, int e)
{
	if (v == 0) return 0.0;
	const int lz = __clzll(v < 0 ? -v : v), ex = 1023 + 63 - lz + e;
	if (ex < 1 || ex > 2045) return scalbn(__ll2double_rn(v), e);
	const unsigned long long a = (unsigned long long)(v < 0 ? -v : v) << lz;
	// 53 bits with the leading one, which carries into the exponent field
	const unsigned long long b = (a >> 11) + ((a >> 10) & 1) + ((unsigned long long)(ex - 1) << 52);
	return __longlong_as_double((long long)(b | ((unsigned long long)v & 0x8000000000000000ull)));
}

// ---------------------------------------------------------------------------------------------------------------
// register DFTs of the composite lengths

// cos and sin of 2*pi*k/n by Taylor series on [0, pi/4], for tables of constants
struct Trig {
	double c, s;
};
constexpr Trig ct_small(double x)
{
	double c = 1, s = x, tc = 1, ts = x;
	for (int i = 1; i < 14; i++) {
		tc = -tc * x * x / ((2 * i - 1) * (2 * i));
		ts = -ts * x * x / ((2 * i) * (2 * i + 1));
		c += tc;
		s += ts;
	}
	return Trig{c, s};
}
constexpr Trig ct_root(int k, int n)
{
	// octant reduction: 8k = oct*n + rem
	const int e = 8 * (k % n), oct = e / n;
	const double a = (double)(e - oct * n) / n * 0.78539816339744830962;
	const Trig A = ct_small(a), B = ct_small(0.78539816339744830962 - a);
	switch (oct) {
		case 0: return Trig{A.c, A.s};
		case 1: return Trig{B.s, B.c};
		case 2: return Trig{-A.s, A.c};
		case 3: return Trig{-B.c, B.s};
		case 4: return Trig{-A.c, -A.s};
		case 5: return Trig{-B.s, -B.c};
		case 6: return Trig{A.s, -A.c};
		default: return Trig{B.c, -B.s};
	}
}
template <int N> struct RootTable {
	double c[N], s[N];
	constexpr RootTable() : c(), s()
	{
		for (int k = 0; k < N; k++) {
			const Trig t = ct_root(k, N);
			c[k] = t.c;
			s[k] = t.s;
		}
	}
};

template <typename C, int R> __device__ __forceinline__ void dftr(C *v, bool inv);

// N = A*B with coprime A and B: Good's index maps, no twiddles (the permutations are register renaming)
template <typename C, int A, int B> __device__ __forceinline__ void dft_coprime(C *v, bool inv)
{
	constexpr int N = A * B;
	constexpr int ba = []() { for (int i = 1; i <= A; i++) if (B * i % A == 1 % A) return i; return 0; }(); // B^-1 mod A
	constexpr int ab = []() { for (int i = 1; i <= B; i++) if (A * i % B == 1 % B) return i; return 0; }(); // A^-1 mod B
	C t[N];
#pragma unroll
	for (int n2 = 0; n2 < B; n2++) {
		C u[A];
#pragma unroll
		for (int n1 = 0; n1 < A; n1++) u[n1] = v[(B * n1 + A * n2) % N];
		dftr<C, A>(u, inv);
#pragma unroll
		for (int k1 = 0; k1 < A; k1++) t[k1 * B + n2] = u[k1];
	}
#pragma unroll
	for (int k1 = 0; k1 < A; k1++) {
		dftr<C, B>(t + k1 * B, inv);
#pragma unroll
		for (int k2 = 0; k2 < B; k2++) v[(B * ba * k1 + A * ab * k2) % N] = t[k1 * B + k2];
	}
}
// N = A*B in general: twiddles between the two factors
template <typename C, int A, int B> __device__ __forceinline__ void dft_twiddled(C *v, bool inv)
{
	constexpr int N = A * B;
	constexpr RootTable<N> w;
	C t[N];
#pragma unroll
	for (int n2 = 0; n2 < B; n2++) {
		C u[A];
#pragma unroll
		for (int n1 = 0; n1 < A; n1++) u[n1] = v[B * n1 + n2];
		dftr<C, A>(u, inv);
#pragma unroll
		for (int k1 = 0; k1 < A; k1++) {
			const int e = (n2 * k1) % N;
			t[k1 * B + n2] = e ? crot(u[k1], w.c[e], inv ? w.s[e] : -w.s[e]) : u[k1];
		}
	}
#pragma unroll
	for (int k1 = 0; k1 < A; k1++) {
		dftr<C, B>(t + k1 * B, inv);
#pragma unroll
		for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = t[k1 * B + k2];
	}
}

// the fixed-point forms of the odd prime DFTs (dft3 and dft_odd of common.cuh with fixed-point constants)
template <int R> __device__ __forceinline__ void fx_dft_odd(fx2 *v, bool inv)
{
	constexpr int H = (R - 1) / 2;
	constexpr RootTable<R> w;
	fx2 a[H], b[H];
#pragma unroll
	for (int p = 1; p <= H; p++) {
		a[p - 1] = cadd(v[p], v[R - p]);
		b[p - 1] = csub(v[p], v[R - p]);
	}
	const fx2 x0 = v[0];
	fx2 sum = x0;
#pragma unroll
	for (int p = 0; p < H; p++) sum = cadd(sum, a[p]);
	v[0] = sum;
#pragma unroll
	for (int k = 1; k <= H; k++) {
		fx2 t = x0, u{0, 0};
#pragma unroll
		for (int p = 1; p <= H; p++) {
			const int i = (p * k) % R;
			t.x += fx_mulc(a[p - 1].x, w.c[i]);
			t.y += fx_mulc(a[p - 1].y, w.c[i]);
			u.x += fx_mulc(b[p - 1].x, w.s[i]);
			u.y += fx_mulc(b[p - 1].y, w.s[i]);
		}
		const fx2 m{t.x + u.y, t.y - u.x}, q{t.x - u.y, t.y + u.x};
		v[k] = inv ? q : m;
		v[R - k] = inv ? m : q;
	}
}

template <typename C, int R> __device__ __forceinline__ void dftr(C *v, bool inv)
{
	constexpr bool fx = std::is_same<C, fx2>::value;
	if constexpr (R == 1) {
	}
	else if constexpr (R == 2 || R == 4 || R == 8 || R == 16 || R == 32) dft<C, R>(v, inv, nullptr, R);
	else if constexpr (R == 3 || R == 5 || R == 7 || R == 11 || R == 13) {
		if constexpr (fx) fx_dft_odd<R>(v, inv);
		else dft<C, R>(v, inv, nullptr, R);
	}
	else if constexpr (R == 6) dft_coprime<C, 2, 3>(v, inv);
	else if constexpr (R == 9) dft_twiddled<C, 3, 3>(v, inv);
	else if constexpr (R == 10) dft_coprime<C, 2, 5>(v, inv);
	else if constexpr (R == 12) dft_coprime<C, 4, 3>(v, inv);
	else if constexpr (R == 14) dft_coprime<C, 2, 7>(v, inv);
	else if constexpr (R == 15) dft_coprime<C, 3, 5>(v, inv);
	else if constexpr (R == 18) dft_coprime<C, 2, 9>(v, inv);
	else if constexpr (R == 20) dft_coprime<C, 4, 5>(v, inv);
	else if constexpr (R == 21) dft_coprime<C, 3, 7>(v, inv);
	else if constexpr (R == 22) dft_coprime<C, 2, 11>(v, inv);
	else if constexpr (R == 24) dft_coprime<C, 8, 3>(v, inv);
	else if constexpr (R == 25) dft_twiddled<C, 5, 5>(v, inv);
	else if constexpr (R == 26) dft_coprime<C, 2, 13>(v, inv);
	else if constexpr (R == 27) dft_twiddled<C, 9, 3>(v, inv);
	else if constexpr (R == 28) dft_coprime<C, 4, 7>(v, inv);
	else if constexpr (R == 30) dft_coprime<C, 2, 15>(v, inv);
	else static_assert(R < 0, "radix not built");
}

// the radices of the run-time switches, by class: RC_SMALL 1 to RADIX_MAX, RC_BIG 9 to RADIX_BIG (a plan is big when one
// of its radices is above RADIX_MAX; the other is then at least 9). CALL sees the radix as the constant RR
enum RadixClass { RC_SMALL = 0, RC_BIG = 1 };
constexpr bool radix_in_class(int r, int rc, bool fx) { return radix_built(r, fx) && (rc == RC_BIG ? r >= 9 : r <= RADIX_MAX); }
#define ADDA_RADIX_CASE(r, ...)                                                                                     \
	case r:                                                                                                         \
		if constexpr (radix_in_class(r, RC, A::FX)) {                                                               \
			constexpr int RR = r;                                                                                   \
			__VA_ARGS__;                                                                                            \
		}                                                                                                           \
		break;
#define ADDA_RADIX_SWITCH(rv, ...)                                                                                  \
	switch (rv) {                                                                                                   \
		ADDA_RADIX_CASE(1, __VA_ARGS__) ADDA_RADIX_CASE(2, __VA_ARGS__) ADDA_RADIX_CASE(3, __VA_ARGS__)             \
		ADDA_RADIX_CASE(4, __VA_ARGS__) ADDA_RADIX_CASE(5, __VA_ARGS__) ADDA_RADIX_CASE(6, __VA_ARGS__)             \
		ADDA_RADIX_CASE(7, __VA_ARGS__) ADDA_RADIX_CASE(8, __VA_ARGS__) ADDA_RADIX_CASE(9, __VA_ARGS__)             \
		ADDA_RADIX_CASE(10, __VA_ARGS__) ADDA_RADIX_CASE(11, __VA_ARGS__) ADDA_RADIX_CASE(12, __VA_ARGS__)          \
		ADDA_RADIX_CASE(13, __VA_ARGS__) ADDA_RADIX_CASE(14, __VA_ARGS__) ADDA_RADIX_CASE(15, __VA_ARGS__)          \
		ADDA_RADIX_CASE(16, __VA_ARGS__) ADDA_RADIX_CASE(18, __VA_ARGS__) ADDA_RADIX_CASE(20, __VA_ARGS__)          \
		ADDA_RADIX_CASE(21, __VA_ARGS__) ADDA_RADIX_CASE(22, __VA_ARGS__) ADDA_RADIX_CASE(24, __VA_ARGS__)          \
		ADDA_RADIX_CASE(25, __VA_ARGS__) ADDA_RADIX_CASE(26, __VA_ARGS__) ADDA_RADIX_CASE(27, __VA_ARGS__)          \
		ADDA_RADIX_CASE(28, __VA_ARGS__) ADDA_RADIX_CASE(30, __VA_ARGS__) ADDA_RADIX_CASE(32, __VA_ARGS__)          \
		default: break;                                                                                             \
	}
constexpr int radix_max(int rc) { return rc == RC_BIG ? RADIX_BIG : RADIX_MAX; }

// ---------------------------------------------------------------------------------------------------------------
// the two passes

struct Ar32 {
	typedef float T;
	typedef float2 C, Tw;
	static constexpr bool FX = false;
};
struct ArFx {
	typedef double T;
	typedef fx2 C;
	typedef int4 Tw;
	static constexpr bool FX = true;
};
__device__ __forceinline__ float2 tw_mul(float2 v, float2 w, bool conj)
{
	if (conj) w.y = -w.y;
	return cmul(v, w);
}
__device__ __forceinline__ fx2 tw_mul(fx2 v, int4 w, bool conj) { return fx_cmul(v, w, conj); }

// elements per row group of the exchange buffer of NL lines: [q][j][l], row groups of r2*NL + pad with the pad that puts
// a warp's second-pass reads on distinct banks
__host__ __device__ __forceinline__ int xch_ks(int nl, int r2) { return r2 * nl + (nl * (17 - r2 % 16)) % 16; }

// first pass of thread (l, j), j < r2: elements ld(j + r2*t) (HALF: t < ceil(R/2), the rest are zero), results to
// xb[q*ks + at], at = j*NL + l (or the caller's own place for j)
template <typename A, int R, bool INV, bool HALF, typename LD>
__device__ __forceinline__ void pass_first(LD ld, typename A::C *xb, int ks, int at, int j, int r2,
	const typename A::Tw *__restrict__ tw, int sh)
{
	typedef typename A::C C;
	constexpr int L = HALF ? (R + 1) / 2 : R;
	C v[R];
#pragma unroll
	for (int t = 0; t < L; t++) v[t] = ld(t, j + r2 * t);
	if constexpr (HALF && !A::FX && (R == 8 || R == 16 || R == 32)) dft_half_in<C, R>(v, INV);
	else {
#pragma unroll
		for (int t = L; t < R; t++) v[t] = cx<C>(0, 0);
		dftr<C, R>(v, INV);
	}
	if constexpr (A::FX) v[0] = fx2{fx_rshift(v[0].x, sh), fx_rshift(v[0].y, sh)};
	xb[at] = v[0];
#pragma unroll
	for (int q = 1; q < R; q++) xb[q * ks + at] = tw_mul(v[q], __ldg(tw + q * r2 + j), INV);
}
// second pass of thread (l, q), q < r1: st(p, q + r1*p, X) for p < R (HALFOUT: p < ceil(R/2))
template <typename A, int R, bool INV, bool HALFOUT, typename LD, typename ST>
__device__ __forceinline__ void pass_second(LD ld, ST st, int q, int r1)
{
	typedef typename A::C C;
	C u[R];
#pragma unroll
	for (int j = 0; j < R; j++) u[j] = ld(j);
	dftr<C, R>(u, INV);
#pragma unroll
	for (int p = 0; p < (HALFOUT ? (R + 1) / 2 : R); p++) st(p, q + r1 * p, u[p]);
}

} // namespace adda
