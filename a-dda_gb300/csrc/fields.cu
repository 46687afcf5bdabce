// fields.cu - scattering amplitudes of the last solve in a set of directions (CalcFieldFree, crosssec.c:506-596):
// E_r(n) = (-i k^3) exp(-i k r0.n) (I - nn) sum_j P_rj exp(-i kd n.pos_j).
//
// One or two directions, or few dipoles: a sincos per dipole and direction (fld_few; the rule is in scattered_fields). Else
// the sum is FP64-exact work on a chip whose FP64 pipe issues one instruction per 76 cycles and scheduler, so it runs on
// the integer pipes:
//   - the lattice makes the phase a product of three factors, one per axis: exp(-i kd n.pos) = X[x] Y[y] Z[z], taken from
//     tables of (boxX + boxY + boxZ) values per direction instead of one sincos per dipole and direction;
//   - along an x-line only X[x] changes: the dipoles of a line are summed with it, and the line's sum is multiplied by
//     Y[y] Z[z];
//   - P (relative to the RHS's largest value of the same component: a field along a dominant component is made of the
//     other two only) and X are 54-bit fixed point in two signed limbs of 27 bits.
//     A complex product is 12 32x32+64-bit multiply-adds (2 cycles each); the limb products of up to FLD_RUN dipoles
//     accumulate in 64 bits without carries.
// One unit is 2^-54 of the largest P component (FP64 rounding of a typical term); the phases of the tables and of the
// box centre are taken to twice the precision before the sine, from the same k gs, and no rounding leans to one side.
// Error of the fields against 80-bit sums (direct FP64 sum with a sincos per dipole -> this): 12^3 box 3.0e-16 -> 2.1e-16,
// 20^3 5.7e-16 -> 2.4e-16, 36x28x22 9.4e-16 -> 2.7e-16, 64^3 1.4e-15 -> 2.9e-16. (A plain FP64 sum in numpy or torch is
// itself 5e-15 off at 64^3.)
// Measured: 64^3 sphere (137 k dipoles), 2 RHS, 2080 directions, with the host copies and the cross sections: 57.1 ms
// with an FP64 sincos per dipole and direction -> 3.36 ms, of which fld_sum 3.2 ms (66 instructions a dipole and warp;
// the multiply-add pipe's bound is 1.3 ms, the rest are the loads' latency at 20 warps an SM). One warp per block: with
// blocks of four warps the last wave was half empty (5.4 ms, with a data-dependent loop over the dipoles).
#include "fft_lines2.cuh"
#include "ctx.cuh"
#include "krylov.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace adda {

namespace {

constexpr int FLD_NT = 192;         // threads per block of the passes over P
constexpr int FEW_NT = 256;         // threads per block of the direct sum
constexpr int FLD_RUN = 128;        // dipoles whose limb products fit 64-bit sums: 2^55 each
constexpr int FLD_SPAN = 512;       // dipoles whose sums stay below 2^62 in fixed point
constexpr int FLD_RESIDENT = 20;    // resident warps (blocks) an SM of the sum
constexpr int FLD_FIN_D = 8;        // directions per block of the last sum
constexpr size_t FLD_TABLE = 64u << 20; // bytes of phase tables per launch (bounds the directions of one)

// largest high word of |P| per RHS and component (hmax [R][3] zeroed before). The stride is a multiple of 3, so a thread
// stays with one component
__global__ void __launch_bounds__(FLD_NT) fld_max(const double2 *P, size_t n3, int *hmax)
{
	static_assert(FLD_NT % 3 == 0, "a thread's component");
	__shared__ int s[3];
	const int r = blockIdx.y, c = threadIdx.x % 3;
	if (threadIdx.x < 3) s[threadIdx.x] = 0;
	__syncthreads();
	int h = 0;
	for (size_t i = blockIdx.x * (size_t)FLD_NT + threadIdx.x; i < n3; i += (size_t)gridDim.x * FLD_NT) {
		const double2 v = P[r * n3 + i];
		h = max(h, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
	}
	atomicMax(s + c, h);
	__syncthreads();
	if (threadIdx.x < 3) atomicMax(hmax + 3 * r + threadIdx.x, s[threadIdx.x]);
}

// two signed limbs of 27 bits of |v| < 2^54
__device__ __forceinline__ void fld_limbs(long long v, int &h, int &l)
{
	l = (int)((unsigned)v << 5) >> 5;
	h = (int)((v - l) >> 27);
}
// d in units of 2^(emax - 1076), |result| < 2^54, rounded once and away from zero in the middle: as many values up as down
// (a second rounding, or one towards +infinity, adds up over the dipoles: 3e-14 of the field of 40000)
__device__ __forceinline__ long long fld_fixed(double d, int emax)
{
	const int hi = __double2hiint(d), ex = (hi >> 20) & 0x7ff, sh = emax - max(ex, 1);
	long long m = ((long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 33) | (long long)(unsigned)__double2loint(d) << 1;
	m = sh > 60 ? 0 : sh ? fx_rshift(m, sh) : m;
	return hi < 0 ? -m : m;
}
// acc += v * w without a rounding: the low words collect in lo (carried over into acc), the rest as fx_cmul
__device__ __forceinline__ void fld_madd(fx2 v, int4 w, long long &ax, long long &ay, unsigned &lx, unsigned &ly)
{
	int xh, xl, yh, yl;
	fx_split(v.x, xh, xl);
	fx_split(v.y, yh, yl);
	long long t = (long long)xh * w.y + (long long)xl * w.x;
	t = (long long)yh * -w.w + t;
	t = (long long)yl * -w.z + t;
	long long u = (long long)xh * w.w + (long long)xl * w.z;
	u = (long long)yh * w.y + u;
	u = (long long)yl * w.x + u;
	lx += (unsigned)t;
	ly += (unsigned)u;
	ax += (long long)xh * w.x + ((long long)yh * -w.z + ((t >> 32) + (lx < (unsigned)t)));
	ay += (long long)xh * w.z + ((long long)yh * w.x + ((u >> 32) + (ly < (unsigned)u)));
}
// P in limbs: element i of RHS r at [r*n3 + i], (re high, re low, im high, im low)
__global__ void __launch_bounds__(FLD_NT) fld_split(const double2 *P, size_t n3, const int *hmax, int4 *out)
{
	const int r = blockIdx.y;
	const int emax = max(1, hmax[3 * r + threadIdx.x % 3] >> 20);
	for (size_t i = blockIdx.x * (size_t)FLD_NT + threadIdx.x; i < n3; i += (size_t)gridDim.x * FLD_NT) {
		const double2 v = P[r * n3 + i];
		int4 o;
		fld_limbs(fld_fixed(v.x, emax), o.x, o.y);
		fld_limbs(fld_fixed(v.y, emax), o.z, o.w);
		out[r * n3 + i] = o;
	}
}

// phase tables of nd directions (row length ld): x factors as limbs of 2^54, y and z factors as 2^62 split for fx_cmul.
// kd + kl: the wave number times the spacing, k gs, to twice the precision, as in fld_finish: a rounding of it that only
// one of the two had would grow with the distance from the box's corner (1.4e-14 at the far end of a 300 long box)
__global__ void __launch_bounds__(256) fld_tables(const double *dirs, int nd, int ld, int bX, int bY, int bZ, double kd,
	double kl, int4 *tab)
{
	const int d = blockIdx.x * blockDim.x + threadIdx.x;
	int t = blockIdx.y; // table row: x, then y, then z
	if (d >= nd) return;
	const int axis = t < bX ? 0 : t < bX + bY ? 1 : 2;
	const int i = t - (axis ? bX : 0) - (axis == 2 ? bY : 0);
	// the phase ph + lo to twice the precision: a table's error is the same for every dipole of a plane, so it averages
	// out less than the rounding of a phase per dipole
	const double n = dirs[3 * d + axis], t0 = n * i, ph = -kd * t0,
				 lo = __fma_rn(-kd, t0, -ph) - kd * __fma_rn(n, i, -t0) - kl * t0;
	double sn, cs;
	sincos(ph, &sn, &cs);
	const long long c = __double2ll_rn(cs * 4611686018427387904.0) + __double2ll_rn(-lo * sn * 4611686018427387904.0);
	const long long q = __double2ll_rn(sn * 4611686018427387904.0) + __double2ll_rn(lo * cs * 4611686018427387904.0);
	int4 o;
	if (axis == 0) {
		fld_limbs(fx_rshift(c, 8), o.x, o.y);
		fld_limbs(fx_rshift(q, 8), o.z, o.w);
	}
	else {
		fx_split(c, o.x, o.y);
		fx_split(q, o.z, o.w);
		o.y = max(o.y, -0x7fffffff); // negated in fx_cmul
		o.w = max(o.w, -0x7fffffff);
	}
	tab[(size_t)t * ld + d] = o;
}

// partial sums over a range of dipoles for 32 directions, one per lane: grid (direction groups, ranges, RHS), one warp a
// block, so that the neighbours in x read the same dipoles through L1. part: [range][R][6][ld]
__global__ void __launch_bounds__(32, FLD_RESIDENT) fld_sum(const int4 *P, const uint16_t *pos, const uint32_t *xy,
	const uint32_t *lstart, size_t N, const int4 *tab, const int *hmax, int nd, int ld, int bX, int bY, int bZ, size_t span,
	double *part, int rpp, size_t lst)
{
	const int r = blockIdx.z, R = gridDim.z;
	const int d = blockIdx.x * 32 + threadIdx.x;
	const size_t lq = (size_t)(r / rpp); // RHS r's particle (group contexts)
	pos += lq * lst * 3;
	xy += lq * lst;
	lstart += lq * ((size_t)bZ * bY + 1);
	P += (size_t)r * 3 * N;
	// the particle's own dipoles (a smaller particle of a group is padded to N)
	const size_t i0 = (size_t)blockIdx.y * span, i1 = min((size_t)lstart[(size_t)bZ * bY], i0 + span);
	const int4 *tx = tab + d, *ty = tx + (size_t)bX * ld, *tz = ty + (size_t)bY * ld;
	const int hm[3] = {hmax[3 * r], hmax[3 * r + 1], hmax[3 * r + 2]};
	double tot[6] = {0, 0, 0, 0, 0, 0};
	size_t i = i0;
	while (i < i1) {
		const size_t iend = min(i1, i + FLD_SPAN);
		long long S[6] = {0, 0, 0, 0, 0, 0};
		unsigned low[6] = {0, 0, 0, 0, 0, 0};
		while (i < iend) {
			// one run: dipoles of one x-line, at most FLD_RUN of them
			const int y = pos[3 * i + 1], z = pos[3 * i + 2];
			const int n = (int)(min(min(iend, i + FLD_RUN), (size_t)lstart[(size_t)z * bY + y + 1]) - i);
			const long long half = 1ll << 26; // rounds T >> 27
			long long U[6] = {0, 0, 0, 0, 0, 0}, T[6] = {half, half, half, half, half, half};
			const int4 *p = P + 3 * i;
			const uint32_t *px = xy + i;
#pragma unroll 2
			for (int t = 0; t < n; t++) {
				const int4 w = __ldg(tx + (size_t)(px[t] & 0xffff) * ld);
				const int nsh = -w.z, nsl = -w.w;
#pragma unroll
				for (int c = 0; c < 3; c++) {
					const int4 v = __ldg(p + 3 * t + c);
					U[2 * c] = (long long)v.x * w.x + U[2 * c];
					U[2 * c] = (long long)v.z * nsh + U[2 * c];
					U[2 * c + 1] = (long long)v.x * w.z + U[2 * c + 1];
					U[2 * c + 1] = (long long)v.z * w.x + U[2 * c + 1];
					T[2 * c] = (long long)v.x * w.y + T[2 * c];
					T[2 * c] = (long long)v.y * w.x + T[2 * c];
					T[2 * c] = (long long)v.z * nsl + T[2 * c];
					T[2 * c] = (long long)v.w * nsh + T[2 * c];
					T[2 * c + 1] = (long long)v.x * w.w + T[2 * c + 1];
					T[2 * c + 1] = (long long)v.y * w.z + T[2 * c + 1];
					T[2 * c + 1] = (long long)v.z * w.y + T[2 * c + 1];
					T[2 * c + 1] = (long long)v.w * w.x + T[2 * c + 1];
				}
			}
			i += n;
			// the line's sum times Y Z (2^60 after the product of the two, back to 2^62)
			const int4 yv = __ldg(ty + (size_t)y * ld), zv = __ldg(tz + (size_t)z * ld);
			const fx2 yy{((long long)yv.x << 32) + yv.y, ((long long)yv.z << 32) + yv.w};
			const fx2 q = fx_cmul(yy, zv, false);
			int4 yz;
			fx_split(q.x << 2, yz.x, yz.y);
			fx_split(q.y << 2, yz.z, yz.w);
			yz.w = max(yz.w, -0x7fffffff); // negated in fld_madd
#pragma unroll
			for (int c = 0; c < 3; c++) {
				// (U * 2^54 + T * 2^27) / 2^54
				fld_madd(fx2{U[2 * c] + (T[2 * c] >> 27), U[2 * c + 1] + (T[2 * c + 1] >> 27)}, yz, S[2 * c], S[2 * c + 1],
					low[2 * c], low[2 * c + 1]);
			}
		}
#pragma unroll
		for (int c = 0; c < 6; c++) {
			// the upper 62 bits of S and low; a unit of S is four of P's
			const int sh = max(0, min(__clzll(S[c] ^ (S[c] >> 63)) - 2, 31)), e = max(1, hm[c / 2] >> 20) - 1074;
			tot[c] += fx_to_double((S[c] << sh) + (long long)(sh ? low[c] >> (32 - sh) : 0), e - sh);
		}
	}
	if (d < nd) {
		double *o = part + ((size_t)blockIdx.y * R + r) * 6 * ld + d;
#pragma unroll
		for (int c = 0; c < 6; c++) o[(size_t)c * ld] = hm[c / 2] >= 0x7ff00000 ? __hiloint2double(0x7ff80000, 0) : tot[c];
	}
}

// Few directions: partial sums in FP64 with a sincos per dipole and direction, grid (ranges, directions, RHS), positions from
// the box centre; part as fld_sum's. The phase is a.(2 r) to twice the precision: a's high parts (few_phase) make exact
// products and sums
__global__ void __launch_bounds__(FEW_NT) fld_few(const double2 *P, const uint16_t *pos, const uint32_t *lstart, size_t N,
	const double *phase, int ld, int bX, int bY, int bZ, double *part, int rpp, size_t lst)
{
	const int d = blockIdx.y, r = blockIdx.z, R = gridDim.z;
	const size_t lq = (size_t)(r / rpp), lines = (size_t)bZ * bY; // RHS r's particle (group contexts)
	pos += lq * lst * 3;
	const size_t n1 = lstart[lq * (lines + 1) + lines];
	double a[6];
#pragma unroll
	for (int c = 0; c < 6; c++) a[c] = phase[6 * d + c];
	double s[6] = {0, 0, 0, 0, 0, 0};
	for (size_t j = blockIdx.x * (size_t)FEW_NT + threadIdx.x; j < n1; j += (size_t)gridDim.x * FEW_NT) {
		// twice the position from the centre: whole numbers
		const double x = 2 * pos[3 * j] - (bX - 1), y = 2 * pos[3 * j + 1] - (bY - 1), z = 2 * pos[3 * j + 2] - (bZ - 1);
		const double lo = __fma_rn(a[3], x, __fma_rn(a[4], y, a[5] * z));
		double sn, cs;
		sincos(__fma_rn(a[0], x, __fma_rn(a[1], y, a[2] * z)), &sn, &cs);
		const double wr = __fma_rn(-lo, sn, cs), wi = __fma_rn(lo, cs, sn);
#pragma unroll
		for (int c = 0; c < 3; c++) {
			const double2 p = P[((size_t)r * N + j) * 3 + c];
			s[2 * c] += p.x * wr - p.y * wi;
			s[2 * c + 1] += p.x * wi + p.y * wr;
		}
	}
	double tot[6];
	block_totals<6>(s, tot);
	if (threadIdx.x == 0)
#pragma unroll
		for (int c = 0; c < 6; c++) part[(((size_t)blockIdx.x * R + r) * 6 + c) * ld + d] = tot[c];
}
// -k gs n / 2 as high parts, whole multiples of a power of two that leaves all phases of the box below 2^51 of it, and the
// rest; kd + kl = k gs
void few_phase(const double n[3], const int box[3], double kd, double kl, double a[6])
{
	double most = 0;
	for (int c = 0; c < 3; c++) most += std::fabs(kd * n[c]) * box[c];
	const double unit = most > 0 && most < 1e300 ? std::ldexp(1.0, std::max(std::ilogb(most) - 51, -1000)) : 1.0;
	for (int c = 0; c < 3; c++) {
		const double v = -0.5 * kd * n[c], lo = -0.5 * (std::fma(kd, n[c], 2 * v) + kl * n[c]);
		a[c] = most < 1e300 ? std::nearbyint(v / unit) * unit : v;
		a[3 + c] = (v - a[c]) + lo;
	}
}

__device__ __forceinline__ double2 cmuld(double2 a, double2 b)
{
	return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// FLD_FIN_D directions of one RHS per block: fixed-order sum of the partials (32 threads a direction), (I - nn), and the
// factor (-i k^3) exp(-i k r0.n) with r0 the centre offset of the box's first dipole (make_particle.c:2305-2308).
// out [R][ndir][3], directions d0...
__global__ void __launch_bounds__(32 * FLD_FIN_D) fld_finish(const double *part, int slices, int nd, int ld, int R,
	const double *dirs, double k, double kd, double kl, int bX, int bY, int bZ, double2 *out, int ndir, int d0)
{
	__shared__ double sh[32][6][FLD_FIN_D], amp[2][FLD_FIN_D];
	const int l = threadIdx.x % FLD_FIN_D, w = threadIdx.x / FLD_FIN_D, r = blockIdx.y, d = blockIdx.x * FLD_FIN_D + l;
	double s[6] = {0, 0, 0, 0, 0, 0};
	if (d < nd)
		for (int b = w; b < slices; b += 32)
#pragma unroll
			for (int c = 0; c < 6; c++) s[c] += part[(((size_t)b * R + r) * 6 + c) * ld + d];
#pragma unroll
	for (int c = 0; c < 6; c++) sh[w][c][l] = s[c];
	double n[3] = {0, 0, 0};
	if (d < nd)
		for (int c = 0; c < 3; c++) n[c] = dirs[3 * d + c];
	if (w == 31) { // the last warp, while the first ones add up
		// phase -k r0.n = k gs n.(box - 1)/2, to twice the precision like the tables' (box 1: no phase, fld_few)
		const double m[3] = {(bX - 1) / 2.0, (bY - 1) / 2.0, (bZ - 1) / 2.0};
		double h = 0, lo = 0;
		for (int c = 0; c < 3; c++) {
			const double t = n[c] * m[c], g = h + t, z = g - h;
			lo += __fma_rn(n[c], m[c], -t) + ((h - (g - z)) + (t - z));
			h = g;
		}
		const double ph = kd * h;
		lo = __fma_rn(kd, h, -ph) + kl * h + kd * lo;
		double sn, cs;
		sincos(ph, &sn, &cs);
		const double c0 = cs;
		cs = __fma_rn(-lo, sn, cs);
		sn = __fma_rn(lo, c0, sn);
		const double k3 = k * k * k;
		amp[0][l] = sn * k3; // -i k^3 (cs + i sn)
		amp[1][l] = -cs * k3;
	}
	__syncthreads();
	if (w < 6) {
		// pairwise: a serial sum of 32 rounds twice as much as the dipoles' sums
		double t[32];
#pragma unroll
		for (int b = 0; b < 32; b++) t[b] = sh[b][w][l];
#pragma unroll
		for (int o = 16; o > 0; o >>= 1)
#pragma unroll
			for (int b = 0; b < o; b++) t[b] += t[b + o];
		sh[0][w][l] = t[0]; // this thread's own
	}
	__syncthreads();
	if (w || d >= nd) return;
#pragma unroll
	for (int c = 0; c < 6; c++) s[c] = sh[0][c][l];
	double2 dpr = make_double2(0, 0);
	for (int c = 0; c < 3; c++) {
		dpr.x += s[2 * c] * n[c];
		dpr.y += s[2 * c + 1] * n[c];
	}
	for (int c = 0; c < 3; c++)
		out[((size_t)r * ndir + d0 + d) * 3 + c] = cmuld(make_double2(amp[0][l], amp[1][l]),
			make_double2(s[2 * c] - dpr.x * n[c], s[2 * c + 1] - dpr.y * n[c]));
}

} // namespace

int scattered_fields(adda_gb300_ctx *c, int R, int ndir, const double *dirs, double *ebuff)
{
	const size_t N = c->N, n3 = 3 * N;
	cudaStream_t s = c->stream;
	const double kd = c->k * c->gridspace, kl = std::fma(c->k, c->gridspace, -kd);
	// few directions for the dipoles and RHS at hand: a sincos each (0.13 ns of the FP64 pipes per dipole, RHS and direction)
	// against two passes over P, the tables and 32 directions whether asked for or not (20 us and 0.3 to 0.5 ns per dipole
	// and RHS). Measured direct / tables, us: 1, 2, 3, 4 directions of a 64^3 sphere with 1 RHS 51, 69, 82, 93 / 126, with
	// 2 RHS 68, 94, 120, 155 / 149, of a 128^3 sphere with 2 RHS 280, 513, 748, 870 / 700; 16 directions of a 32^3 sphere
	// with 1 RHS 60 / 65, 2 RHS 87 / 68; 60 directions of 8^3 34 / 52, 16^3 with 1 and 2 RHS 46, 58 / 52
	const size_t work = N * (size_t)R;
	const bool few = ndir <= 2 || work * (ndir - 2) < 250000;
	const size_t rows = (size_t)c->bX + c->bY + c->bZ;
	// directions per launch: the tables' budget, a multiple of 32 within the grid's limit
	const int per = (int)std::max<size_t>(32, std::min<size_t>(32768, FLD_TABLE / (rows * sizeof(int4)) / 32 * 32));
	const int ld = std::min(per, few ? ndir : (ndir + 31) / 32 * 32), groups = ld / 32;
	// ranges of dipoles: three waves of resident warps (lines of different length even out); where few directions leave the
	// chip emptier than that, sqrt(N / 16) dipoles each, at least 16: a dipole costs a lone warp 0.44 us (latency), a range
	// 0.025 us in fld_finish. Measured with 33 to 80 directions (sum and finish, ranges of 256 -> this): 16x8x8 box 119 ->
	// 20 us, 36x27x22 ellipsoid 127 -> 36, 42^3 sphere 142 -> 62
	const size_t warps = (size_t)152 * FLD_RESIDENT * 3, per_slice = (size_t)groups * R;
	const size_t least = std::max<size_t>(16, (size_t)std::sqrt((double)N / 16));
	// the direct sum: one to eight dipoles a thread, so that the FP64 pipes of all SMs have work, at most 128 ranges
	const size_t each = FEW_NT * std::min<size_t>(8, std::max<size_t>(1, work * ndir / ((size_t)152 * 4 * FEW_NT)));
	const size_t slices = std::max<size_t>(1, few ? std::min<size_t>((N + each - 1) / each, 128)
		: std::min<size_t>((N + least - 1) / least, warps / per_slice));
	const size_t span = std::max<size_t>(1, (N + slices - 1) / slices);
	const auto up = [](size_t v) { return (v + 255) / 256 * 256; };
	const size_t b_dirs = up(sizeof(double) * 3 * ndir), b_out = up(sizeof(double2) * 3 * (size_t)ndir * R),
				 b_max = up(sizeof(int) * 3 * R), b_tab = few ? 0 : up(sizeof(int4) * rows * ld), b_part = up(sizeof(double) * slices * R * 6 * ld);
	const size_t b_phase = few ? up(sizeof(double) * 6 * ndir) : 0, need = b_dirs + b_phase + b_out + b_max + b_tab + b_part;
	// the work space is the matvec's chunk buffer, free between two matvecs of the context's stream, where that is large
	// enough: allocating 2 MB costs a context's first call 100 us
	const bool own = need > c->Tz_bytes;
	if (own && need > c->fld_bytes) {
		if (c->fld) cudaFree(c->fld);
		c->fld = nullptr;
		c->fld_bytes = 0;
		ADDA_CUDA(cudaMalloc(&c->fld, need));
		c->fld_bytes = need;
	}
	unsigned char *at = (unsigned char *)(own ? c->fld : c->Tz);
	const auto take = [&](size_t n) {
		unsigned char *q = at;
		at += n;
		return q;
	};
	double *d_dirs = (double *)take(b_dirs), *d_phase = (double *)take(b_phase);
	double2 *d_out = (double2 *)take(b_out);
	int *d_max = (int *)take(b_max);
	int4 *d_tab = (int4 *)take(b_tab);
	int4 *d_p = (int4 *)c->vin; // the staging buffer of the host-pointer matvec: R*3N complex doubles
	double *d_part = (double *)take(b_part);
	ADDA_CUDA(cudaMemcpyAsync(d_dirs, dirs, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, s));
	if (few) {
		const int box[3] = {c->bX, c->bY, c->bZ};
		std::vector<double> a(6 * (size_t)ndir);
		for (int d = 0; d < ndir; d++) few_phase(dirs + 3 * (size_t)d, box, kd, kl, &a[6 * (size_t)d]);
		ADDA_CUDA(cudaMemcpyAsync(d_phase, a.data(), sizeof(double) * a.size(), cudaMemcpyHostToDevice, s));
	}
	else {
		ADDA_CUDA(cudaMemsetAsync(d_max, 0, sizeof(int) * 3 * R, s));
		const dim3 gp((unsigned)std::max<size_t>(1, std::min<size_t>((n3 + FLD_NT - 1) / FLD_NT, 152 * 10)), R);
		fld_max<<<gp, FLD_NT, 0, s>>>(c->pvec64, n3, d_max);
		ADDA_LAUNCHED();
		fld_split<<<gp, FLD_NT, 0, s>>>(c->pvec64, n3, d_max, d_p);
		ADDA_LAUNCHED();
	}
	for (int d0 = 0; d0 < ndir; d0 += ld) {
		const int nd = std::min(ld, ndir - d0);
		const double *dd = d_dirs + 3 * (size_t)d0;
		if (few) {
			fld_few<<<dim3((unsigned)slices, nd, R), FEW_NT, 0, s>>>(c->pvec64, c->d_pos, c->d_line_start, N,
				d_phase + 6 * (size_t)d0, ld, c->bX, c->bY, c->bZ, d_part, c->rpp, c->lat_stride);
			ADDA_LAUNCHED();
		}
		else {
			fld_tables<<<dim3((nd + 255) / 256, (unsigned)rows), 256, 0, s>>>(dd, nd, ld, c->bX, c->bY, c->bZ, kd, kl, d_tab);
			ADDA_LAUNCHED();
			fld_sum<<<dim3(groups, (unsigned)slices, R), 32, 0, s>>>(d_p, c->d_pos, c->d_xy, c->d_line_start, N, d_tab, d_max, nd,
				ld, c->bX, c->bY, c->bZ, span, d_part, c->rpp, c->lat_stride);
			ADDA_LAUNCHED();
		}
		fld_finish<<<dim3((nd + FLD_FIN_D - 1) / FLD_FIN_D, R), 32 * FLD_FIN_D, 0, s>>>(d_part, (int)slices, nd, ld, R, dd, c->k, kd,
			kl, few ? 1 : c->bX, few ? 1 : c->bY, few ? 1 : c->bZ, d_out, ndir, d0);
		ADDA_LAUNCHED();
	}
	ADDA_CUDA(cudaMemcpyAsync(ebuff, d_out, sizeof(double2) * 3 * (size_t)ndir * R, cudaMemcpyDeviceToHost, s));
	ADDA_CUDA(cudaStreamSynchronize(s));
	return ADDA_GB300_OK;
}

} // namespace adda
