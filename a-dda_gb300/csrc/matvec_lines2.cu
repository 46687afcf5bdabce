// matvec_lines2.cu - the matvec's y/z stage on two-pass transforms (matvec_lines2.cuh) in both arithmetics, and D in
// fixed point.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {

size_t fx_exps_ints(const adda_gb300_ctx *c)
{
	size_t n;
	mv::fx_tables(c, &n);
	return n;
}

namespace mv {

// one row (kx, kz) of D per block: the row's largest exponent, then every component scaled to |v| < 2^60 and split
__global__ void __launch_bounds__(128) fx_drow(const double2 *D, int4 *Dfx, int *eD, int n)
{
	__shared__ int smax;
	if (threadIdx.x == 0) smax = 0;
	__syncthreads();
	D += (size_t)blockIdx.x * n;
	Dfx += (size_t)blockIdx.x * n;
	int h = 0;
	for (int t = threadIdx.x; t < n; t += blockDim.x) {
		const double2 d = D[t];
		h = max(h, max(__double2hiint(d.x) & 0x7fffffff, __double2hiint(d.y) & 0x7fffffff));
	}
	h = block_max(h, &smax);
	const int emax = max(1, h >> 20), up = 60 - FX_TOP;
	for (int t = threadIdx.x; t < n; t += blockDim.x) {
		const double2 d = D[t];
		int v[4];
		const double part[2] = {d.x, d.y};
#pragma unroll
		for (int k = 0; k < 2; k++) {
			// 53 bits and 7 more below them
			const int hi = __double2hiint(part[k]), ex = (hi >> 20) & 0x7ff, sh = emax - max(ex, 1);
			const long long m = ((long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(part[k]);
			long long w = sh > 63 ? 0 : (m << (up + FX_TOP - 53)) >> sh;
			if (hi < 0) w = -w;
			const int lo = max((int)w, -0x7fffffff);
			v[2 * k] = lo;
			v[2 * k + 1] = (int)((w - lo + 1) >> 32);
		}
		Dfx[t] = make_int4(v[0], v[1], v[2], v[3]);
	}
	if (threadIdx.x == 0) eD[blockIdx.x] = h >= 0x7ff00000 ? FX_BAD : emax - 1075 - (up + FX_TOP - 53);
}

int l2_fftz_run(adda_gb300_ctx *c, const MvGeom<float> &p, int mode, int w2, dim3 g, cudaStream_t st)
{
	const Lines2<Ar32> q = make_lines2<Ar32>(c);
	const int nt = l2_threads(w2, c->p2[2]);
	const size_t sm = l2_z_smem<Ar32>(c->p2[2], w2);
#define ADDA_L2Z(W, MODE)                                                                                            \
	if (w2 == W && mode == MODE) launch_next((l2_fftz<Ar32, W, MODE, 8>), g, nt, sm, st, p, q);
	ADDA_L2Z(8, 0) ADDA_L2Z(8, 1) ADDA_L2Z(8, 2) ADDA_L2Z(16, 0) ADDA_L2Z(16, 1) ADDA_L2Z(16, 2)
	ADDA_L2Z(32, 0) ADDA_L2Z(32, 1) ADDA_L2Z(32, 2)
#undef ADDA_L2Z
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

int l2_ffty_run(adda_gb300_ctx *c, const MvGeom<float> &p, int ck, int pairs, cudaStream_t st)
{
	const Lines2<Ar32> q = make_lines2<Ar32>(c);
	const int P = std::max(c->p2[1].r1, c->p2[1].r2), G = pairs;
	const dim3 g((c->gZ * p.R + G - 1) / G, ck);
	launch_next((l2_fft_y<Ar32, 16>), g, (3 * G * P + 31) / 32 * 32, l2_y_smem<Ar32>(c->p2[1], G), st, p, q, G, P);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

int fx_yz_run(adda_gb300_ctx *c, const MvGeom<double> &p, int ck, cudaStream_t st)
{
	constexpr int W1 = FX_W1, W2 = FX_W2;
	const Lines2<ArFx> q = make_lines2<ArFx>(c);
	const dim3 g2((c->bY + W2 - 1) / W2, 3 * ck, p.R);
	const int ntz = l2_threads(W2, c->p2[2]);
	const size_t smz = l2_z_smem<ArFx>(c->p2[2], W2);
	launch_next((l2_fftz<ArFx, W2, 0, W1>), g2, ntz, smz, st, p, q);
	ADDA_LAUNCHED();
	const int P = std::max(c->p2[1].r1, c->p2[1].r2), G = std::min(8, 128 / (3 * P));
	const dim3 g((c->gZ * p.R + G - 1) / G, ck);
	launch_next((l2_fft_y<ArFx, W2>), g, (3 * G * P + 31) / 32 * 32, l2_y_smem<ArFx>(c->p2[1], G), st, p, q, G, P);
	ADDA_LAUNCHED();
	launch_next((l2_fftz<ArFx, W2, 1, W1>), g2, ntz, smz, st, p, q);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

int l2_setup_yz()
{
	constexpr int W1 = FX_W1, W2 = FX_W2;
	ADDA_L2_SMEM((l2_fftz<ArFx, W2, 0, W1>));
	ADDA_L2_SMEM((l2_fftz<ArFx, W2, 1, W1>));
	ADDA_L2_SMEM((l2_fft_y<ArFx, W2>));
	ADDA_L2_SMEM((l2_fft_y<Ar32, 16>));
	ADDA_L2_SMEM((l2_fftz<Ar32, 32, 0, 8>));
	ADDA_L2_SMEM((l2_fftz<Ar32, 32, 1, 8>));
	ADDA_L2_SMEM((l2_fftz<Ar32, 32, 2, 8>));
	return ADDA_GB300_OK;
}

} // namespace mv

int fx_dmatrix(adda_gb300_ctx *c)
{
	mv::fx_drow<<<c->gX * c->DsZ, 128, 0, c->stream>>>(c->D64, (int4 *)c->Dfx, c->fx_eD, c->DsY * 6);
	ADDA_LAUNCHED();
	ADDA_CUDA(cudaStreamSynchronize(c->stream));
	return ADDA_GB300_OK;
}

} // namespace adda
