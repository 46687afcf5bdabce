// matvec_lines2.cu - the matvec's y/z stage on two-pass transforms (matvec_lines2.cuh) in both arithmetics, and D in
// fixed point.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {

bool matvec_same_kernels(const adda_gb300_ctx *c, const MvShape &a, const MvShape &b)
{
	// x and z axes with a radix above 16 have one width; the two-pass y kernel as many columns as its threads allow
	const bool x = a.w1 == b.w1 || (mv::use_l2_x(c, a) && mv::use_l2_x(c, b) && c->p2[0].big);
	const bool z = a.w2 == b.w2 || (mv::use_l2_z(c, a) && mv::use_l2_z(c, b) && c->p2[2].big);
	const auto columns = [&](const MvShape &s) {
		return mv::l2_columns<Ar32>(c->p2[1], c->surface ? std::max(1, s.pairs / 2) : s.pairs);
	};
	const bool y = a.pairs == b.pairs || (mv::use_l2_y(c) && columns(a) == columns(b));
	return x && y && z && a.nt == b.nt;
}

size_t fx_exps_ints(const adda_gb300_ctx *c)
{
	size_t n;
	mv::fx_tables(c, &n);
	return n;
}

namespace mv {

// one row (kx, kz) of D per block: the row's largest exponent, then every component scaled to |v| < 2^60 and split. Dfx may
// be D's own memory: a thread reads an entry before it writes that entry, all of them after the row's largest is known
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

int l2_fftz_run(adda_gb300_ctx *c, const MvGeom<float> &p, int mode, int w2, int ck, cudaStream_t st)
{
	if (c->p2[2].big) return l2_fftz_big(c, p, mode, ck, st);
#define ADDA_L2Z(W, MODE)                                                                                            \
	if (w2 == W && mode == MODE) return l2_z<Ar32, W, MODE, 8, RC_SMALL>(c, p, ck, st);
	ADDA_L2Z(8, 0) ADDA_L2Z(8, 1) ADDA_L2Z(8, 2) ADDA_L2Z(16, 0) ADDA_L2Z(16, 1) ADDA_L2Z(16, 2)
	ADDA_L2Z(32, 0) ADDA_L2Z(32, 1) ADDA_L2Z(32, 2)
#undef ADDA_L2Z
	return ADDA_GB300_EINVAL;
}

int l2_ffty_run(adda_gb300_ctx *c, const MvGeom<float> &p, int ck, int pairs, cudaStream_t st)
{
	return c->p2[1].big ? l2_ffty_big(c, p, ck, pairs, st) : l2_y<Ar32, 16, RC_SMALL>(c, p, ck, pairs, st);
}

int fx_yz_run(adda_gb300_ctx *c, const MvGeom<double> &p, int ck, cudaStream_t st)
{
	int rc = c->p2x[2].big ? fx_fftz_big(c, p, 0, ck, st) : l2_z<ArFx, FX_W2, 0, FX_W1, RC_SMALL>(c, p, ck, st);
	if (!rc && c->surface)
		rc = c->p2x[2].big ? fx_fftz_big(c, p, 2, ck, st) : l2_z<ArFx, FX_W2, 2, FX_W1, RC_SMALL>(c, p, ck, st);
	if (!rc) rc = c->p2x[1].big ? fx_ffty_big(c, p, ck, st) : l2_y<ArFx, FX_W2, RC_SMALL>(c, p, ck, 0, st);
	if (!rc) rc = c->p2x[2].big ? fx_fftz_big(c, p, 1, ck, st) : l2_z<ArFx, FX_W2, 1, FX_W1, RC_SMALL>(c, p, ck, st);
	return rc;
}

} // namespace mv

int fx_dmatrix(adda_gb300_ctx *c, const double2 *D, const double2 *R)
{
	if (D) {
		mv::fx_drow<<<c->gX * c->DsZ, 128, 0, c->stream>>>(D, (int4 *)c->Dfx, c->fx_eD, c->DsY * 6);
		ADDA_LAUNCHED();
	}
	if (R) {
		mv::fx_drow<<<c->gX * c->gZ, 128, 0, c->stream>>>(R, (int4 *)c->Rfx, c->fx_eD + (size_t)c->gX * c->DsZ, (c->gY / 2 + 1) * 6);
		ADDA_LAUNCHED();
	}
	ADDA_CUDA(cudaStreamSynchronize(c->stream));
	return ADDA_GB300_OK;
}

} // namespace adda
