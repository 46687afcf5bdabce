// matvec_lines2_x.cu - K1 and K3 on two-pass transforms (matvec_lines2.cuh): FP32 arithmetic for the three dipole-vector
// types, and FP64 in fixed point.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {
namespace mv {

template <typename V> int l2_scatter_run(adda_gb300_ctx *c, const MvP<float, V> &p, int w1, dim3 g, cudaStream_t st)
{
	const Lines2<Ar32> q = make_lines2<Ar32>(c);
	const int nt = l2_threads(3 * w1, c->p2[0]);
	const size_t sm = l2_xtile_smem<Ar32>(c->bX, c->p2[0], w1);
	if (w1 == 4) launch_next((l2_scatter_x<Ar32, V, 4, 16>), g, nt, sm, st, p, q);
	else launch_next((l2_scatter_x<Ar32, V, 8, 16>), g, nt, sm, st, p, q);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

template <typename V>
int l2_gather_run(adda_gb300_ctx *c, const MvP<float, V> &p, int w1, dim3 g, const MvEpi &e, cudaStream_t st)
{
	const Lines2<Ar32> q = make_lines2<Ar32>(c);
	const int nt = l2_threads(3 * w1, c->p2[0]);
	const size_t sm = l2_xtile_smem<Ar32>(c->bX, c->p2[0], w1);
	if (w1 == 4) launch_next((l2_gather_x<Ar32, V, 4, 16>), g, nt, sm, st, p, q, e);
	else launch_next((l2_gather_x<Ar32, V, 8, 16>), g, nt, sm, st, p, q, e);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

#define ADDA_L2_INST(V)                                                                                              \
	template int l2_scatter_run<V>(adda_gb300_ctx *, const MvP<float, V> &, int, dim3, cudaStream_t);               \
	template int l2_gather_run<V>(adda_gb300_ctx *, const MvP<float, V> &, int, dim3, const MvEpi &, cudaStream_t);
ADDA_L2_INST(float2)
ADDA_L2_INST(double2)
ADDA_L2_INST(dd2)

int fx_scatter_run(adda_gb300_ctx *c, const MvP<double, double2> &p, cudaStream_t st)
{
	constexpr int W1 = FX_W1, W2 = FX_W2;
	const dim3 g((c->bY + W1 - 1) / W1, c->bZ, p.R);
	launch_next((l2_scatter_x<ArFx, double2, W1, W2>), g, l2_threads(3 * W1, c->p2[0]), l2_xtile_smem<ArFx>(c->bX, c->p2[0], W1), st, p,
		make_lines2<ArFx>(c));
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

int fx_gather_run(adda_gb300_ctx *c, const MvP<double, double2> &p, const MvEpi &e, cudaStream_t st)
{
	constexpr int W1 = FX_W1, W2 = FX_W2;
	const dim3 g((c->bY + W1 - 1) / W1, c->bZ, p.R);
	launch_next((l2_gather_x<ArFx, double2, W1, W2>), g, l2_threads(3 * W1, c->p2[0]), l2_xtile_smem<ArFx>(c->bX, c->p2[0], W1), st, p,
		make_lines2<ArFx>(c), e);
	ADDA_LAUNCHED();
	return ADDA_GB300_OK;
}

template <typename V> static int setup_v()
{
	ADDA_L2_SMEM((l2_scatter_x<Ar32, V, 4, 16>));
	ADDA_L2_SMEM((l2_scatter_x<Ar32, V, 8, 16>));
	ADDA_L2_SMEM((l2_gather_x<Ar32, V, 4, 16>));
	ADDA_L2_SMEM((l2_gather_x<Ar32, V, 8, 16>));
	return ADDA_GB300_OK;
}

int l2_setup_x()
{
	constexpr int W1 = FX_W1, W2 = FX_W2;
	int rc;
	if ((rc = setup_v<float2>()) || (rc = setup_v<double2>()) || (rc = setup_v<dd2>())) return rc;
	ADDA_L2_SMEM((l2_scatter_x<ArFx, double2, W1, W2>));
	ADDA_L2_SMEM((l2_gather_x<ArFx, double2, W1, W2>));
	return ADDA_GB300_OK;
}

} // namespace mv
} // namespace adda
