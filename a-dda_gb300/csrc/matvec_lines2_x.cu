// matvec_lines2_x.cu - K1 and K3 on two-pass transforms (matvec_lines2.cuh): FP32 arithmetic for the three dipole-vector
// types, and FP64 in fixed point.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {
namespace mv {

template <typename V> int l2_scatter_run(adda_gb300_ctx *c, const MvP<float, V> &p, int w1, cudaStream_t st)
{
	if (c->p2[0].big) return l2_scatter_big(c, p, st);
	return w1 == 4 ? l2_k1<Ar32, V, 4, 16, RC_SMALL>(c, p, st) : l2_k1<Ar32, V, 8, 16, RC_SMALL>(c, p, st);
}

template <typename V>
int l2_gather_run(adda_gb300_ctx *c, const MvP<float, V> &p, int w1, const MvEpi &e, cudaStream_t st)
{
	if (c->p2[0].big) return l2_gather_big(c, p, e, st);
	return w1 == 4 ? l2_k3<Ar32, V, 4, 16, RC_SMALL>(c, p, e, st) : l2_k3<Ar32, V, 8, 16, RC_SMALL>(c, p, e, st);
}

#define ADDA_L2_INST(V)                                                                                              \
	template int l2_scatter_run<V>(adda_gb300_ctx *, const MvP<float, V> &, int, cudaStream_t);                     \
	template int l2_gather_run<V>(adda_gb300_ctx *, const MvP<float, V> &, int, const MvEpi &, cudaStream_t);
ADDA_L2_INST(float2)
ADDA_L2_INST(double2)
ADDA_L2_INST(dd2)

int fx_scatter_run(adda_gb300_ctx *c, const MvP<double, double2> &p, cudaStream_t st)
{
	return c->p2x[0].big ? fx_scatter_big(c, p, st) : l2_k1<ArFx, double2, FX_W1, FX_W2, RC_SMALL>(c, p, st);
}

int fx_gather_run(adda_gb300_ctx *c, const MvP<double, double2> &p, const MvEpi &e, cudaStream_t st)
{
	return c->p2x[0].big ? fx_gather_big(c, p, e, st) : l2_k3<ArFx, double2, FX_W1, FX_W2, RC_SMALL>(c, p, e, st);
}

} // namespace mv
} // namespace adda
