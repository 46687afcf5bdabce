// matvec_lines2_big.cu - the FP32 stages on two-pass transforms with a radix above 16 (axis lengths such as 162, 200, 220
// and most between 256 and 512). One width each: L2_BIG_W1 y-lines per K1/K3 block, 16 per K2a/K2c block.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {
namespace mv {

int l2_fftz_big(adda_gb300_ctx *c, const MvGeom<float> &p, int mode, int ck, cudaStream_t st)
{
	if (mode == 0) return l2_z<Ar32, 16, 0, 8, RC_BIG>(c, p, ck, st);
	if (mode == 1) return l2_z<Ar32, 16, 1, 8, RC_BIG>(c, p, ck, st);
	return l2_z<Ar32, 16, 2, 8, RC_BIG>(c, p, ck, st);
}
int l2_ffty_big(adda_gb300_ctx *c, const MvGeom<float> &p, int ck, int pairs, cudaStream_t st)
{
	return l2_y<Ar32, 16, RC_BIG>(c, p, ck, pairs, st);
}
template <typename V> int l2_scatter_big(adda_gb300_ctx *c, const MvP<float, V> &p, cudaStream_t st)
{
	return l2_k1<Ar32, V, L2_BIG_W1, 16, RC_BIG>(c, p, st);
}
template <typename V> int l2_gather_big(adda_gb300_ctx *c, const MvP<float, V> &p, const MvEpi &e, cudaStream_t st)
{
	return l2_k3<Ar32, V, L2_BIG_W1, 16, RC_BIG>(c, p, e, st);
}
#define ADDA_L2_INST(V)                                                                                              \
	template int l2_scatter_big<V>(adda_gb300_ctx *, const MvP<float, V> &, cudaStream_t);                          \
	template int l2_gather_big<V>(adda_gb300_ctx *, const MvP<float, V> &, const MvEpi &, cudaStream_t);
ADDA_L2_INST(float2)
ADDA_L2_INST(double2)
ADDA_L2_INST(dd2)

} // namespace mv
} // namespace adda
