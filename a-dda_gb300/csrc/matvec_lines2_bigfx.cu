// matvec_lines2_bigfx.cu - the fixed-point stages on two-pass transforms with a radix above 16.
#define ADDA_MATVEC_YZ_TU
#include "matvec_lines2.cuh"

namespace adda {
namespace mv {

int fx_fftz_big(adda_gb300_ctx *c, const MvGeom<double> &p, int mode, int ck, cudaStream_t st)
{
	if (mode == 2) return l2_z<ArFx, FX_W2, 2, FX_W1, RC_BIG>(c, p, ck, st);
	return mode ? l2_z<ArFx, FX_W2, 1, FX_W1, RC_BIG>(c, p, ck, st) : l2_z<ArFx, FX_W2, 0, FX_W1, RC_BIG>(c, p, ck, st);
}
int fx_ffty_big(adda_gb300_ctx *c, const MvGeom<double> &p, int ck, cudaStream_t st)
{
	return l2_y<ArFx, FX_W2, RC_BIG>(c, p, ck, 0, st);
}
int fx_scatter_big(adda_gb300_ctx *c, const MvP<double, double2> &p, cudaStream_t st)
{
	return l2_k1<ArFx, double2, FX_W1, FX_W2, RC_BIG>(c, p, st);
}
int fx_gather_big(adda_gb300_ctx *c, const MvP<double, double2> &p, const MvEpi &e, cudaStream_t st)
{
	return l2_k3<ArFx, double2, FX_W1, FX_W2, RC_BIG>(c, p, e, st);
}

} // namespace mv
} // namespace adda
