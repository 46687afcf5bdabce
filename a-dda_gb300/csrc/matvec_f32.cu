// matvec_f32.cu - FP32-arithmetic instantiations of the matvec kernels (float2, double2 and double-float dipole
// vectors).
#include "matvec_kernels.cuh"

namespace adda {

namespace {

// K1 and K3 for one vector type: the two-pass kernels of the x axis where it takes them, and the others, which any axis may
// fall back to with a narrow tile shape
template <typename V> int prepare_x(adda_gb300_ctx *c)
{
	int rc = mv::set_attrs_tv<float, V>(c);
	if (!mv::use_l2_f32(c, 0, c->gX)) return rc;
	mv::MvP<float, V> p{};
	for (int w1 : {4, 8})
		if (rc || (rc = mv::l2_scatter_run<V>(c, p, w1, c->stream)) || (rc = mv::l2_gather_run<V>(c, p, w1, MvEpi{}, c->stream)))
			return rc;
	return rc;
}

} // namespace

int matvec_setup_f32(adda_gb300_ctx *c)
{
	int rc = mv::setup_yz<float>(c);
	if (rc || (rc = prepare_x<float2>(c)) || (rc = prepare_x<double2>(c)) || (rc = prepare_x<dd2>(c))) return rc;
	const mv::MvGeom<float> g{};
	if (mv::use_l2_f32(c, 2, c->gZ))
		for (int w2 : {8, 16, 32})
			for (int mode : {0, 1, 2})
				if ((mode < 2 || c->surface) && (rc = mv::l2_fftz_run(c, g, mode, w2, 1, c->stream))) return rc;
	return mv::use_l2_y(c) ? mv::l2_ffty_run(c, g, 1, 8, c->stream) : rc;
}

template <typename T, typename V>
int matvec_run(adda_gb300_ctx *c, int R, const V *arg, V *res, int her, const MvEpi &epi, const int *done)
{
	return mv::launch_matvec<T, V>(c, R, arg, res, her, epi, done);
}

template int matvec_run<float, float2>(adda_gb300_ctx *, int, const float2 *, float2 *, int, const MvEpi &,
	const int *);
template int matvec_run<float, double2>(adda_gb300_ctx *, int, const double2 *, double2 *, int, const MvEpi &,
	const int *);
template int matvec_run<float, dd2>(adda_gb300_ctx *, int, const dd2 *, dd2 *, int, const MvEpi &, const int *);

} // namespace adda
