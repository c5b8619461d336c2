// The convolution's passes in double precision.
#include "conv_passes.cuh"

namespace mm {

mm_status conv_setup_f64(ConvPlan *p, const double *N, bool octant, cudaStream_t st) { return plan_setup<double>(p, N, octant, st); }

mm_status conv_run_f64(ConvPlan *p, const double *M, const uint8_t *reg, const double *ms_tab, double *H, cudaStream_t st, const int *flags, int gate)
{
	return execute<double>(p, M, reg, ms_tab, H, st, Gate{flags, gate});
}

void conv_lengths_f64(const int (&n)[3], const int (&e)[3], int (&p)[3]) { choose_lengths<double>(n, e, p); }

} // namespace mm
