// The convolution's passes in single precision.
#include "conv_passes.cuh"

namespace mm {

mm_status conv_setup_f32(ConvPlan *p, const double *N, bool octant, cudaStream_t st) { return plan_setup<float>(p, N, octant, st); }

mm_status conv_run_f32(ConvPlan *p, const float *M, const uint8_t *reg, const float *ms_tab, float *H, cudaStream_t st, const int *flags, int gate)
{
	return execute<float>(p, M, reg, ms_tab, H, st, Gate{flags, gate});
}

void conv_lengths_f32(const int (&n)[3], const int (&e)[3], int (&p)[3]) { choose_lengths<float>(n, e, p); }

} // namespace mm
