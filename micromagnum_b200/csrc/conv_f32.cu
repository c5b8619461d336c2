// The convolution's passes in single precision.
#include "conv_passes.cuh"

namespace mm {

mm_status conv_setup_f32(ConvPlan *p, const double *N, bool octant, cudaStream_t st) { return plan_setup<float>(p, N, octant, st); }

mm_status conv_run_f32(ConvPlan *p, const float *M, const uint8_t *reg, const float *ms_tab, float *H, cudaStream_t st, const int *flags, int gate)
{
	return execute<float>(p, M, reg, ms_tab, H, st, Gate{flags, gate});
}

int conv_fit_length_f32(int n, int e, bool z) { return fit_length<float>(n, e, z); }

} // namespace mm
