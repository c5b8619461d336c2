// Convolution plans (the passes: conv_passes.cuh).
#include "conv.cuh"
#include "tma.cuh"

namespace mm {

FftRadices fft_factor(int n)
{
	FftRadices f{};
	f.n = n;
	int m = n;
	auto push = [&](int r) { f.r[f.count++] = r; m /= r; };
	while (m % 8 == 0 && f.count < FFT_MAX_PASSES) push(8);
	while (m % 4 == 0 && f.count < FFT_MAX_PASSES) push(4);
	while (m % 2 == 0 && f.count < FFT_MAX_PASSES) push(2);
	for (int p : {3, 5, 7})
		while (m % p == 0 && f.count < FFT_MAX_PASSES) push(p);
	for (int p = 11; m > 1 && f.count < FFT_MAX_PASSES; p += 2)
		while (m % p == 0 && f.count < FFT_MAX_PASSES) push(p);
	if (m != 1) f.count = -1;  // too many factors (cannot happen for n < 2^24)
	return f;
}

// ---- parts of a tensor by parity -------------------------------------------------------------------
namespace {

// The eight values of component c at (+-i, +-j, +-k), index bits x, y, z: mirrored.
__device__ __forceinline__ void mirrored(const double *__restrict__ N, int3 e, int c, int i, int j, int k, double (&v)[8])
{
	const int x[2] = {i, i ? e.x - i : 0}, y[2] = {j, j ? e.y - j : 0}, z[2] = {k, k ? e.z - k : 0};
#pragma unroll
	for (int s = 0; s < 8; ++s) v[s] = N[(((size_t)z[s >> 2] * e.y + y[s >> 1 & 1]) * e.x + x[s & 1]) * 6 + c];
}
__device__ __forceinline__ double part(const double (&v)[8], int parity)
{
	double sum = 0;
#pragma unroll
	for (int s = 0; s < 8; ++s) sum += __popc(parity & s) & 1 ? -v[s] : v[s];
	return 0.125 * sum;
}

// A block takes a stretch of one row (j, k) of the octant, a thread an entry, the components and then x fastest:
// both directions of every axis are read in whole lines, once, and a row costs no division per entry.
__global__ void __launch_bounds__(256) k_tensor_part(const double *__restrict__ N, int3 e, int3 m, int q, double *__restrict__ out)
{
	const int t = blockIdx.x * 256 + threadIdx.x, c = t % 6, i = t / 6;
	if (i >= m.x) return;
	for (int k = blockIdx.z; k < m.z; k += gridDim.z)
		for (int j = blockIdx.y; j < m.y; j += gridDim.y) {
			double v[8];
			mirrored(N, e, c, i, j, k, v);
			out[((size_t)k * m.y + j) * m.x * 6 + t] = part(v, component_parity(c) ^ q);
		}
}

// most[0]: the largest entry, most[1]: the largest of parts 3, 5 and 6
__global__ void __launch_bounds__(256) k_tensor_parity(const double *__restrict__ N, int3 e, int3 m, double *most)
{
	const int t = blockIdx.x * 256 + threadIdx.x, c = t % 6, i = t / 6;
	double all = 0, other = 0;
	if (i < m.x)
		for (int k = blockIdx.z; k < m.z; k += gridDim.z)
			for (int j = blockIdx.y; j < m.y; j += gridDim.y) {
				double v[8];
				mirrored(N, e, c, i, j, k, v);
#pragma unroll
				for (int s = 0; s < 8; ++s) all = fmax(all, fabs(v[s]));
				for (int q : {3, 5, 6}) other = fmax(other, fabs(part(v, component_parity(c) ^ q)));
			}
	block_max_to(most, all);
	__syncthreads();
	block_max_to(most + 1, other);
}

// Blocks over the rows: a few rows each where there are many, to keep the maxima's atomic updates few.
dim3 part_grid(const int (&m)[3])
{
	const int x = (6 * m[0] + 255) / 256, rows = (num_sms() * 32 + x - 1) / x;
	const int y = m[1] < rows ? m[1] : rows;
	const int z = (rows + y - 1) / y;
	return dim3(x, y, m[2] < z ? m[2] : z);
}

} // namespace

mm_status tensor_part(const double *N, const int (&e)[3], const int (&m)[3], int q, double *out, cudaStream_t st)
{
	k_tensor_part<<<part_grid(m), 256, 0, st>>>(N, make_int3(e[0], e[1], e[2]), make_int3(m[0], m[1], m[2]), q, out);
	return after_launch("k_tensor_part");
}

mm_status tensor_mixed_parity(const double *N, const int (&e)[3], bool *mixed, cudaStream_t st)
{
	const int m[3] = {e[0] / 2 + 1, e[1] / 2 + 1, e[2] / 2 + 1};
	double *most = nullptr, h[2] = {0, 0};
	MM_TRY(setup_alloc((void **)&most, sizeof(h), st));
	mm_status r = cuda_status(cudaMemsetAsync(most, 0, sizeof(h), st), "cudaMemsetAsync");
	if (r == MM_OK) {
		k_tensor_parity<<<part_grid(m), 256, 0, st>>>(N, make_int3(e[0], e[1], e[2]), make_int3(m[0], m[1], m[2]), most);
		r = after_launch("k_tensor_parity");
	}
	if (r == MM_OK) r = cuda_status(cudaMemcpyAsync(h, most, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
	setup_free(most, st);
	if (r == MM_OK) r = cuda_status(cudaStreamSynchronize(st), "cudaStreamSynchronize");
	// (entries that vanish by symmetry are sums of a few rounded terms)
	*mixed = h[1] > 8 * 0x1p-53 * h[0];
	return r;
}

size_t ConvPlan::spec_bytes() const
{
	const size_t c = prec == MM_F64 ? sizeof(double2) : sizeof(float2);
	return c * 3 * (size_t)nz * py * lx;
}

mm_status tma_encode(CUtensorMap *map, const void *base, int rank, const uint64_t *dims, const uint64_t *strides,
                     const uint32_t *box)
{
	return tma_encode_as(map, base, rank, dims, strides, box, 8);
}

mm_status tma_encode_as(CUtensorMap *map, const void *base, int rank, const uint64_t *dims, const uint64_t *strides,
                        const uint32_t *box, int esize)
{
	using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
	                            const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
	                            CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
	static Encode encode = nullptr;
	if (!encode) {
		void *fn = nullptr;
		cudaDriverEntryPointQueryResult q{};
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
		    q != cudaDriverEntryPointSuccess || !fn) {
			cudaGetLastError();
			return fail(MM_ERR_UNSUPPORTED, "conv: cuTensorMapEncodeTiled is not available from the driver");
		}
		encode = reinterpret_cast<Encode>(fn);
	}
	if (esize != 1 && esize != 4 && esize != 8) return fail(MM_ERR_INVALID_ARGUMENT, "tensor map element size");
	if (rank < 1 || rank > 5 || (reinterpret_cast<uintptr_t>(base) & 15) || ((box[0] * esize) & 15))
		return fail(MM_ERR_INVALID_ARGUMENT, "conv: tensor map not 16-byte aligned");
	cuuint64_t d[5], sb[4];
	cuuint32_t bx[5], estr[5];
	for (int i = 0; i < rank; ++i) {
		d[i] = dims[i];
		bx[i] = box[i];
		estr[i] = 1;
		if (box[i] < 1 || box[i] > 256) return fail(MM_ERR_INVALID_ARGUMENT, "conv: tensor map box beyond 256");
	}
	for (int i = 0; i + 1 < rank; ++i) {
		sb[i] = strides[i];
		if (strides[i] & 15) return fail(MM_ERR_INVALID_ARGUMENT, "conv: tensor map stride not 16-byte aligned");
	}
	const CUtensorMapDataType dt = esize == 1   ? CU_TENSOR_MAP_DATA_TYPE_UINT8
	                               : esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32
	                                            : CU_TENSOR_MAP_DATA_TYPE_UINT64;
	const CUresult r = encode(map, dt, (cuuint32_t)rank, const_cast<void *>(base), d, sb,
	                          bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
	                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS)
		return fail(MM_ERR_CUDA, "conv: cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
	return MM_OK;
}

mm_status tma_encode_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                        uint64_t stride1, uint64_t stride2, uint32_t b0, uint32_t b1, uint32_t b2)
{
	const uint64_t dims[3] = {d0, d1, d2}, strides[2] = {stride1, stride2};
	const uint32_t box[3] = {b0, b1, b2};
	return tma_encode(map, base, 3, dims, strides, box);
}

ConvPlan::~ConvPlan()
{
	cudaFree(tw_x);
	cudaFree(tw_y);
	cudaFree(tw_z);
	cudaFree(tensor);
	cudaFree(tensor_kx);
	cudaFree(spec);
	cudaFree(err);
}

int conv_launches(const ConvPlan *p) { return p->is2d ? 3 : 5; }

// The plan of n cells and a tensor of layout e at FFT lengths `len`.
static mm_status plan_at(ConvPlan **out, int prec, const int (&n)[3], const int (&e)[3], const int (&len)[3], bool mixed,
                         const double *N, bool octant, cudaStream_t st)
{
	const int px = len[0], py = len[1], pz = len[2];
	ConvPlan *p = new ConvPlan();
	p->prec = prec;
	p->nx = n[0]; p->ny = n[1]; p->nz = n[2];
	p->ex = e[0]; p->ey = e[1]; p->ez = e[2];
	p->px = px; p->py = py; p->pz = pz;
	p->hx = px / 2 + 1;
	{
		// row stride: 8-byte elements per row a multiple of 2 * xbox_n, so that a row splits into
		// xbox_n TMA boxes of xbox_w (even, <= 256) elements with 16-byte aligned rows
		const int E = prec == MM_F32 ? 1 : 2;
		int w = p->hx * E;
		const int nb = (w + 255) / 256;
		w = (w + 2 * nb - 1) / (2 * nb) * (2 * nb);
		p->lx = w / E;
		p->xbox_n = nb;
		p->xbox_w = w / nb;
	}
	p->qy = py / 2 + 1;
	p->qz = pz / 2 + 1;
	p->is2d = (n[2] == 1 && pz == 1);
	p->mixed_parity = mixed;
	p->rx = fft_factor(px);
	p->ry = fft_factor(py);
	p->rz = fft_factor(pz);
	if (p->rx.count < 0 || p->ry.count < 0 || p->rz.count < 0) {
		delete p;
		return fail(MM_ERR_UNSUPPORTED, "conv: FFT length has too many prime factors");
	}
	const mm_status s = prec == MM_F64 ? conv_setup_f64(p, N, octant, st) : conv_setup_f32(p, N, octant, st);
	if (s != MM_OK) {
		delete p;
		return s;
	}
	*out = p;
	return MM_OK;
}

mm_status conv_plan_create(ConvPlan **out, int prec, int nx, int ny, int nz, int ex, int ey, int ez,
                           const double *N, cudaStream_t st, bool keep_lengths, bool octant)
{
	if (prec != MM_F64 && prec != MM_F32) return fail(MM_ERR_INVALID_ARGUMENT, "conv: bad precision");
	if (nx <= 0 || ny <= 0 || nz <= 0 || ex < nx || ey < ny || ez < nz || !N ||
	    (octant && (ex < 2 * nx - 1 || ey < 2 * ny - 1 || ez < 2 * nz - 1)))
		return fail(MM_ERR_INVALID_ARGUMENT, "conv: invalid sizes or null tensor");
	const int n[3] = {nx, ny, nz}, e[3] = {ex, ey, ez};
	bool mixed = false;
	if (!octant) MM_TRY(tensor_mixed_parity(N, e, &mixed, st));
	keep_lengths = keep_lengths || mixed;  // (its spectrum depends on the length)
	int len[3] = {ex, ey, ez};
	if (!keep_lengths) (prec == MM_F64 ? conv_lengths_f64 : conv_lengths_f32)(n, e, len);
	const mm_status r = plan_at(out, prec, n, e, len, mixed, N, octant, st);
	if (r != MM_ERR_OUT_OF_MEMORY || (len[0] == ex && len[1] == ey && len[2] == ez)) return r;
	// the plan's lengths need up to 2.2 times the spectrum and 3.4 times the tensor of the tensor's own
	cudaGetLastError();
	clear_error();
	return plan_at(out, prec, n, e, e, mixed, N, octant, st);
}

mm_status conv_execute(ConvPlan *p, const void *M, const uint8_t *regions, const void *ms_table,
                       void *H, cudaStream_t st)
{
	if (p->prec == MM_F64)
		return conv_run_f64(p, (const double *)M, regions, (const double *)ms_table, (double *)H, st);
	return conv_run_f32(p, (const float *)M, regions, (const float *)ms_table, (float *)H, st);
}

} // namespace mm
