// Zero-padded FFT convolution H = N * M with the symmetric demag tensor (internal API).
#pragma once

#include <cuda.h>

#include "mm_common.cuh"
#include "fft.cuh"

namespace mm {

struct ConvPlan {
	int prec = MM_F64;
	int nx = 0, ny = 0, nz = 0;     // grid
	int ex = 0, ey = 0, ez = 0;     // padded lengths of the tensor's layout
	int px = 0, py = 0, pz = 0;     // FFT lengths (an axis the tensor pads may take another length)
	int hx = 0;                     // px/2 + 1 stored x frequencies
	int lx = 0;                     // spectrum row stride (>= hx complex, rows 16-byte aligned)
	int xbox_n = 1, xbox_w = 0;     // a spectrum row as xbox_n TMA boxes of xbox_w 8-byte elements
	int qy = 0, qz = 0;             // py/2 + 1, pz/2 + 1 stored tensor frequencies
	bool is2d = false;              // nz == 1 && pz == 1
	bool mixed_parity = false;      // the tensor has parts of other parities (tensor_mixed_parity)
	bool fast_x = false, fast_y = false, fast_z = false;  // compile-time register-FFT passes (2^k, 3 * 2^k)
	bool reg_z = false;             // z pass with whole columns in registers (nz <= pz/2, pz up to 32)
	bool tma_y = false;             // y passes fed by TMA-staged tiles (persistent CTAs)
	CUtensorMap tm_yf{}, tm_yi{};   // spectrum views of the forward (ny rows) and inverse (py rows) y pass
	int grid_yf = 0, grid_yi = 0;   // persistent grid sizes of those passes
	int *err = nullptr;             // device word set when a bounded wait of a staged pass gave up
	bool tma_xf = false, tma_xi = false;  // x passes fed by TMA-staged tiles
	bool tma_xf_scale = false;            // ... also with the Ms[region] input scale
	int grid_xf = 0, grid_xi = 0;
	int xf_box_n = 1, xf_box_w = 0;       // a real input row as boxes of 8-byte elements
	CUtensorMap tm_xi{};                  // spectrum rows y < ny of each plane, for the inverse x pass
	static constexpr int XF_CACHE = 4;    // forward-pass maps, one per input buffer seen
	const void *xf_ptr[XF_CACHE] = {};
	CUtensorMap xf_map[XF_CACHE] = {};
	int xf_next = 0;
	const void *xr_ptr = nullptr;         // region map the region tensor map was encoded for
	CUtensorMap xr_map{};                 // region bytes of the forward pass's rows
	FftRadices rx{}, ry{}, rz{};
	void *tw_x = nullptr, *tw_y = nullptr, *tw_z = nullptr;  // cplx<T> twiddle tables (plain, then per pass)
	void *tensor = nullptr;         // reduced real tensor spectrum, T[6][qz][qy][hx]
	void *tensor_kx = nullptr;      // the same, kx-major T[hx][qz][qy][6] (made by the first grouped
	                                // convolution whose fused y+z pass takes this plan)
	void *spec = nullptr;           // cplx<T>[3][nz][py][lx]
	// launch geometry
	int lp_x = 1;                   // complex lines (= 2 real rows) per CTA in the x passes
	int tb_y = 1, tb_z = 1;         // columns per CTA in the y and z passes
	size_t smem_x = 0, smem_y = 0, smem_z = 0;

	size_t spec_bytes() const;
	~ConvPlan();
};

// Builds the plan and the tensor spectrum from an FP64 tensor in the reference layout
// (component fastest, then x, y, z) of padded size ex*ey*ez.  The FFT lengths of zero-padded axes are
// the plan's choice (keep_lengths: the tensor's own, as the grouped passes need powers of two).
// octant: N holds only the offsets >= 0 of a box without periodic axes, [nz][ny][nx][6].
mm_status conv_plan_create(ConvPlan **out, int prec, int nx, int ny, int nz, int ex, int ey,
                           int ez, const double *N_device, cudaStream_t st, bool keep_lengths = false,
                           bool octant = false);

// The components xx, xy, xz, yy, yz, zz of a demagnetising tensor are even or odd along each axis (bits x, y,
// z: odd), which the plan's spectrum relies on.  A tensor that is handed in may have parts of other
// parities; sorted by what they are multiplied with, part q of component c has the parity c's own ^ q.
//   q with an odd number of bits: not symmetric under inversion; the transform's real part leaves it out
//   q = 3, 5, 6: the real part contains it
__host__ __device__ constexpr int component_parity(int c) { return c == 1 ? 3 : c == 2 ? 5 : c == 4 ? 6 : 0; }
// Whether the tensor (layout e) has parts 3, 5 or 6 beyond the rounding of its largest entry; waits.
mm_status tensor_mixed_parity(const double *N, const int (&e)[3], bool *mixed, cudaStream_t st);
// Part q at the offsets [0, m) of each axis, out[m2][m1][m0][6].
mm_status tensor_part(const double *N, const int (&e)[3], const int (&m)[3], int q, double *out, cudaStream_t st);

// The tensor's octant of offsets >= 0 of a box without periodic axes, [nz][ny][nx][6] (tensor.cu).
mm_status tensor_octant(int nx, int ny, int nz, double dx, double dy, double dz, double *N, cudaStream_t st);

// H = N * (Ms[region] * M) when regions/ms_table are given (ms_table: 256 entries), else H = N * M.
// M and H are SoA arrays of T (T = double for MM_F64, float for MM_F32).
mm_status conv_execute(ConvPlan *p, const void *M, const uint8_t *regions, const void *ms_table,
                       void *H, cudaStream_t st);

// Number of kernel launches one conv_execute issues.
int conv_launches(const ConvPlan *p);

// Grouped convolution over many plans of the same precision, each with power-of-two 3-D padding
// and a register z pass: one launch per pass and transform length covers every member.  M[k]
// are up to four candidate inputs per member and H[k] up to two outputs (each selected per call;
// H[1] may be NULL, then only output 0 is allowed); flags (device, optional) are the member's run
// flags: flags[0] == 0 skips it, and with gate != 0 so does flags[gate] == 0.
struct ConvGroup;
struct ConvGroupMember {
	ConvPlan *plan;
	const void *M[4];
	void *H[2];
	const uint8_t *reg;
	const void *ms_tab;  // 256 entries
	const int *flags;    // device run flags, NULL: always run
	const void *ms_uniform;  // the one entry that scales every cell (inputs zero where Ms is zero); NULL: by region
};
mm_status conv_group_create(ConvGroup **out, const ConvGroupMember *members, int count, cudaStream_t st);
mm_status conv_group_execute(ConvGroup *g, int input, int gate, cudaStream_t st, int output = 0);
void conv_group_destroy(ConvGroup *g);
// Whether a member with these padded lengths takes the grouped fused y+z pass (which keeps a
// second, kx-major copy of its reduced tensor).
int conv_group_fused(int prec, int py, int pz, int nz);

FftRadices fft_factor(int n);

// Twiddles of a plan's axis: a plain table and one per set of pass tables.
constexpr int TW_SETS = 3;
inline size_t conv_twiddle_entries(int px, int py, int pz) { return (size_t)TW_SETS * (px + py + pz); }

// conv_f64.cu, conv_f32.cu (flags, gate: a batch member's run flags, see ConvGroupMember)
mm_status conv_setup_f64(ConvPlan *p, const double *N, bool octant, cudaStream_t st);
mm_status conv_run_f64(ConvPlan *p, const double *M, const uint8_t *reg, const double *ms_tab, double *H, cudaStream_t st,
                       const int *flags = nullptr, int gate = 0);
void conv_lengths_f64(const int (&n)[3], const int (&e)[3], int (&p)[3]);
mm_status conv_setup_f32(ConvPlan *p, const double *N, bool octant, cudaStream_t st);
mm_status conv_run_f32(ConvPlan *p, const float *M, const uint8_t *reg, const float *ms_tab, float *H, cudaStream_t st,
                       const int *flags = nullptr, int gate = 0);
void conv_lengths_f32(const int (&n)[3], const int (&e)[3], int (&p)[3]);

} // namespace mm
