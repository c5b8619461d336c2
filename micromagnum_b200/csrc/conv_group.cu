// Grouped convolution over many plans (see conv.cuh).
#include "conv_passes.cuh"

namespace mm {

// ---- grouped convolution: many plans, one launch per pass and transform length -------------------
// Every member plan uses the power-of-two passes (register z pass included).  The members' blocks
// of one pass and one length form a work list (member, block); a member whose run flag is 0
// skips its blocks, so finished instances drop out without rebuilding the lists.
namespace {

template <typename T>
struct GDesc {
	cplx<T> *spec;
	const T *tensor;
	const T *tensor_t;  // fused y+z members: the reduced tensor kx-major, [hx][qz][qy][6]
	const cplx<T> *tw_x, *tw_y;
	const T *M[4];
	T *H[2];
	const uint8_t *reg;
	const T *ms_tab;
	const int *flags;   // the member's run flags: [0] runs, [1] gated runs (NULL: always)
	int nx, ny, nz, py, hx, lx, qy, qz;
};

// Tile-shape variants the autotuner chooses from per pass and length: 0 the default (radix 16,
// the single-instance tile), 1 half the lines/columns per CTA, 2 radix-8 passes, 3 (y passes
// only) TMA-staged tiles on persistent CTAs.
constexpr int GRP_VARIANTS = 4;
__host__ __device__ constexpr int var_radix(int n, int v) { return v == 2 ? (n < 8 ? n : 8) : ct_radix(n); }
__host__ __device__ constexpr int var_tb(int n, int csize, int v)
{
	return v == 1 ? (ct_tb(n, csize) > 1 ? ct_tb(n, csize) / 2 : 1) : ct_tb(n, csize);
}
__host__ __device__ constexpr int var_lpb(int n, int csize, int v)
{
	return v == 1 ? (ct_lpb(n, csize) > 1 ? ct_lpb(n, csize) / 2 : 1) : ct_lpb(n, csize);
}

__device__ __forceinline__ bool member_skips(const int *flags, int gate)
{
	return flags && (!flags[0] || (gate && !flags[gate]));
}

template <typename T, int N, int LPB, int R>
__global__ void __launch_bounds__(LPB * (N / R)) k_x_fwd_grp(const GDesc<T> *__restrict__ d,
                                                                      const int2 *__restrict__ items, int input,
                                                                      int gate)
{
	const int2 it = items[blockIdx.x];
	if (member_skips(d[it.x].flags, gate)) return;
	const GDesc<T> g = d[it.x];
	x_fwd_ct_body<T, N, LPB, true, R, true>(g.M[input], g.reg, g.ms_tab, g.spec, g.nx, g.ny, g.nz, g.py, g.hx, g.lx,
	                                  tw_of(g.tw_x, N, R), it.y);
}

template <typename T, int N, int LPB, int R>
__global__ void __launch_bounds__(LPB * (N / R)) k_x_inv_grp(const GDesc<T> *__restrict__ d,
                                                                      const int2 *__restrict__ items, int output,
                                                                      int gate)
{
	const int2 it = items[blockIdx.x];
	if (member_skips(d[it.x].flags, gate)) return;
	const GDesc<T> g = d[it.x];
	x_inv_ct_body<T, N, LPB, R>(g.spec, g.H[output], g.nx, g.ny, g.nz, g.py, g.hx, g.lx, tw_of(g.tw_x, N, R), it.y);
}

template <typename T, int N, int TB, bool INV, int R>
__global__ void __launch_bounds__(TB * (N / R)) k_y_grp(const GDesc<T> *__restrict__ d,
                                                                    const int2 *__restrict__ items, int gate)
{
	const int2 it = items[blockIdx.x];
	if (member_skips(d[it.x].flags, gate)) return;
	const GDesc<T> g = d[it.x];
	const int tiles = (g.hx + TB - 1) / TB;
	y_ct_body<T, N, TB, INV, R>(g.spec, INV ? N : g.ny, INV ? g.ny : N, g.hx, g.lx, tw_of(g.tw_y, N, R), it.y % tiles,
	                            it.y / tiles);
}

template <typename T, int PZ>
__global__ void __launch_bounds__(ZR_THREADS, 3) k_z_grp(const GDesc<T> *__restrict__ d, const int2 *__restrict__ items,
                                                        int gate)
{
	const int2 it = items[blockIdx.x];
	if (member_skips(d[it.x].flags, gate)) return;
	const GDesc<T> g = d[it.x];
	const int tiles = (g.hx + 31) / 32;
	z_reg_body<T, PZ>(g.spec, g.tensor, g.nz, g.py, g.hx, g.lx, g.qy, g.qz, it.y % tiles, it.y / tiles);
}

// Grouped y pass through TMA-staged tiles (the autotuner's variant 3): persistent CTAs walk the
// work list (member, column tile) of one length, skipping members whose run flags say so; each
// member has its own tensor maps (maps[2 member + INV], in global memory).  Pipeline as k_y_tma.
template <typename T, int N, bool INV>
__global__ void __launch_bounds__(ct_tb(N, sizeof(cplx<T>)) * (N / ct_radix(N)), 1)
    k_y_tma_grp(const GDesc<T> *__restrict__ d, const CUtensorMap *__restrict__ maps, const int2 *__restrict__ items,
                int n_items, int gate, int *err)
{
	using C = cplx<T>;
	constexpr int TB = ct_tb(N, sizeof(C));
	using G = YTmaGeom<N, TB, INV, C>;
	constexpr int R = ct_radix(N);
	using SI = SmCols<N, TB, 4>;
	extern __shared__ __align__(128) unsigned char smem_tma[];
	C *stage0 = reinterpret_cast<C *>(smem_tma);
	C *stage1 = stage0 + TB * G::ROWS;
	C *work = reinterpret_cast<C *>(smem_tma + 2 * (size_t)G::TILE_BYTES);
	uint64_t *bar = reinterpret_cast<uint64_t *>(smem_tma + 2 * (size_t)G::TILE_BYTES + G::WORK);
	const int tid = threadIdx.x;
	const int line = tid & (TB - 1), j0 = tid / TB;
	// this CTA's tiles: t = blockIdx.x + k gridDim.x, members that run only
	auto next_tile = [&](int t) {
		while (t < n_items && member_skips(d[items[t].x].flags, gate)) t += gridDim.x;
		return t;
	};
	auto issue = [&](int t, int b) {
		const int2 it = items[t];
		const int tiles_x = (d[it.x].hx + TB - 1) / TB;
		const int tx = it.y % tiles_x, plane = it.y / tiles_x;
		C *dst = b ? stage1 : stage0;
		const CUtensorMap *map = &maps[2 * it.x + (INV ? 1 : 0)];
		// the maps were written by a host copy before the launch: order those writes before the
		// tensor-map proxy reads them
		asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
		mbar_expect_tx(&bar[b], G::TILE_BYTES);
#pragma unroll
		for (int q = 0; q < G::NBOX; ++q)
			tma_load_3d(dst + q * G::BR * TB, map, tx * TB * G::E, q * G::BR, plane, &bar[b]);
	};
	if (tid == 0) {
		mbar_init(&bar[0], 1);
		mbar_init(&bar[1], 1);
		fence_proxy_async();
	}
	__syncthreads();
	int t = next_tile(blockIdx.x);
	int t1 = t < n_items ? next_tile(t + gridDim.x) : n_items;
	if (tid == 0) {
		if (t < n_items) issue(t, 0);
		if (t1 < n_items) issue(t1, 1);
	}
	uint32_t parity = 0;
	for (int k = 0; t < n_items; ++k) {
		const int b = k & 1;
		const bool late = !mbar_wait(&bar[b], (parity >> b) & 1u);
		if (__syncthreads_or(late)) {
			if (tid == 0) {
				atomicExch(err, 1);
				mbar_drain2(bar, parity, b, t1 < n_items);
			}
			return;
		}
		parity ^= 1u << b;
		const int2 it = items[t];
		const GDesc<T> &g = d[it.x];
		const int tiles_x = (g.hx + TB - 1) / TB;
		const int tx = it.y % tiles_x, plane = it.y / tiles_x;
		const int kx = tx * TB + line;
		const bool ok = kx < g.hx;
		const int lx = g.lx, n_out = INV ? g.ny : N;
		C *base = g.spec + (size_t)plane * N * lx + (ok ? kx : 0);
		const C *sb = b ? stage1 : stage0;
		auto ld = [&](int, int r) -> C { return r < G::ROWS ? sb[r * TB + line] : C{0, 0}; };
		auto st = [&](int, int r, C v) {
			if (ok && r < n_out) base[(size_t)r * lx] = v;
		};
		const int t2 = t1 < n_items ? next_tile(t1 + gridDim.x) : n_items;
		auto release = [&]() {
			__syncthreads();  // every thread has read stage buffer b
			if (tid == 0 && t2 < n_items) {
				fence_proxy_async();
				issue(t2, b);
			}
		};
		if constexpr (INV) cta_fft<T, N, R, TB, INV, SI>(work, tw_of(g.tw_y, N, R), line, j0, ld, st, release);
		else cta_fft_h0<T, N, R, TB, SI>(work, tw_of(g.tw_y, N, R), line, j0, ld, st, release);
		t = t1;
		t1 = t2;
	}
}

// Asynchronous copy of one complex value global -> shared (LDGSTS, 8 or 16 bytes).
template <class C>
__device__ __forceinline__ void cp_async_c(C *dst, const C *src)
{
	const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
	if constexpr (sizeof(C) == 8)
		asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
	else
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all_c() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit_c() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group_c() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Fused y and z passes for small members (the autotuner-free path of the grouped convolution):
// one CTA takes a tile of TB x-frequency columns of one member and keeps all of its y-z data in
// shared memory: the forward y transforms of the 3*NZ (component, z) lines of every column (ny
// data rows, zero padded to PY), the z transform, tensor multiply and inverse z transform of every
// (ky, column) in registers (3 components x PZ values per thread, the zero half of each z column
// skipped), and the inverse y transforms, whose rows y < ny go back to HBM.  The full y spectrum
// never reaches HBM: the pass reads and writes the x-transformed rows once and reads the tensor.
// Lines are split into G groups of LG lines so that a group's transform needs at most 512 threads
// (128 registers per thread for the z columns); tiles stay within ~104 KB of shared memory so
// that two CTAs share an SM.
// Reduced tensor [6][qz][qy][hx] -> kx-major [hx][qz][qy][6] (one thread per destination entry).
template <typename T>
__global__ void k_tensor_kx(const T *__restrict__ src, T *__restrict__ dst, int hx, int qy, int qz)
{
	const size_t ne = (size_t)6 * hx * qy * qz;
	for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < ne; e += (size_t)gridDim.x * blockDim.x) {
		const int c = (int)(e % 6);
		size_t r = e / 6;
		const int ky = (int)(r % qy);
		r /= qy;
		const int kz = (int)(r % qz);
		const int kx = (int)(r / qz);
		dst[e] = src[(((size_t)c * qz + kz) * qy + ky) * hx + kx];
	}
}

// NARROW: one kx column per CTA (a small group, such as the tail of a batch, then spreads over more
// SMs); each line's transforms and each (ky, column)'s multiply are the same operations either
// way, so the results do not depend on the choice.
template <int PY, int PZ, class C, bool NARROW = false>
struct YZGeom {
	static constexpr int NZ = PZ / 2;  // planes a member of this group can have (nz <= pz/2)
	static constexpr int R = ct_radix(PY), TPL = PY / R;
	static constexpr size_t line_bytes = (size_t)PY * sizeof(C);
	static constexpr int tb_for(int tb)
	{
		return (tb > 1 && (size_t)3 * NZ * tb * line_bytes * 33 / 32 > 104 * 1024) ? tb_for(tb / 2) : tb;
	}
	static constexpr int TB = NARROW ? 1 : tb_for(8);
	static constexpr int L = 3 * NZ * TB;
	static constexpr int g_for(int g) { return ((L / g) * TPL > 512 && L % (2 * g) == 0) ? g_for(g * 2) : g; }
	static constexpr int G = g_for(1);
	static constexpr int LG = L / G;
	static constexpr int THREADS = LG * TPL;
	static constexpr size_t GROUP_ELEMS = SmCols<PY, LG, 4>::SIZE;
	static constexpr size_t DATA = ((size_t)G * GROUP_ELEMS * sizeof(C) + 15) / 16 * 16;
	// behind the y-z data: the tile's reduced tensor entries, kx-major [TB][PZ/2+1][PY/2+1][6],
	// copied in while the forward y transforms run
	static constexpr int QY = PY / 2 + 1, QZ = PZ / 2 + 1;
	static constexpr size_t TENS = (size_t)TB * QZ * QY * 6 * (sizeof(C) / 2);
	static constexpr size_t SMEM = DATA + TENS;
	static constexpr bool fits = SMEM <= 227 * 1024 && THREADS >= 32 && THREADS <= 1024 && L % G == 0;
};

template <typename T, int PY, int PZ, bool NARROW = false>
__global__ void __launch_bounds__(YZGeom<PY, PZ, cplx<T>, NARROW>::THREADS)
    k_yz_grp(const GDesc<T> *__restrict__ d, const int2 *__restrict__ items, int gate)
{
	using C = cplx<T>;
	using G = YZGeom<PY, PZ, C, NARROW>;
	constexpr int TB = G::TB, LG = G::LG, NZ = G::NZ, H = PZ / 2;
	using SI = SmCols<PY, LG, 4>;
	const int2 it = items[blockIdx.x];
	if (member_skips(d[it.x].flags, gate)) return;
	const GDesc<T> &g = d[it.x];
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *smem = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int nz = g.nz, ny = g.ny, hx = g.hx, lx = g.lx;
	const int kx0 = it.y * TB;
	// line l = (c * NZ + z) * TB + col of group l / LG
	auto elem = [&](int l, int k) -> C & { return smem[(size_t)(l / LG) * G::GROUP_ELEMS + SI::at(l % LG, k)]; };
	// the tile's x-transformed rows (y < ny) land in the groups' buffers by asynchronous copies
	// issued all at once; lines outside the member (z >= nz, kx >= hx) are never stored
	{
		// a thread keeps its column and walks the (component-plane, row) pairs, y fastest, with
		// the row position carried forward instead of divided out per element
		static_assert(G::THREADS % TB == 0, "a thread keeps its column");
		constexpr int STEP = G::THREADS / TB;
		const int col = tid % TB, kx = kx0 + col, rows = 3 * NZ * ny;
		int row = tid / TB, cz = row / ny, y = row - cz * ny;
		if (kx < hx) {
			while (row < rows) {
				const int c = cz / NZ, z = cz % NZ;
				if (z < nz) {
					const int l = cz * TB + col;
					cp_async_c(&smem[(size_t)(l / LG) * G::GROUP_ELEMS + SI::at(l % LG, y)],
					           g.spec + ((size_t)(c * nz + z) * g.py + y) * lx + kx);
				}
				row += STEP;
				if (row >= rows) break;
				y += STEP;
				while (y >= ny) {
					y -= ny;
					++cz;
				}
			}
		}
	}
	cp_async_commit_c();
	// the tile's tensor entries: one contiguous run of the kx-major tensor (columns kx < hx)
	using T2 = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
	T2 *tsm = reinterpret_cast<T2 *>(smem_raw + G::DATA);
	{
		const int cols = hx - kx0 < TB ? hx - kx0 : TB;
		const int pairs = cols * G::QZ * G::QY * 3;
		const C *src = reinterpret_cast<const C *>(g.tensor_t + (size_t)kx0 * G::QZ * G::QY * 6);
		for (int e = tid; e < pairs; e += G::THREADS) cp_async_c(reinterpret_cast<C *>(tsm) + e, src + e);
	}
	cp_async_commit_c();
	cp_async_wait_group_c<1>();  // the y-z data (the tensor may still be arriving)
	__syncthreads();
	// forward y transforms in place (rows ny.. are the zero padding)
	for (int grp = 0; grp < G::G; ++grp) {
		const int line = tid % LG, j0 = tid / LG;
		C *sm = smem + (size_t)grp * G::GROUP_ELEMS;
		auto ld = [&](int ll, int y) -> C { return y < ny ? sm[SI::at(ll, y)] : C{0, 0}; };
		auto st = [&](int ll, int k, C v) { sm[SI::at(ll, k)] = v; };
		cta_fft_h0<T, PY, G::R, LG, SI, true>(sm, tw_of(g.tw_y, PY, G::R), line, j0, ld, st);  // rows ny <= PY/2 .. are zero
	}
	cp_async_wait_group_c<0>();
	__syncthreads();
	// z transforms, tensor multiply, inverse z transforms: one thread per (ky, column)
	for (int item = tid; item < PY * TB; item += G::THREADS) {
		const int col = item % TB, ky = item / TB;
		const int kx = kx0 + col;
		if (kx >= hx) continue;
		C v[3][PZ];
#pragma unroll
		for (int c = 0; c < 3; ++c) {
#pragma unroll
			for (int z = 0; z < H; ++z) v[c][z] = z < nz ? elem((c * NZ + (z < NZ ? z : 0)) * TB + col, ky) : C{0, 0};
			dft_reg_halfzero<T, PZ>(v[c]);
		}
		const bool fy = ky > PY / 2;
		const int kyr = fy ? PY - ky : ky;
		const T sy = fy ? T(-1) : T(1);
		// kz and PZ - kz share the tensor entries (sign of the z-odd components flipped): each
		// reduced entry is read once
#pragma unroll
		for (int kzr = 0; kzr <= H; ++kzr) {
			// the six components of entry (kx, kzr, kyr), contiguous pairs in shared memory
			const T2 *t = tsm + ((col * G::QZ + kzr) * G::QY + kyr) * 3;
			const T2 t0 = t[0], t1 = t[1], t2 = t[2];
			const T nxx = t0.x, nxy = t0.y, nxz = t1.x, nyy = t1.y, nyz = t2.x, nzz = t2.y;
#pragma unroll
			for (int q = 0; q < ((kzr == 0 || kzr == H) ? 1 : 2); ++q) {
				const int p = brev<PZ>(q ? PZ - kzr : kzr);
				const T sz = q ? T(-1) : T(1);
				const T xy = sy * nxy, xz = sz * nxz, yz = sy * sz * nyz;
				const C m0 = v[0][p], m1 = v[1][p], m2 = v[2][p];
				v[0][p] = C{nxx * m0.x + xy * m1.x + xz * m2.x, nxx * m0.y + xy * m1.y + xz * m2.y};
				v[1][p] = C{xy * m0.x + nyy * m1.x + yz * m2.x, xy * m0.y + nyy * m1.y + yz * m2.y};
				v[2][p] = C{xz * m0.x + yz * m1.x + nzz * m2.x, xz * m0.y + yz * m1.y + nzz * m2.y};
			}
		}
#pragma unroll
		for (int c = 0; c < 3; ++c) {
			C w[PZ];
#pragma unroll
			for (int k = 0; k < PZ; ++k) w[k] = v[c][brev<PZ>(k)];  // natural order for the inverse
			dft_reg<T, PZ, true>(w);
#pragma unroll
			for (int z = 0; z < H; ++z)
				if (z < nz && z < NZ) elem((c * NZ + z) * TB + col, ky) = w[brev<PZ>(z)];
		}
	}
	__syncthreads();
	// inverse y transforms, rows y < ny to HBM
	for (int grp = 0; grp < G::G; ++grp) {
		const int line = tid % LG, j0 = tid / LG;
		const int l = grp * LG + line;
		const int col = l % TB, cz = l / TB, c = cz / NZ, z = cz % NZ;
		const int kx = kx0 + col;
		const bool ok = kx < hx && z < nz;
		C *dst = g.spec + ((size_t)(c * nz + (ok ? z : 0)) * g.py) * lx + (ok ? kx : 0);
		C *sm = smem + (size_t)grp * G::GROUP_ELEMS;
		auto ld = [&](int ll, int k) -> C { return sm[SI::at(ll, k)]; };
		auto st = [&](int, int y, C val) {
			if (ok && y < ny) dst[(size_t)y * lx] = val;
		};
		if (grp > 0) __syncthreads();
		cta_fft<T, PY, G::R, LG, true, SI, true>(sm, tw_of(g.tw_y, PY, G::R), line, j0, ld, st);
	}
}

} // namespace

struct ConvGroup {
	int prec = MM_F32;
	int count = 0;
	std::vector<ConvGroupMember> solo;  // members whose convolution runs as passes of their own
	void *desc = nullptr;  // GDesc<T>[count]
	struct List {
		int pass;     // 0 x forward, 1 y forward, 2 z, 3 y inverse, 4 x inverse, 6 fused y+z (len = py*64+pz)
		int len;      // transform length of the pass
		int variant;  // tile shape chosen by the autotuner (GRP_VARIANTS)
		int2 *items;
		int n;
		int grid;     // persistent grid of variant 3
	};
	std::vector<List> lists;
	CUtensorMap *maps = nullptr;  // [2 member + inverse]: spectrum views of the y passes
	bool maps_ok = false;         // every member's maps exist (variant 3 possible)
	int *err = nullptr;           // set when a staged pass gave up waiting
	bool one_output = false;      // some member has no second output
	// the lists of one phase (independent members) run side by side on these streams
	static constexpr int POOL = 8;
	cudaStream_t pool[POOL] = {};
	cudaEvent_t fork = nullptr, join[POOL] = {};
	// ... and the members of `solo` beside them (made by group_create where there are such members: a
	// group is made for every relaxation of newly set states, and four streams and five events more took a
	// tenth of the time of a small batch's call)
	static constexpr int SOLO = 4;
	int used_solo = 0;
	cudaStream_t solo_st[SOLO] = {};
	cudaEvent_t solo_fork = nullptr, solo_join[SOLO] = {};
	~ConvGroup()
	{
		for (auto &q : solo_st)
			if (q) cudaStreamDestroy(q);
		for (auto &e : solo_join)
			if (e) cudaEventDestroy(e);
		if (solo_fork) cudaEventDestroy(solo_fork);
		cudaFree(desc);
		cudaFree(maps);
		cudaFree(err);
		for (auto &l : lists) cudaFree(l.items);
		for (auto &q : pool)
			if (q) cudaStreamDestroy(q);
		for (auto &e : join)
			if (e) cudaEventDestroy(e);
		if (fork) cudaEventDestroy(fork);
	}
};

namespace {

// Calls f(std::integral_constant<int, N>, std::integral_constant<int, V>) for a length and a
// variant; variants other than 0 exist for lengths 16..512.
template <typename T, class F>
void with_len_variant(int len, int v, F &&f)
{
	auto go = [&](auto nc) {
		constexpr int N = decltype(nc)::value;
		if constexpr (N >= 16 && N <= 512) {
			if (v == 1) { f(nc, std::integral_constant<int, 1>()); return; }
			if (v == 2) { f(nc, std::integral_constant<int, 2>()); return; }
		}
		f(nc, std::integral_constant<int, 0>());
	};
#define MM_WLV(N) go(std::integral_constant<int, N>())
	MM_FS_SWITCH(len, MM_WLV);
#undef MM_WLV
}

// Calls f(integral_constant PY, integral_constant PZ) for a fused y+z pass key (py * 64 + pz).
template <class F>
void with_yz(int key, F &&f)
{
	const int py = key / 64, pz = key % 64;
	auto by_pz = [&](auto pyc) {
		switch (pz) {
		case 2: f(pyc, std::integral_constant<int, 2>()); break;
		case 4: f(pyc, std::integral_constant<int, 4>()); break;
		case 8: f(pyc, std::integral_constant<int, 8>()); break;
		}
	};
	switch (py) {
	case 16: by_pz(std::integral_constant<int, 16>()); break;
	case 32: by_pz(std::integral_constant<int, 32>()); break;
	case 64: by_pz(std::integral_constant<int, 64>()); break;
	case 128: by_pz(std::integral_constant<int, 128>()); break;
	case 256: by_pz(std::integral_constant<int, 256>()); break;
	case 512: by_pz(std::integral_constant<int, 512>()); break;
	}
}

// Whether a member takes the fused y+z pass (and its columns per CTA).
template <typename T>
int yz_tb_dims(int py, int pz, int nz)
{
	int tb = 0;
	if (py < 16 || py > 512 || (pz != 2 && pz != 4 && pz != 8) || 2 * nz > pz) return 0;
	with_yz(py * 64 + pz, [&](auto pyc, auto pzc) {
		using G = YZGeom<decltype(pyc)::value, decltype(pzc)::value, cplx<T>>;
		if constexpr (G::fits) tb = G::TB;
	});
	return tb;
}
template <typename T>
int yz_tb(const ConvPlan *p)
{
	return yz_tb_dims<T>(p->py, p->pz, p->nz);
}

} // namespace

int conv_group_fused(int prec, int py, int pz, int nz)
{
	return prec == MM_F32 ? yz_tb_dims<float>(py, pz, nz) > 0 : yz_tb_dims<double>(py, pz, nz) > 0;
}

namespace {

// Threads of one CTA of a pass/length/variant (0 when the variant does not exist).
template <typename T>
int group_threads(int pass, int len, int v)
{
	using C = cplx<T>;
	if (pass == 2) return v == 0 ? ZR_THREADS : 0;
	if (pass == 6) {
		int t = 0;
		with_yz(len, [&](auto pyc, auto pzc) {
			constexpr int PY = decltype(pyc)::value, PZ = decltype(pzc)::value;
			using G0 = YZGeom<PY, PZ, C>;
			using G1 = YZGeom<PY, PZ, C, true>;
			if (v == 0 && G0::fits) t = G0::THREADS;
			if (v == 1 && G1::fits && G0::fits && G0::TB > 1) t = G1::THREADS;
		});
		return t;
	}
	if (v == 3) {
		if (pass != 1 && pass != 3) return 0;
		const int tb = ct_tb(len, (int)sizeof(C));
		if (tb * (int)sizeof(C) < 16 || tb * (int)(sizeof(C) / 8) > 256) return 0;
		return tb * (len / ct_radix(len));
	}
	if (v != 0 && (len < 16 || len > 512)) return 0;
	const int csz = (int)sizeof(C);
	const int lines = (pass == 0 || pass == 4) ? var_lpb(len, csz, v) : var_tb(len, csz, v);
	if (v == 1 && lines == ((pass == 0 || pass == 4) ? ct_lpb(len, csz) : ct_tb(len, csz))) return 0;
	const int t = lines * (len / var_radix(len, v));
	return (t >= 32 && t <= 1024 && (v != 2 || var_radix(len, v) != ct_radix(len))) ? t : 0;
}

// Blocks of one member for a pass/length/variant.
template <typename T>
int group_blocks(const ConvPlan *p, int pass, int len, int v)
{
	const int csz = (int)sizeof(cplx<T>);
	if (pass == 0 || pass == 4) {
		const int lpb = var_lpb(len, csz, v);
		return ((3 * p->ny * p->nz + 1) / 2 + lpb - 1) / lpb;
	}
	if (pass == 6) {
		const int tb = v == 1 ? 1 : yz_tb<T>(p);
		return (p->hx + tb - 1) / tb;
	}
	if (pass == 1 || pass == 3) {
		const int tb = var_tb(len, csz, v == 3 ? 0 : v);
		return (p->hx + tb - 1) / tb * 3 * p->nz;
	}
	return (p->hx + 31) / 32 * p->qy;
}

template <typename T>
size_t group_smem_bytes(int pass, int len, int v)
{
	using C = cplx<T>;
	size_t r = 0;
	if (pass == 2) return zr_smem<T>(len);
	if (pass == 6) {
		with_yz(len, [&](auto pyc, auto pzc) {
			constexpr int PY = decltype(pyc)::value, PZ = decltype(pzc)::value;
			r = v == 1 ? YZGeom<PY, PZ, C, true>::SMEM : YZGeom<PY, PZ, C>::SMEM;
		});
		return r;
	}
	if (v == 3) {
		auto y3 = [&](auto nc) {
			constexpr int N = decltype(nc)::value, TB = ct_tb(N, sizeof(C));
			r = pass == 1 ? YTmaGeom<N, TB, false, C>::SMEM : YTmaGeom<N, TB, true, C>::SMEM;
		};
#define MM_Y3(N) y3(std::integral_constant<int, N>())
		MM_FS_SWITCH(len, MM_Y3);
#undef MM_Y3
		return r;
	}
	with_len_variant<T>(len, v, [&](auto nc, auto vc) {
		constexpr int N = decltype(nc)::value, V = decltype(vc)::value;
		constexpr int LPB = var_lpb(N, sizeof(C), V), TB = var_tb(N, sizeof(C), V);
		r = (pass == 0 || pass == 4) ? (size_t)SmRows<N, LPB>::SIZE * sizeof(C) : (size_t)SmCols<N, TB>::SIZE * sizeof(C);
	});
	return r;
}

template <typename T>
mm_status group_smem(int pass, int len, int v)
{
	using C = cplx<T>;
	mm_status r = MM_OK;
	const size_t sm = group_smem_bytes<T>(pass, len, v);
	if (pass == 6) {
		with_yz(len, [&](auto pyc, auto pzc) {
			constexpr int PY = decltype(pyc)::value, PZ = decltype(pzc)::value;
			if (v == 1) {
				if constexpr (YZGeom<PY, PZ, C, true>::fits) r = set_smem<T>((const void *)k_yz_grp<T, PY, PZ, true>, sm);
			} else {
				if constexpr (YZGeom<PY, PZ, C>::fits) r = set_smem<T>((const void *)k_yz_grp<T, PY, PZ>, sm);
			}
		});
		return r;
	}
	if (pass == 2) {
		switch (len) {
		case 2: r = set_smem<T>((const void *)k_z_grp<T, 2>, sm); break;
		case 4: r = set_smem<T>((const void *)k_z_grp<T, 4>, sm); break;
		case 8: r = set_smem<T>((const void *)k_z_grp<T, 8>, sm); break;
		case 16: r = set_smem<T>((const void *)k_z_grp<T, 16>, sm); break;
		case 32: if constexpr (sizeof(T) == 4) { r = set_smem<T>((const void *)k_z_grp<T, 32>, sm); } break;
		}
		return r;
	}
	if (v == 3) {
		auto y3 = [&](auto nc) {
			constexpr int N = decltype(nc)::value;
			r = set_smem<T>(pass == 1 ? (const void *)k_y_tma_grp<T, N, false> : (const void *)k_y_tma_grp<T, N, true>, sm);
		};
#define MM_Y3(N) y3(std::integral_constant<int, N>())
		MM_FS_SWITCH(len, MM_Y3);
#undef MM_Y3
		return r;
	}
	with_len_variant<T>(len, v, [&](auto nc, auto vc) {
		constexpr int N = decltype(nc)::value, V = decltype(vc)::value;
		constexpr int LPB = var_lpb(N, sizeof(C), V), TB = var_tb(N, sizeof(C), V), R = var_radix(N, V);
		if (pass == 0) r = set_smem<T>((const void *)k_x_fwd_grp<T, N, LPB, R>, sm);
		if (pass == 4) r = set_smem<T>((const void *)k_x_inv_grp<T, N, LPB, R>, sm);
		if (pass == 1) r = set_smem<T>((const void *)k_y_grp<T, N, TB, false, R>, sm);
		if (pass == 3) r = set_smem<T>((const void *)k_y_grp<T, N, TB, true, R>, sm);
	});
	return r;
}

template <typename T>
void group_launch_v(const ConvGroup *g, int pass, int len, int v, const int2 *items, int n, int grid, int input,
                    int output, int gate, cudaStream_t st)
{
	using C = cplx<T>;
	const GDesc<T> *d = (const GDesc<T> *)g->desc;
	const size_t sm = group_smem_bytes<T>(pass, len, v);
	if (pass == 6) {
		with_yz(len, [&](auto pyc, auto pzc) {
			constexpr int PY = decltype(pyc)::value, PZ = decltype(pzc)::value;
			using G = YZGeom<PY, PZ, C>;
			using GN = YZGeom<PY, PZ, C, true>;
			if (v == 1) {
				if constexpr (GN::fits) k_yz_grp<T, PY, PZ, true><<<n, GN::THREADS, sm, st>>>(d, items, gate);
			} else {
				if constexpr (G::fits) k_yz_grp<T, PY, PZ><<<n, G::THREADS, sm, st>>>(d, items, gate);
			}
		});
		return;
	}
	if (v == 3) {
		auto y3 = [&](auto nc) {
			constexpr int N = decltype(nc)::value, TB = ct_tb(N, sizeof(C));
			const int threads = TB * (N / ct_radix(N));
			const int gr = grid < n ? grid : n;
			if (pass == 1) k_y_tma_grp<T, N, false><<<gr, threads, sm, st>>>(d, g->maps, items, n, gate, g->err);
			else k_y_tma_grp<T, N, true><<<gr, threads, sm, st>>>(d, g->maps, items, n, gate, g->err);
		};
#define MM_Y3(N) y3(std::integral_constant<int, N>())
		MM_FS_SWITCH(len, MM_Y3);
#undef MM_Y3
		return;
	}
	if (pass == 2) {
		switch (len) {
		case 2: k_z_grp<T, 2><<<n, ZR_THREADS, sm, st>>>(d, items, gate); break;
		case 4: k_z_grp<T, 4><<<n, ZR_THREADS, sm, st>>>(d, items, gate); break;
		case 8: k_z_grp<T, 8><<<n, ZR_THREADS, sm, st>>>(d, items, gate); break;
		case 16: k_z_grp<T, 16><<<n, ZR_THREADS, sm, st>>>(d, items, gate); break;
		case 32: if constexpr (sizeof(T) == 4) { k_z_grp<T, 32><<<n, ZR_THREADS, sm, st>>>(d, items, gate); } break;
		}
		return;
	}
	with_len_variant<T>(len, v, [&](auto nc, auto vc) {
		constexpr int N = decltype(nc)::value, V = decltype(vc)::value;
		constexpr int LPB = var_lpb(N, sizeof(C), V), TB = var_tb(N, sizeof(C), V), R = var_radix(N, V);
		constexpr int TPL = N / R;
		if (pass == 0) k_x_fwd_grp<T, N, LPB, R><<<n, LPB * TPL, sm, st>>>(d, items, input, gate);
		if (pass == 4) k_x_inv_grp<T, N, LPB, R><<<n, LPB * TPL, sm, st>>>(d, items, output, gate);
		if (pass == 1) k_y_grp<T, N, TB, false, R><<<n, TB * TPL, sm, st>>>(d, items, gate);
		if (pass == 3) k_y_grp<T, N, TB, true, R><<<n, TB * TPL, sm, st>>>(d, items, gate);
	});
}

template <typename T>
void group_launch(const ConvGroup *g, const ConvGroup::List &l, int input, int output, int gate, cudaStream_t st)
{
	group_launch_v<T>(g, l.pass, l.len, l.variant, l.items, l.n, l.grid, input, output, gate, st);
}

// Persistent grid of the TMA-staged grouped y pass (resident CTAs on the whole device).
template <typename T>
int group_grid(int pass, int len)
{
	using C = cplx<T>;
	int occ = 0;
	auto y3 = [&](auto nc) {
		constexpr int N = decltype(nc)::value, TB = ct_tb(N, sizeof(C));
		const int threads = TB * (N / ct_radix(N));
		const size_t sm = group_smem_bytes<T>(pass, N, 3);
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, pass == 1 ? (const void *)k_y_tma_grp<T, N, false>
		                                                                  : (const void *)k_y_tma_grp<T, N, true>,
		                                                  threads, sm) != cudaSuccess)
			cudaGetLastError();
	};
#define MM_Y3(N) y3(std::integral_constant<int, N>())
	MM_FS_SWITCH(len, MM_Y3);
#undef MM_Y3
	return (occ > 0 ? occ : 1) * num_sms();
}

// The autotuner's choices, per precision, pass and length, for the process (tuned once, on the
// first group that uses a pass and length, by timing every variant on that group's members).
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int>, int> g_tuned;

template <typename T>
std::vector<int2> group_items(const ConvGroupMember *m, const std::vector<int> &mem, int pass, int len, int v)
{
	std::vector<int2> items;
	for (int i : mem) {
		const int nb = group_blocks<T>(m[i].plan, pass, len, v);
		for (int b = 0; b < nb; ++b) items.push_back(make_int2(i, b));
	}
	return items;
}

// Times every variant of one pass and length on the group's members (run flags ignored) and
// returns the fastest.
template <typename T>
mm_status group_tune(const ConvGroup *g, const ConvGroupMember *m, const std::vector<int> &mem, int pass, int len,
                     cudaStream_t st, int *best)
{
	*best = 0;
	float best_ms = 0.f;
	cudaEvent_t e0 = nullptr, e1 = nullptr;
	MM_CUDA(cudaEventCreate(&e0));
	MM_CUDA(cudaEventCreate(&e1));
	mm_status r = MM_OK;
	for (int v = 0; v < GRP_VARIANTS && r == MM_OK; ++v) {
		if (!group_threads<T>(pass, len, v) || group_smem_bytes<T>(pass, len, v) > 227 * 1024) continue;
		if (v == 3 && !g->maps_ok) continue;
		const int grid = v == 3 ? group_grid<T>(pass, len) : 0;
		const std::vector<int2> items = group_items<T>(m, mem, pass, len, v);
		int2 *di = nullptr;
		r = cuda_status(cudaMalloc(&di, sizeof(int2) * items.size()), "cudaMalloc");
		if (r == MM_OK) r = cuda_status(cudaMemcpyAsync(di, items.data(), sizeof(int2) * items.size(),
		                                                cudaMemcpyHostToDevice, st), "cudaMemcpyAsync");
		if (r == MM_OK) r = group_smem<T>(pass, len, v);
		if (r == MM_OK) {
			group_launch_v<T>(g, pass, len, v, di, (int)items.size(), grid, 0, 0, 0, st);  // warm-up
			cudaEventRecord(e0, st);
			for (int k = 0; k < 3; ++k) group_launch_v<T>(g, pass, len, v, di, (int)items.size(), grid, 0, 0, 0, st);
			cudaEventRecord(e1, st);
			r = cuda_status(cudaEventSynchronize(e1), "autotune launch");
		}
		float ms = 0.f;
		if (r == MM_OK) r = cuda_status(cudaEventElapsedTime(&ms, e0, e1), "cudaEventElapsedTime");
		if (r == MM_OK && (v == 0 || ms < best_ms)) {
			best_ms = ms;
			*best = v;
		}
		cudaFree(di);
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	return r;
}

// A member large enough to fill the device by itself takes the single-instance passes, which are staged
// through TMA along every axis where its rows allow: its x passes alone have four times as many tiles
// as there are SMs.  Depends on the member only, so its arithmetic does not depend on the others.  A
// round of FP32 members of 512x400x4 cells, a little above that line: one 0.82 ms, against 1.04 in the grouped
// passes, four 2.91 against 3.50; 512x512x4 0.91 against 1.12, 3.24 against 3.90; 1024x1024x4 3.35 against
// 4.05; FP64 512x200x4 0.82 against 0.91, four 3.07 against 3.09; 512x512x4 1.64 against 1.94.  (Below the line:
// not measured on their own.)
template <typename T>
bool group_solo(const ConvPlan *p)
{
	const int lpb = ct_lpb(p->px, (int)sizeof(cplx<T>));
	return (3 * p->ny * p->nz + 1) / 2 / lpb >= 4 * num_sms();
}

template <typename T>
mm_status group_create(ConvGroup *g, const ConvGroupMember *m, int count, cudaStream_t st)
{
	std::vector<GDesc<T>> h(count);
	std::map<std::pair<int, int>, std::vector<int>> lists;  // (pass, length) -> members
	for (int i = 0; i < count; ++i) {
		ConvPlan *p = m[i].plan;
		if (!p || p->prec != g->prec || p->is2d || !p->fast_x || !p->fast_y || !p->reg_z)
			return fail(MM_ERR_UNSUPPORTED, "conv group: every member needs power-of-two 3-D padding with a register z pass");
		// (the lengths of MM_FS_SWITCH, which the grouped passes are instantiated for)
		const int most = sizeof(T) == 4 ? 2048 : 1024;
		if (p->px > most || p->py > most || !fft_is_pow2(p->px) || !fft_is_pow2(p->py) || !fft_is_pow2(p->pz))
			return fail(MM_ERR_UNSUPPORTED, "conv group: a member's padded lengths are beyond the grouped passes");
		if (2 * p->nx > p->px || 2 * p->ny > p->py || 2 * p->nz > p->pz)
			return fail(MM_ERR_UNSUPPORTED, "conv group: every member needs zero padding to at least twice its size");
		GDesc<T> &d = h[i];
		d.spec = (cplx<T> *)p->spec;
		d.tensor = (const T *)p->tensor;
		d.tw_x = (const cplx<T> *)p->tw_x;
		d.tw_y = (const cplx<T> *)p->tw_y;
		for (int k = 0; k < 4; ++k) d.M[k] = (const T *)m[i].M[k];
		for (int k = 0; k < 2; ++k) d.H[k] = (T *)m[i].H[k];
		if (!d.H[1]) g->one_output = true;
		d.reg = m[i].ms_uniform ? nullptr : m[i].reg;
		d.ms_tab = (const T *)(m[i].ms_uniform ? m[i].ms_uniform : m[i].ms_tab);
		d.flags = nullptr;  // the autotuner runs every member; the real flags are set below
		if (!d.ms_tab || !d.H[0]) return fail(MM_ERR_INVALID_ARGUMENT, "conv group: member without Ms table or output");
		d.nx = p->nx; d.ny = p->ny; d.nz = p->nz; d.py = p->py; d.hx = p->hx; d.lx = p->lx; d.qy = p->qy; d.qz = p->qz;
		d.tensor_t = nullptr;
		if (group_solo<T>(p)) {
			g->solo.push_back(m[i]);
			continue;
		}
		lists[{0, p->px}].push_back(i);
		if (yz_tb<T>(p) > 0) {
			lists[{6, p->py * 64 + p->pz}].push_back(i);  // y, z and the multiply in one pass
			// the fused pass reads the tensor by (kx, kz, ky) with its six components together;
			// the plan keeps that copy, so regrouping (members joining or leaving) allocates nothing
			if (!p->tensor_kx) {
				const size_t ne = (size_t)6 * p->hx * p->qy * p->qz;
				MM_CUDA(cudaMalloc(&p->tensor_kx, ne * sizeof(T)));
				k_tensor_kx<T><<<(unsigned)((ne + 255) / 256), 256, 0, st>>>((const T *)p->tensor, (T *)p->tensor_kx,
				                                                               p->hx, p->qy, p->qz);
				MM_CUDA(cudaGetLastError());
			}
			d.tensor_t = (const T *)p->tensor_kx;
		} else {
			lists[{1, p->py}].push_back(i);
			lists[{2, p->pz}].push_back(i);
			lists[{3, p->py}].push_back(i);
		}
		lists[{4, p->px}].push_back(i);
	}
	MM_CUDA(cudaMalloc(&g->desc, sizeof(GDesc<T>) * count));
	MM_CUDA(cudaMemcpyAsync(g->desc, h.data(), sizeof(GDesc<T>) * count, cudaMemcpyHostToDevice, st));
	// tensor maps of the TMA-staged y passes (variant 3): every member's spectrum, forward view of
	// its ny data rows (zero fill to N/2), inverse view of all py rows
	{
		std::vector<CUtensorMap> maps(2 * (size_t)count);
		bool ok = true;
		for (int i = 0; i < count && ok; ++i) {
			const ConvPlan *p = m[i].plan;
			const int E = (int)(sizeof(cplx<T>) / 8), tb = ct_tb(p->py, (int)sizeof(cplx<T>));
			if (2 * p->ny > p->py || tb * (int)sizeof(cplx<T>) < 16 || tb * E > 256) { ok = false; break; }
			const int rows_f = p->py / 2, rows_i = p->py;
			const uint64_t d0 = (uint64_t)p->lx * E, rowb = (uint64_t)p->lx * sizeof(cplx<T>), planeb = rowb * p->py;
			ok = tma_encode_3d(&maps[2 * i], p->spec, d0, (uint64_t)p->ny, 3ull * p->nz, rowb, planeb, tb * E,
			                   rows_f < 256 ? rows_f : 256, 1) == MM_OK &&
			     tma_encode_3d(&maps[2 * i + 1], p->spec, d0, (uint64_t)p->py, 3ull * p->nz, rowb, planeb, tb * E,
			                   rows_i < 256 ? rows_i : 256, 1) == MM_OK;
		}
		if (ok) {
			MM_CUDA(cudaMalloc(&g->maps, sizeof(CUtensorMap) * maps.size()));
			MM_CUDA(cudaMemcpyAsync(g->maps, maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice, st));
			MM_CUDA(cudaMalloc(&g->err, sizeof(int)));
			MM_CUDA(cudaMemsetAsync(g->err, 0, sizeof(int), st));
			g->maps_ok = true;
		} else {
			clear_error();
		}
	}
	for (const auto &kv : lists) {
		const int pass = kv.first.first, len = kv.first.second;
		int v = 0;
		bool known = false;
		{
			std::lock_guard<std::mutex> lock(g_tune_mu);
			auto it = g_tuned.find(std::make_tuple(g->prec, pass, len));
			if (it != g_tuned.end()) { v = it->second; known = true; }
		}
		// MMB200_GROUP_VARIANT=0|1|2 fixes the variant (where it exists) instead of timing them
		if (const char *fv = std::getenv("MMB200_GROUP_VARIANT")) {
			const int f = std::atoi(fv);
			v = (f >= 0 && f < GRP_VARIANTS && group_threads<T>(pass, len, f)) ? f : 0;
			known = true;
		}
		if (pass == 6) {
			// the narrow tiles when the default ones would not fill the device twice over
			int blocks = 0;
			for (int i : kv.second) blocks += group_blocks<T>(m[i].plan, 6, len, 0);
			known = true;
			v = blocks < 2 * num_sms() && group_threads<T>(6, len, 1) > 0 ? 1 : 0;
		}
		if (!known) {
			MM_TRY(group_tune<T>(g, m, kv.second, pass, len, st, &v));
			std::lock_guard<std::mutex> lock(g_tune_mu);
			g_tuned[std::make_tuple(g->prec, pass, len)] = v;
		}
		const std::vector<int2> items = group_items<T>(m, kv.second, pass, len, v);
		if (v == 3 && !g->maps_ok) v = 0;
		ConvGroup::List l{pass, len, v, nullptr, (int)items.size(), v == 3 ? group_grid<T>(pass, len) : 0};
		MM_CUDA(cudaMalloc(&l.items, sizeof(int2) * l.n));
		MM_CUDA(cudaMemcpyAsync(l.items, items.data(), sizeof(int2) * l.n, cudaMemcpyHostToDevice, st));
		MM_TRY(group_smem<T>(pass, len, v));
		g->lists.push_back(l);
	}
	// lists in pass order (x forward, y forward, z, y inverse, x inverse)
	auto rank = [](int pass) { return pass == 6 ? 1 : (pass >= 1 ? pass + 1 : pass); };
	std::stable_sort(g->lists.begin(), g->lists.end(),
	                 [&](const ConvGroup::List &a, const ConvGroup::List &b) { return rank(a.pass) < rank(b.pass); });
	// members on their own: one on the caller's stream when it is alone, else beside the grouped passes
	if (!g->solo.empty() && (!g->lists.empty() || g->solo.size() > 1)) {
		g->used_solo = std::min<int>((int)g->solo.size(), ConvGroup::SOLO);
		MM_CUDA(cudaEventCreateWithFlags(&g->solo_fork, cudaEventDisableTiming));
		for (int q = 0; q < g->used_solo; ++q) {
			MM_CUDA(cudaStreamCreateWithFlags(&g->solo_st[q], cudaStreamNonBlocking));
			MM_CUDA(cudaEventCreateWithFlags(&g->solo_join[q], cudaEventDisableTiming));
		}
	}
	for (int i = 0; i < count; ++i) h[i].flags = m[i].flags;
	MM_CUDA(cudaMemcpyAsync(g->desc, h.data(), sizeof(GDesc<T>) * count, cudaMemcpyHostToDevice, st));
	MM_CUDA(cudaStreamSynchronize(st));
	return MM_OK;
}

} // namespace

mm_status conv_group_create(ConvGroup **out, const ConvGroupMember *members, int count, cudaStream_t st)
{
	if (!out || !members || count < 1) return fail(MM_ERR_INVALID_ARGUMENT, "conv group: no members");
	ConvGroup *g = new ConvGroup();
	g->prec = members[0].plan ? members[0].plan->prec : MM_F32;
	g->count = count;
	mm_status rs = cuda_status(cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming), "cudaEventCreate");
	for (int q = 0; q < ConvGroup::POOL && rs == MM_OK; ++q) {
		rs = cuda_status(cudaStreamCreateWithFlags(&g->pool[q], cudaStreamNonBlocking), "cudaStreamCreate");
		if (rs == MM_OK) rs = cuda_status(cudaEventCreateWithFlags(&g->join[q], cudaEventDisableTiming), "cudaEventCreate");
	}
	if (rs != MM_OK) {
		delete g;
		return rs;
	}
	const mm_status r = g->prec == MM_F64 ? group_create<double>(g, members, count, st)
	                                       : group_create<float>(g, members, count, st);
	if (r != MM_OK) {
		delete g;
		return r;
	}
	*out = g;
	return MM_OK;
}

// The lists of one phase (x forward; y forward and fused y+z; z; y inverse; x inverse) touch
// disjoint members, so each phase forks onto the group's stream pool and joins back on `st`
// (inside a stream capture this becomes parallel graph branches).
mm_status conv_group_execute(ConvGroup *g, int input, int gate, cudaStream_t st, int output)
{
	if (!g || input < 0 || input > 3) return fail(MM_ERR_INVALID_ARGUMENT, "conv group: bad input selector");
	if (output < 0 || output > 1 || (output == 1 && g->one_output))
		return fail(MM_ERR_INVALID_ARGUMENT, "conv group: bad output selector");
	auto rank = [](int pass) { return pass == 6 ? 1 : pass; };
	if (g->used_solo) {
		MM_CUDA(cudaEventRecord(g->solo_fork, st));
		for (int q = 0; q < g->used_solo; ++q) MM_CUDA(cudaStreamWaitEvent(g->solo_st[q], g->solo_fork, 0));
	}
	for (size_t k = 0; k < g->solo.size(); ++k) {
		const ConvGroupMember &m = g->solo[k];
		cudaStream_t sq = g->used_solo ? g->solo_st[k % g->used_solo] : st;
		MM_TRY(g->prec == MM_F64 ? conv_run_f64(m.plan, (const double *)m.M[input], m.reg, (const double *)m.ms_tab,
		                                        (double *)m.H[output], sq, m.flags, gate)
		                         : conv_run_f32(m.plan, (const float *)m.M[input], m.reg, (const float *)m.ms_tab,
		                                        (float *)m.H[output], sq, m.flags, gate));
	}
	size_t i = 0;
	while (i < g->lists.size()) {
		size_t j = i;
		while (j < g->lists.size() && rank(g->lists[j].pass) == rank(g->lists[i].pass)) ++j;
		const int n = (int)(j - i);
		if (n == 1) {
			if (g->prec == MM_F64) group_launch<double>(g, g->lists[i], input, output, gate, st);
			else group_launch<float>(g, g->lists[i], input, output, gate, st);
			MM_TRY(after_launch("k_conv_grp"));
		} else {
			MM_CUDA(cudaEventRecord(g->fork, st));
			const int used = n < ConvGroup::POOL ? n : ConvGroup::POOL;
			for (int q = 0; q < used; ++q) MM_CUDA(cudaStreamWaitEvent(g->pool[q], g->fork, 0));
			for (size_t k = i; k < j; ++k) {
				cudaStream_t sq = g->pool[(k - i) % ConvGroup::POOL];
				if (g->prec == MM_F64) group_launch<double>(g, g->lists[k], input, output, gate, sq);
				else group_launch<float>(g, g->lists[k], input, output, gate, sq);
				MM_TRY(after_launch("k_conv_grp"));
			}
			for (int q = 0; q < used; ++q) {
				MM_CUDA(cudaEventRecord(g->join[q], g->pool[q]));
				MM_CUDA(cudaStreamWaitEvent(st, g->join[q], 0));
			}
		}
		i = j;
	}
	for (int q = 0; q < g->used_solo; ++q) {
		MM_CUDA(cudaEventRecord(g->solo_join[q], g->solo_st[q]));
		MM_CUDA(cudaStreamWaitEvent(st, g->solo_join[q], 0));
	}
	return MM_OK;
}

void conv_group_destroy(ConvGroup *g) { delete g; }

} // namespace mm

struct mm_conv {
	mm::ConvPlan *plan;
};

using namespace mm;

extern "C" {

MM_API mm_status mm_conv_create(mm_conv **out, int prec, int nx, int ny, int nz, int ex, int ey,
                                int ez, const double *N_device, void *stream)
{
	if (!out) return fail(MM_ERR_INVALID_ARGUMENT, "mm_conv_create: null out");
	ConvPlan *p = nullptr;
	MM_TRY(conv_plan_create(&p, prec, nx, ny, nz, ex, ey, ez, N_device, as_stream(stream)));
	*out = new mm_conv{p};
	return MM_OK;
}

MM_API mm_status mm_conv_execute(mm_conv *conv, const void *M, void *H, void *stream)
{
	if (!conv || !conv->plan || !M || !H) return fail(MM_ERR_INVALID_ARGUMENT, "mm_conv_execute: null argument");
	return conv_execute(conv->plan, M, nullptr, nullptr, H, as_stream(stream));
}

MM_API mm_status mm_conv_destroy(mm_conv *conv)
{
	if (conv) {
		delete conv->plan;
		delete conv;
	}
	return MM_OK;
}

} // extern "C"
