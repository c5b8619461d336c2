// Demagnetisation tensor on the GPU in FP64.  Replaces GenerateDemagTensor / calculateDemagTensor
// (mmm/demag/demag_tensor.cpp:116-186, mmm/demag/tensor.cpp:35-191), non-periodic case.
//
// For a cell offset X = (i dx, j dy, k dz) the tensor of two uniformly magnetised boxes is
//   N_ab(X) = (1/V) * Int_{[-d,d]^3} prod_c (d_c - |u_c|) K_ab(X + u) du,
//   K_ab(r) = (delta_ab r^2 - 3 r_a r_b) / (4 pi |r|^5),
// the average of the point-dipole kernel over all pairs of points of the two cells (the tent
// weights are the overlap lengths).  The reference evaluates Newell's closed forms in long double
// near the origin and truncated asymptotic series further out (tensor_integrals.h:370-462).
// Here:
//  * offsets whose boxes touch (|i|,|j|,|k| <= 1) use Newell's closed forms f and g (Newell,
//    Williams & Dunlop, JGR 98 (1993) 9551) with the 27-point second difference in FP64 -- the
//    cancellation there is mild;
//  * every other offset uses tensor-product Gauss-Legendre quadrature on the two linear halves
//    of each tent, with n nodes per half chosen from the distance D between the box X+[-d,d]
//    and the singularity at 0: rho = r + sqrt(r^2+1), r = D/(d_c/2), n = ceil(20/ln rho) + 1.
//    This keeps the relative error near 1e-15 (checked against a binary128 Newell evaluation),
//    including the far field where the reference's series truncation is visible (~1e-8 in H).
// Output: the NEGATED tensor in the reference's Matrix(Shape(6, ex, ey, ez)) layout (component
// fastest), components (xx, xy, xz, yy, yz, zz), scattered into the eight octants with the
// parities of tensor.cpp:167-180.
#include "mm_common.cuh"
#include "conv.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace mm {
namespace {

constexpr int GL_MAX = 40;

// Quadrature of one tent of half-width 1: 2 n (node, weight) pairs for n nodes per half, the table for
// n starting at n (n - 1).  The weights include the tent, 1 - |node|.
struct GLTable {
	double2 *xw = nullptr;
};

// Gauss-Legendre nodes and weights by Newton iteration on P_n (long double).
void gauss_legendre(int n, std::vector<double> &x, std::vector<double> &w)
{
	x.resize(n);
	w.resize(n);
	for (int i = 0; i < n; ++i) {
		long double z = cosl(3.14159265358979323846264338327950288L * (i + 0.75L) / (n + 0.5L));
		long double dp = 0;
		for (int it = 0; it < 100; ++it) {
			long double p0 = 1, p1 = z;
			for (int k = 2; k <= n; ++k) {
				const long double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
				p0 = p1;
				p1 = p2;
			}
			if (n == 1) { p1 = z; p0 = 1; }
			dp = n * (z * p1 - p0) / (z * z - 1);
			const long double dz = p1 / dp;
			z -= dz;
			if (fabsl(dz) < 1e-21L) break;
		}
		{
			long double p0 = 1, p1 = z;
			for (int k = 2; k <= n; ++k) {
				const long double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
				p0 = p1;
				p1 = p2;
			}
			dp = n * (z * p1 - p0) / (z * z - 1);
		}
		x[i] = (double)z;
		w[i] = (double)(2.0L / ((1 - z * z) * dp * dp));
	}
}

// The node/weight table lives in device memory, so each device gets its own (built on first use).
mm_status gl_table(GLTable **out)
{
	static std::mutex mu;
	static std::vector<GLTable> tabs;
	int dev = 0;
	MM_CUDA(cudaGetDevice(&dev));
	std::lock_guard<std::mutex> lock(mu);
	if ((int)tabs.size() <= dev) tabs.resize(dev + 1);
	GLTable &tab = tabs[dev];
	if (!tab.xw) {
		std::vector<double> x, w;
		std::vector<double2> h;
		for (int n = 1; n <= GL_MAX; ++n) {
			if (n == 1) { x = {0.0}; w = {2.0}; }
			else gauss_legendre(n, x, w);
			for (double half : {-0.5, 0.5})
				for (int q = 0; q < n; ++q) {
					const double u = half + 0.5 * x[q];
					h.push_back(double2{u, 0.5 * w[q] * (1.0 - std::fabs(u))});
				}
		}
		MM_CUDA(cudaMalloc(&tab.xw, h.size() * sizeof(double2)));
		MM_CUDA(cudaMemcpy(tab.xw, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice));
	}
	*out = &tab;
	return MM_OK;
}

// Newell f (even in every argument).
__device__ double newell_f(double x, double y, double z)
{
	const double x2 = x * x, y2 = y * y, z2 = z * z, R2 = x2 + y2 + z2;
	if (R2 == 0.0) return 0.0;
	const double R = sqrt(R2);
	double r = (2 * x2 - y2 - z2) * R / 6;
	if (x2 + z2 > 0 && y != 0) r += y / 2 * (z2 - x2) * asinh(y / sqrt(x2 + z2));
	if (x2 + y2 > 0 && z != 0) r += z / 2 * (y2 - x2) * asinh(z / sqrt(x2 + y2));
	if (x != 0 && y != 0 && z != 0) r -= x * y * z * atan(y * z / (x * R));
	return r;
}

// Newell g (odd in x and y, even in z).
__device__ double newell_g(double x, double y, double z)
{
	const double x2 = x * x, y2 = y * y, z2 = z * z, R2 = x2 + y2 + z2;
	if (R2 == 0.0) return 0.0;
	const double R = sqrt(R2);
	double r = -x * y * R / 3;
	if (x != 0 && y != 0 && z != 0) r += x * y * z * asinh(z / sqrt(x2 + y2));
	if (x != 0 && y != 0) {
		if (y2 + z2 > 0) r += y / 6 * (3 * z2 - y2) * asinh(x / sqrt(y2 + z2));
		if (x2 + z2 > 0) r += x / 6 * (3 * z2 - x2) * asinh(y / sqrt(x2 + z2));
	}
	if (x != 0 && y != 0 && z != 0) {
		r -= z * z2 / 6 * atan(x * y / (z * R));
		r -= z * y2 / 2 * atan(x * z / (y * R));
		r -= z * x2 / 2 * atan(y * z / (x * R));
	}
	return r;
}

// Negated tensor (xx, xy, xz, yy, yz, zz) at offset (i, j, k) from Newell's formulas.
__device__ void tensor_newell(int i, int j, int k, double dx, double dy, double dz, double *v)
{
	double acc[6] = {0, 0, 0, 0, 0, 0};
	for (int cz = -1; cz <= 1; ++cz)
		for (int cy = -1; cy <= 1; ++cy)
			for (int cx = -1; cx <= 1; ++cx) {
				const double w = (cx ? -1.0 : 2.0) * (cy ? -1.0 : 2.0) * (cz ? -1.0 : 2.0);
				const double X = (i + cx) * dx, Y = (j + cy) * dy, Z = (k + cz) * dz;
				acc[0] += w * newell_f(X, Y, Z);
				acc[3] += w * newell_f(Y, X, Z);
				acc[5] += w * newell_f(Z, Y, X);
				acc[1] += w * newell_g(X, Y, Z);
				acc[2] += w * newell_g(X, Z, Y);
				acc[4] += w * newell_g(Y, Z, X);
			}
	const double pref = -1.0 / (4.0 * PI * dx * dy * dz);
	for (int c = 0; c < 6; ++c) v[c] = pref * acc[c];
}

__host__ __device__ inline int gl_order(double D, double halfwidth)
{
	const double r = D / halfwidth;
	const double rho = r + sqrt(r * r + 1.0);
	const double lr = log(rho);
	if (!(lr > 0.0)) return GL_MAX + 1;
	const double n = ceil(20.0 / lr) + 1.0;
	return n < 3.0 ? 3 : (n > GL_MAX ? GL_MAX + 1 : (int)n);
}

// Nodes per half tent along each axis for offset (i, j, k); false if they exceed the table (the
// caller then uses Newell's formulas).
__host__ __device__ inline bool quad_orders(int i, int j, int k, double dx, double dy, double dz, int (&n)[3])
{
	const double X[3] = {i * dx, j * dy, k * dz};
	const double a[3] = {dx, dy, dz};
	double g2 = 0;
	for (int c = 0; c < 3; ++c) {
		const double g = fmax(fabs(X[c]) - a[c], 0.0);
		g2 += g * g;
	}
	const double D = sqrt(g2);
	for (int c = 0; c < 3; ++c) {
		n[c] = gl_order(D, 0.5 * a[c]);
		if (n[c] > GL_MAX) return false;
	}
	return true;
}

// Quadrature sums of offset (i, j, k) over the (y, z) node pairs first, first + step, ...: the
// negated tensor without its factor V / 4 pi.  Along x four moments of the row are summed (of
// r^-3 and 3 r^-5 with rx^0, rx^1, rx^2), from which the six components of the row follow.
__device__ __forceinline__ void quad_sums(int i, int j, int k, double dx, double dy, double dz, const int (&n)[3],
                                          const double2 *__restrict__ gl, int first, int step, double (&acc)[6])
{
	const double X = i * dx, Y = j * dy, Z = k * dz;
	const double2 *gx = gl + n[0] * (n[0] - 1), *gy = gl + n[1] * (n[1] - 1), *gz = gl + n[2] * (n[2] - 1);
	const int nx = 2 * n[0], ny = 2 * n[1], rows = ny * 2 * n[2];
	for (int c = 0; c < 6; ++c) acc[c] = 0.0;
	for (int row = first; row < rows; row += step) {
		const int qz = row / ny, qy = row - qz * ny;
		const double2 ny2 = gy[qy], nz2 = gz[qz];
		const double ry = Y + ny2.x * dy, rz = Z + nz2.x * dz, wyz = ny2.y * nz2.y;
		const double ryz2 = ry * ry + rz * rz;
		double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll 4
		for (int qx = 0; qx < nx; ++qx) {
			const double2 nd = gx[qx];
			const double rx = X + nd.x * dx;
			const double r2 = rx * rx + ryz2;
			const double ir = rsqrt(r2);
			const double ir2 = ir * ir;
			const double w3 = nd.y * (ir2 * ir);
			const double w5 = 3.0 * w3 * ir2, w5x = w5 * rx;
			a0 += w3;
			a1 += w5;
			a2 += w5x;
			a3 += w5x * rx;
		}
		acc[0] += wyz * (a0 - a3);
		acc[1] -= wyz * ry * a2;
		acc[2] -= wyz * rz * a2;
		acc[3] += wyz * (a0 - ry * ry * a1);
		acc[4] -= wyz * (ry * rz * a1);
		acc[5] += wyz * (a0 - rz * rz * a1);
	}
}

// The offsets next to the origin need high orders (27,000 points two cells away, 1,000 to 1,700 for
// most of a mesh), and one thread per offset made them the kernel's whole time (7.6 ms at 240x120x10
// cells, FP64, of which 0.6 ms are the other offsets).  So the box of offsets that need more than
// NEAR_POINTS points is computed first, a block per offset, and looked up by the kernels that follow.
constexpr int NEAR_POINTS = 2000, NEAR_MAX = 1 << 16, NEAR_THREADS = 128;

struct NearBox {
	int x = 0, y = 0, z = 0;    // offsets i < x, j < y, k < z
	int lx = 0, ly = 0;         // layout: six values at v + 6 ((k ly + j) lx + i)
	double *v = nullptr;
	__host__ __device__ double *at(int i, int j, int k) const { return v + 6 * (((size_t)k * ly + j) * lx + i); }
};

__global__ void __launch_bounds__(NEAR_THREADS) k_tensor_near(NearBox nb, double dx, double dy, double dz,
                                                              const double2 *__restrict__ gl)
{
	const int q = blockIdx.x, i = q % nb.x, j = q / nb.x % nb.y, k = q / (nb.x * nb.y);
	double *out = nb.at(i, j, k);
	int n[3];
	if ((i <= 1 && j <= 1 && k <= 1) || !quad_orders(i, j, k, dx, dy, dz, n)) {
		if (threadIdx.x == 0) tensor_newell(i, j, k, dx, dy, dz, out);
		return;
	}
	double acc[6];
	quad_sums(i, j, k, dx, dy, dz, n, gl, threadIdx.x, NEAR_THREADS, acc);
	__shared__ double red[6][NEAR_THREADS / 32];
	for (int c = 0; c < 6; ++c) {
		const double w = warp_sum(acc[c]);
		if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = w;
	}
	__syncthreads();
	if (threadIdx.x < 6) {
		double sum = 0;
		for (int w = 0; w < NEAR_THREADS / 32; ++w) sum += red[threadIdx.x][w];
		out[threadIdx.x] = -dx * dy * dz / (4.0 * PI) * sum;
	}
}

// Host: the extents of the near box for offsets up to nx, ny, nz (not included).
void near_extents(int nx, int ny, int nz, double dx, double dy, double dz, NearBox &nb)
{
	const int lim[3] = {nx, ny, nz};
	int ext[3];
	const long long most = 8LL * GL_MAX * GL_MAX * GL_MAX;
	for (long long points = NEAR_POINTS;; points *= 2) {
		for (int a = 0; a < 3; ++a) {
			// along the axis: the first offset that needs few points (the orders fall with distance)
			int lo = std::min(2, lim[a]), hi = points <= most ? lim[a] : lo;
			while (lo < hi) {
				const int mid = lo + (hi - lo) / 2;
				int n[3];
				const bool few = quad_orders(a == 0 ? mid : 0, a == 1 ? mid : 0, a == 2 ? mid : 0, dx, dy, dz, n) &&
				                 8LL * n[0] * n[1] * n[2] <= points;
				if (few) hi = mid;
				else lo = mid + 1;
			}
			ext[a] = lo;
		}
		if ((long long)ext[0] * ext[1] * ext[2] <= NEAR_MAX) break;  // (a box of two cells a side at the last)
	}
	nb.x = ext[0];
	nb.y = ext[1];
	nb.z = ext[2];
}

mm_status tensor_near(const NearBox &nb, double dx, double dy, double dz, const double2 *gl, cudaStream_t st)
{
	k_tensor_near<<<nb.x * nb.y * nb.z, NEAR_THREADS, 0, st>>>(nb, dx, dy, dz, gl);
	return after_launch("k_tensor_near");
}

// Negated tensor (xx, xy, xz, yy, yz, zz) at offset (i, j, k) >= 0.
__device__ __forceinline__ void tensor_at(int i, int j, int k, double dx, double dy, double dz, const NearBox &nb,
                                          const double2 *__restrict__ gl, double (&v)[6])
{
	if (i < nb.x && j < nb.y && k < nb.z) {
		const double *t = nb.at(i, j, k);
		for (int c = 0; c < 6; ++c) v[c] = t[c];
		return;
	}
	int n[3];
	if (!quad_orders(i, j, k, dx, dy, dz, n)) {
		tensor_newell(i, j, k, dx, dy, dz, v);
		return;
	}
	quad_sums(i, j, k, dx, dy, dz, n, gl, 0, 1, v);
	const double f = -dx * dy * dz / (4.0 * PI);
	for (int c = 0; c < 6; ++c) v[c] *= f;
}

// OCTANT: offsets >= 0 only, [nz][ny][nx][6] (ex = nx, ey = ny); else the padded layout, every octant.
template <bool OCTANT>
__global__ void __launch_bounds__(128) k_demag_tensor(int nx, int ny, int nz, double dx, double dy,
                                                      double dz, int ex, int ey, int ez, NearBox nb,
                                                      const double2 *__restrict__ gl, double *out)
{
	const size_t cnt = (size_t)nx * ny * nz;
	for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < cnt; q += (size_t)gridDim.x * blockDim.x) {
		const int i = (int)(q % nx), j = (int)((q / nx) % ny), k = (int)(q / ((size_t)nx * ny));
		double v[6];
		tensor_at(i, j, k, dx, dy, dz, nb, gl, v);
		if (OCTANT) {
			for (int c = 0; c < 6; ++c) out[6 * q + c] = v[c];
			continue;
		}
		for (int o = -1; o <= 1; o += 2)
			for (int p = -1; p <= 1; p += 2)
				for (int r = -1; r <= 1; r += 2) {
					if ((i == 0 && o < 0) || (j == 0 && p < 0) || (k == 0 && r < 0)) continue;
					const int I = (o * i + ex) % ex, J = (p * j + ey) % ey, K = (r * k + ez) % ez;
					double *d = out + 6 * (((size_t)K * ey + J) * ex + I);
					d[0] = v[0];
					d[1] = o * p * v[1];
					d[2] = o * r * v[2];
					d[3] = v[3];
					d[4] = p * r * v[4];
					d[5] = v[5];
				}
	}
}

// The near box goes to its place in the output, where the next kernel's thread of the same offset
// reads it (no other thread writes offsets i < nx, j < ny, k < nz).
template <bool OCTANT>
mm_status tensor_run(int nx, int ny, int nz, double dx, double dy, double dz, int ex, int ey, int ez, double *out,
                     cudaStream_t st)
{
	GLTable *gl = nullptr;
	MM_TRY(gl_table(&gl));
	NearBox nb;
	near_extents(nx, ny, nz, dx, dy, dz, nb);
	nb.lx = ex;
	nb.ly = ey;
	nb.v = out;
	MM_TRY(tensor_near(nb, dx, dy, dz, gl->xw, st));
	const size_t want = ((size_t)nx * ny * nz + 127) / 128;
	const int grid = (int)(want < 65535u * 16 ? want : 65535u * 16);
	k_demag_tensor<OCTANT><<<grid, 128, 0, st>>>(nx, ny, nz, dx, dy, dz, ex, ey, ez, nb, gl->xw, out);
	return after_launch("k_demag_tensor");
}

// ---- periodic boundaries (tensor.cpp:35-165 with demag_tensor.cpp:116-186) --------------------
// Along a periodic axis the tensor of offset i sums the images i + r n (r < R, the repetitions);
// the octant scatter adds the mirrored images -(i + r n), so an entry sums displacements from
// -R n to (R - 1) n around it.  Offsets that coincide with their mirror (i + r n == 0) count
// half on each side, as the reference divides by its "mcs" factor.  The images beyond the R-th
// (the reference's infinity correction, tensor.cpp:60-165) are far from the box: their sum is the
// point-dipole tensor (V / 4 pi) d_a d_b (1 / r), here summed explicitly over TAIL_M further images
// and integrated in closed form beyond (line integrals with the first Euler-Maclaurin correction for
// the images along one periodic axis, quadrant integrals for the far corner of two periodic axes,
// tensor.cpp:104-161), below 1e-9 of the tail sums.  The reference approximates the same sums
// by asymptotic expansions; no three-axis corner term exists there, nor here.
constexpr int TAIL_M = 32;

// (V / 4 pi) d_a d_b (1 / r) at r = P: the far-field negated tensor of one cell (xx xy xz yy yz zz)
__device__ void point_dipole(const double P[3], double V4, double *v)
{
	const double r2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
	const double ir = rsqrt(r2), ir3 = ir * ir * ir, ir5 = ir3 * ir * ir;
	v[0] += V4 * (3 * P[0] * P[0] * ir5 - ir3);
	v[1] += V4 * 3 * P[0] * P[1] * ir5;
	v[2] += V4 * 3 * P[0] * P[2] * ir5;
	v[3] += V4 * (3 * P[1] * P[1] * ir5 - ir3);
	v[4] += V4 * 3 * P[1] * P[2] * ir5;
	v[5] += V4 * (3 * P[2] * P[2] * ir5 - ir3);
}

__device__ __forceinline__ int sym_idx(int a, int b)
{
	const int lo = a < b ? a : b, hi = a < b ? b : a;
	return lo == 0 ? hi : (lo == 1 ? 2 + hi : 5);
}

// Integral over s in [0, inf) of d_a d_b (1 / r) at r = P + s e_A (P_A > 0), added times f.
__device__ void line_integral(const double P[3], int A, double f, double *v)
{
	const int B = (A + 1) % 3, C = (A + 2) % 3;
	const double x0 = P[A], y = P[B], z = P[C];
	const double r0 = sqrt(x0 * x0 + y * y + z * z), w = x0 + r0, ir3 = 1.0 / (r0 * r0 * r0);
	const double q = (w + r0) * ir3 / (w * w);
	v[sym_idx(A, A)] += f * x0 * ir3;
	v[sym_idx(A, B)] += f * y * ir3;
	v[sym_idx(A, C)] += f * z * ir3;
	v[sym_idx(B, B)] += f * (y * y * q - 1.0 / (r0 * w));
	v[sym_idx(B, C)] += f * y * z * q;
	v[sym_idx(C, C)] += f * (z * z * q - 1.0 / (r0 * w));
}

// Integral over s, t in [0, inf) of d_a d_b (1 / r) at r = P + s e_A + t e_B (P_A, P_B > 0).
__device__ void quadrant_integral(const double P[3], int A, int B, double f, double *v)
{
	const int C = 3 - A - B;
	const double x0 = P[A], y0 = P[B], z = P[C];
	const double r0 = sqrt(x0 * x0 + y0 * y0 + z * z);
	const double a2 = x0 * x0 + z * z, b2 = y0 * y0 + z * z;
	const double xx = x0 / a2 * (1.0 - y0 / r0), yy = y0 / b2 * (1.0 - x0 / r0);
	v[sym_idx(A, A)] += f * xx;
	v[sym_idx(B, B)] += f * yy;
	v[sym_idx(C, C)] -= f * (xx + yy);
	v[sym_idx(A, B)] += f / r0;
	v[sym_idx(A, C)] += f * z / a2 * (1.0 - y0 / r0);
	v[sym_idx(B, C)] += f * z / b2 * (1.0 - x0 / r0);
}

// f d_A d_a d_b (1 / r) at r = P, added (the derivative along A of d_a d_b (1 / r)).
__device__ void line_derivative(const double P[3], int A, double f, double *v)
{
	const double r2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
	const double ir = rsqrt(r2), ir5 = ir * ir * ir * ir * ir, ir7 = ir5 * ir * ir;
	const int ab[6][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}};
	for (int c = 0; c < 6; ++c) {
		const int a = ab[c][0], b = ab[c][1];
		double t = -15.0 * P[a] * P[b] * P[A] * ir7;
		if (a == b) t += 3.0 * P[A] * ir5;
		if (a == A) t += 3.0 * P[b] * ir5;
		if (b == A) t += 3.0 * P[a] * ir5;
		v[c] += f * t;
	}
}

// The images P + r L e_A for r >= TAIL_M, in place of their sum: the midpoint rule with its first
// Euler-Maclaurin correction, L^-1 int_{s_M}^inf f + (L / 24) d_A f(s_M), s_M = P + (TAIL_M - 1/2) L e_A
// (the next term is below 1e-9 of the sum).
__device__ void line_continuum(double P[3], int A, double L, double V4, double *v)
{
	const double p0 = P[A];
	P[A] = p0 + (TAIL_M - 0.5) * L;
	line_integral(P, A, V4 / L, v);
	line_derivative(P, A, V4 * L / 24.0, v);
	P[A] = p0;
}

// Images P + r L e_A, r >= 0 (point dipoles of one cell).
__device__ void line_tail(double P[3], int A, double L, double V4, double *v)
{
	const double p0 = P[A];
	for (int r = 0; r < TAIL_M; ++r) {
		P[A] = p0 + r * L;
		point_dipole(P, V4, v);
	}
	P[A] = p0;
	line_continuum(P, A, L, V4, v);
}

// Images P + r L_A e_A + s L_B e_B, r, s >= 0.
__device__ void corner_tail(double P[3], int A, int B, double LA, double LB, double V4, double *v)
{
	const double pa = P[A], pb = P[B];
	for (int s = 0; s < TAIL_M; ++s) {
		P[B] = pb + s * LB;
		for (int r = 0; r < TAIL_M; ++r) {
			P[A] = pa + r * LA;
			point_dipole(P, V4, v);
		}
		P[A] = pa;
		line_continuum(P, A, LA, V4, v);
	}
	P[B] = pb;
	for (int r = 0; r < TAIL_M; ++r) {
		P[A] = pa + r * LA;
		line_continuum(P, B, LB, V4, v);
	}
	P[B] = pb + (TAIL_M - 0.5) * LB;
	P[A] = pa + (TAIL_M - 0.5) * LA;
	quadrant_integral(P, A, B, V4 / (LA * LB), v);
	P[A] = pa;
	P[B] = pb;
}

// Sum over images of the negated tensor of source offset (i, j, k), halved for each coordinate
// at zero displacement, plus the far images (tails); out[6] per source offset.
__global__ void __launch_bounds__(128) k_tensor_images(int nx, int ny, int nz, double dx, double dy, double dz,
                                                       int Rx, int Ry, int Rz, int tails, NearBox nb,
                                                       const double2 *__restrict__ gl, double *__restrict__ out)
{
	const size_t cnt = (size_t)nx * ny * nz;
	const int n3[3] = {nx, ny, nz}, R3[3] = {Rx, Ry, Rz};
	const double d3[3] = {dx, dy, dz};
	const double V4 = dx * dy * dz / (4.0 * PI);
	for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < cnt; q += (size_t)gridDim.x * blockDim.x) {
		const int ijk[3] = {(int)(q % nx), (int)((q / nx) % ny), (int)(q / ((size_t)nx * ny))};
		double S[6] = {0, 0, 0, 0, 0, 0};
		for (int rz = 0; rz < Rz; ++rz)
			for (int ry = 0; ry < Ry; ++ry)
				for (int rx = 0; rx < Rx; ++rx) {
					const int I = ijk[0] + rx * nx, J = ijk[1] + ry * ny, K = ijk[2] + rz * nz;
					const double w = (I == 0 ? 0.5 : 1.0) * (J == 0 ? 0.5 : 1.0) * (K == 0 ? 0.5 : 1.0);
					double v[6];
					tensor_at(I, J, K, dx, dy, dz, nb, gl, v);
					for (int c = 0; c < 6; ++c) S[c] += w * v[c];
				}
		if (tails) {
			// one periodic axis beyond its repetitions, the others within theirs (tensor.cpp:60-104)
			for (int A = 0; A < 3; ++A) {
				if (R3[A] <= 1) continue;
				const int B = (A + 1) % 3, C = (A + 2) % 3;
				for (int rc = 0; rc < R3[C]; ++rc)
					for (int rb = 0; rb < R3[B]; ++rb) {
						const int IB = ijk[B] + rb * n3[B], IC = ijk[C] + rc * n3[C];
						const double w = (IB == 0 ? 0.5 : 1.0) * (IC == 0 ? 0.5 : 1.0);
						double P[3];
						P[A] = (ijk[A] + R3[A] * n3[A]) * d3[A];
						P[B] = IB * d3[B];
						P[C] = IC * d3[C];
						double v[6] = {0, 0, 0, 0, 0, 0};
						line_tail(P, A, n3[A] * d3[A], V4, v);
						for (int c = 0; c < 6; ++c) S[c] += w * v[c];
					}
			}
			// two periodic axes beyond their repetitions (tensor.cpp:105-161)
			for (int A = 0; A < 3; ++A)
				for (int B = A + 1; B < 3; ++B) {
					if (R3[A] <= 1 || R3[B] <= 1) continue;
					const int C = 3 - A - B;
					for (int rc = 0; rc < R3[C]; ++rc) {
						const int IC = ijk[C] + rc * n3[C];
						const double w = IC == 0 ? 0.5 : 1.0;
						double P[3];
						P[A] = (ijk[A] + R3[A] * n3[A]) * d3[A];
						P[B] = (ijk[B] + R3[B] * n3[B]) * d3[B];
						P[C] = IC * d3[C];
						double v[6] = {0, 0, 0, 0, 0, 0};
						corner_tail(P, A, B, n3[A] * d3[A], n3[B] * d3[B], V4, v);
						for (int c = 0; c < 6; ++c) S[c] += w * v[c];
					}
				}
		}
		for (int c = 0; c < 6; ++c) out[6 * q + c] = S[c];
	}
}

// Every entry (I, J, K) of the padded tensor gathers its sources of the eight octants: along an
// axis, octant o = +-1 reads source offset (o I + e) mod e when that is below n (tensor.cpp:166-180
// scatters the same sums), with the parity signs of the off-diagonal components.
__global__ void __launch_bounds__(128) k_tensor_gather(int nx, int ny, int nz, int ex, int ey, int ez,
                                                       const double *__restrict__ S, double *__restrict__ out)
{
	const size_t cnt = (size_t)ex * ey * ez;
	for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < cnt; q += (size_t)gridDim.x * blockDim.x) {
		const int I = (int)(q % ex), J = (int)((q / ex) % ey), K = (int)(q / ((size_t)ex * ey));
		double acc[6] = {0, 0, 0, 0, 0, 0};
		for (int o = -1; o <= 1; o += 2) {
			const int i = (o * I + ex) % ex;
			if (i >= nx) continue;
			for (int p = -1; p <= 1; p += 2) {
				const int j = (p * J + ey) % ey;
				if (j >= ny) continue;
				for (int r = -1; r <= 1; r += 2) {
					const int k = (r * K + ez) % ez;
					if (k >= nz) continue;
					const double *s = S + 6 * (((size_t)k * ny + j) * nx + i);
					acc[0] += s[0];
					acc[1] += o * p * s[1];
					acc[2] += o * r * s[2];
					acc[3] += s[3];
					acc[4] += p * r * s[4];
					acc[5] += s[5];
				}
			}
		}
		for (int c = 0; c < 6; ++c) out[6 * q + c] = acc[c];
	}
}

} // namespace

mm_status tensor_octant(int nx, int ny, int nz, double dx, double dy, double dz, double *N, cudaStream_t st)
{
	return tensor_run<true>(nx, ny, nz, dx, dy, dz, nx, ny, nz, N, st);
}

} // namespace mm

using namespace mm;

extern "C" {

MM_API int mm_round_tensor_dimension(int dim, int periodic, int padding)
{
	// mmm/demag/tensor_round.cpp:90-106
	if (periodic) return dim;
	const int t = 2 * dim - 1;
	if (t == 1) return 1;
	auto round_to = [](int x, int m) { return (x % m) ? x + (m - x % m) : x; };
	switch (padding) {
	case MM_PADDING_DISABLE: return t;
	case MM_PADDING_ROUND_2: return round_to(t, 2);
	case MM_PADDING_ROUND_4: return round_to(t, 4);
	case MM_PADDING_ROUND_8: return round_to(t, 8);
	case MM_PADDING_ROUND_POT: { int p = 1; while (p < t) p <<= 1; return p; }
	case MM_PADDING_SMALL_PRIME_FACTORS: {
		int x = t + 1;
		for (;; ++x) {
			int m = x;
			for (int p : {2, 3, 5}) while (m % p == 0) m /= p;
			if (m == 1) return x;
		}
	}
	default: return -1;
	}
}

MM_API mm_status mm_demag_tensor(int nx, int ny, int nz, double dx, double dy, double dz, int ex,
                                 int ey, int ez, double *N_out, void *stream)
{
	if (nx <= 0 || ny <= 0 || nz <= 0 || !(dx > 0) || !(dy > 0) || !(dz > 0) || !N_out)
		return fail(MM_ERR_INVALID_ARGUMENT, "mm_demag_tensor: invalid argument");
	if (ex < 2 * nx - 1 || ey < 2 * ny - 1 || ez < 2 * nz - 1)
		return fail(MM_ERR_UNSUPPORTED,
		            "mm_demag_tensor: padded sizes below 2n-1 (periodic boundaries) are not supported");
	cudaStream_t st = as_stream(stream);
	MM_CUDA(cudaMemsetAsync(N_out, 0, sizeof(double) * 6 * (size_t)ex * ey * ez, st));
	return tensor_run<false>(nx, ny, nz, dx, dy, dz, ex, ey, ez, N_out, st);
}

MM_API mm_status mm_demag_tensor_periodic(int nx, int ny, int nz, double dx, double dy, double dz, int pbc_x,
                                          int pbc_y, int pbc_z, int repeat, int ex, int ey, int ez, double *N_out,
                                          void *stream)
{
	if (nx <= 0 || ny <= 0 || nz <= 0 || !(dx > 0) || !(dy > 0) || !(dz > 0) || !N_out || repeat < 1)
		return fail(MM_ERR_INVALID_ARGUMENT, "mm_demag_tensor_periodic: invalid argument");
	const int n3[3] = {nx, ny, nz}, e3[3] = {ex, ey, ez}, pb[3] = {pbc_x, pbc_y, pbc_z};
	for (int a = 0; a < 3; ++a)
		if (pb[a] ? e3[a] != n3[a] : e3[a] < 2 * n3[a] - 1)
			return fail(MM_ERR_INVALID_ARGUMENT, "mm_demag_tensor_periodic: a periodic axis needs e == n, the "
			                                     "others e >= 2n - 1 (round_tensor_dimension)");
	if (!pbc_x && !pbc_y && !pbc_z) return mm_demag_tensor(nx, ny, nz, dx, dy, dz, ex, ey, ez, N_out, stream);
	cudaStream_t st = as_stream(stream);
	GLTable *gl = nullptr;
	MM_TRY(gl_table(&gl));
	const size_t cnt = (size_t)nx * ny * nz;
	const char *off = std::getenv("MAGNUM_DEMAG_NO_INFINITY_CORRECTION");  // tensor.cpp:45
	const int Rx = pbc_x ? repeat : 1, Ry = pbc_y ? repeat : 1, Rz = pbc_z ? repeat : 1;
	NearBox nb;  // (the images' offsets run past the mesh)
	auto reach = [](int n, int R) { return (int)std::min<long long>((long long)n * R, 1 << 30); };
	near_extents(reach(nx, Rx), reach(ny, Ry), reach(nz, Rz), dx, dy, dz, nb);
	nb.lx = nb.x;
	nb.ly = nb.y;
	double *S = nullptr;  // the source offsets' sums, then the near box
	MM_CUDA(cudaMallocAsync(&S, 6 * (cnt + (size_t)nb.x * nb.y * nb.z) * sizeof(double), st));
	nb.v = S + 6 * cnt;
	mm_status r = tensor_near(nb, dx, dy, dz, gl->xw, st);
	const size_t want = (cnt + 127) / 128;
	if (r == MM_OK) {
		k_tensor_images<<<(int)(want < 65535u * 16 ? want : 65535u * 16), 128, 0, st>>>(
		    nx, ny, nz, dx, dy, dz, Rx, Ry, Rz, off ? 0 : 1, nb, gl->xw, S);
		r = after_launch("k_tensor_images");
	}
	if (r == MM_OK) {
		const size_t out = (size_t)ex * ey * ez, w2 = (out + 127) / 128;
		k_tensor_gather<<<(int)(w2 < 65535u * 16 ? w2 : 65535u * 16), 128, 0, st>>>(nx, ny, nz, ex, ey, ez, S, N_out);
		r = after_launch("k_tensor_gather");
	}
	cudaFreeAsync(S, st);
	return r;
}

} // extern "C"
