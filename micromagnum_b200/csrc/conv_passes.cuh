// Demag convolution H = N * M, zero-padded to (px, py, pz), as shared-memory FFT passes over
// HBM-resident spectra.  Replaces the reference's MatrixVectorConvolution_FFT::execute
// (math/conv/MatrixVectorConvolution_FFT.cpp:110-375): pad, 3x R2C along x, transpose,
// 3x C2C along y, transpose, 3x C2C along z, tensor multiply, and the inverses.
//
// B200 design:
//  * no transposes: the y and z passes read tiles of TB consecutive x-frequencies per row, so
//    every global access is a contiguous run of TB complex numbers;
//  * zero padding is never stored: the x pass reads only the nx real samples of each row and
//    writes only the rows y < ny, z < nz; the y pass pads in shared memory; the z pass pads,
//    transforms, multiplies, inverse-transforms and writes back only z < nz;
//  * two real rows share one complex FFT in the x passes (z = a + i b);
//  * the tensor spectrum is real (Nxx, Nyy, Nzz even in every axis; Nxy, Nxz, Nyz odd in
//    exactly two), so only Re N^ on ky <= py/2, kz <= pz/2 is stored, with the parity signs
//    restored on the fly: 4x fewer tensor bytes than the reference's 12 complex matrices
//    (SymmetricMatrixVectorConvolution_FFT.cpp:60-64 notes but does not use this);
//  * for 2-D problems (nz == 1) the forward y FFT, the multiply and the inverse y FFT are one
//    kernel.
// Spectra layout: cplx<T> S[c][z][y][kx], c < 3, z < nz, y < py, kx < hx, rows lx >= hx apart
// (lx even in FP32, so that every row starts on a 16-byte boundary).
//
// This header holds the passes and their set-up and dispatch as templates; conv_f64.cu and conv_f32.cu
// instantiate them per precision, conv_group.cu the grouped forms (one translation unit took over
// five minutes to compile).
#pragma once

#include "conv.cuh"
#include "fft_reg.cuh"
#include "tma.cuh"

#include <cmath>
#include <cstdlib>
#include <vector>
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

namespace mm {
namespace {

// Run flags of a batch member whose convolution runs as passes of its own: flags[0] == 0 skips it, and with
// gate != 0 so does flags[gate] == 0.
struct Gate {
	const int *flags = nullptr;
	int gate = 0;
	__device__ __forceinline__ bool skip() const { return flags && (!flags[0] || (gate && !flags[gate])); }
};

constexpr int NT = 256;                 // threads per CTA for all passes
constexpr size_t SMEM_TARGET = 100 * 1024;

// Twiddles of a plan's axis: the plain table W_n^k of the mixed-radix passes, rounded, and, for powers of
// two (and three times one) behind it the per-pass tables of the register passes (fft_tw_off), the
// usual radices first, then those of radix 8.
template <class C>
__host__ __device__ __forceinline__ const C *tw_of(const C *base, int n, int R)
{
	return base + (size_t)n * (R == 8 ? 2 : 1);
}
// The pair of T next to (c, s), a point of the unit circle, whose modulus is closest to one: its own
// rounding would scale every line of both transforms alike, while an error of the angle turns the
// inverse back by what the forward transform turned (mul_w).  Among the neighbours one step away, the
// error of the modulus weighs 16 times that of the angle.
template <typename T>
cplx<T> unit_near(long double c, long double s)
{
	cplx<T> best{(T)c, (T)s};
	if (best.x == 0 || best.y == 0) return best;
	long double least = 1;
	for (T x : {(T)c, std::nextafter((T)c, T(2)), std::nextafter((T)c, T(-2))})
		for (T y : {(T)s, std::nextafter((T)s, T(2)), std::nextafter((T)s, T(-2))}) {
			const long double ex = x - c, ey = y - s, mod = ex * c + ey * s, ang = ey * c - ex * s;
			const long double cost = 16 * mod * mod + ang * ang;
			if (cost < least) {
				least = cost;
				best = {x, y};
			}
		}
	return best;
}

template <typename T>
mm_status make_twiddles(int n, void **out)
{
	std::vector<cplx<T>> h((size_t)n * TW_SETS, cplx<T>{0, 0});
	const bool ct = fft_is_pow2(n) || (n % 3 == 0 && fft_is_pow2(n / 3)), oct = ct && n % 8 == 0;
	std::vector<cplx<T>> u(oct ? n : 0);  // the values of the pass tables
	// (for the lengths with passes of their own an eighth of the circle, and the rest by symmetry)
	for (int k = 0; k < (oct ? n / 8 + 1 : n); ++k) {
		const long double a = -2.0L * 3.14159265358979323846264338327950288L * (long double)k / (long double)n;
		const long double c = cosl(a), s = sinl(a);
		h[k] = {(T)c, (T)s};
		if (oct) u[k] = unit_near<T>(c, s);
	}
	if (oct)
		for (cplx<T> *w : {h.data(), u.data()}) {
			for (int k = n / 8 + 1; k <= n / 4; ++k) w[k] = {-w[n / 4 - k].y, -w[n / 4 - k].x};
			for (int k = n / 4 + 1; k < n; ++k) w[k] = {w[k - n / 4].y, -w[k - n / 4].x};
		}
	if (ct)
		for (int R : {fft_is_pow2(n) ? 16 : 24, 8}) {
			if (n < R || (R == 8 && !fft_is_pow2(n))) continue;
			cplx<T> *t = h.data() + (tw_of<cplx<T>>(nullptr, n, R) - (const cplx<T> *)nullptr);
			for (int p = 1, ns = fft_radix(n, R, 0); p < fft_npasses(n, R); ++p) {
				const int rp = fft_radix(n, R, p);
				for (int q = 1; q < rp; ++q)
					for (int jm = 0; jm < ns; ++jm)
						t[fft_tw_off(n, R, p) + (q - 1) * ns + jm] = (oct ? u : h)[(size_t)q * jm * (n / (ns * rp))];
				ns *= rp;
			}
		}
	MM_CUDA(cudaMalloc(out, sizeof(cplx<T>) * h.size()));
	MM_CUDA(cudaMemcpy(*out, h.data(), sizeof(cplx<T>) * h.size(), cudaMemcpyHostToDevice));
	return MM_OK;
}

template <typename T>
__device__ __forceinline__ void load_twiddles(cplx<T> *tw_s, const cplx<T> *tw_g, int n)
{
	const int tid = threadIdx.x, nthr = blockDim.x;
	for (int k = tid; k < n; k += nthr) tw_s[k] = tw_g[k];
}

// ---- x forward: real rows -> half spectra ------------------------------------------------------
// Real row r = (c*nz + z)*ny + y is M[r*nx .. r*nx+nx); its spectrum goes to S row
// (c*nz + z)*py + y.  Rows 2q and 2q+1 share complex line q.
template <typename T, bool SCALE>
__global__ void __launch_bounds__(NT) k_x_fwd(const T *__restrict__ M, const uint8_t *__restrict__ reg,
                                             const T *__restrict__ ms_tab, cplx<T> *__restrict__ S,
                                             int nx, int ny, int nz, int py, int hx, int lx, FftRadices rad,
                                             const cplx<T> *__restrict__ tw_g, int LP)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int px = rad.n;
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + px;
	C *b1 = b0 + (size_t)LP * px;
	load_twiddles<T>(tw, tw_g, px);
	const int rows = 3 * ny * nz;
	const int nyz = ny * nz;
	const int line0 = blockIdx.x * LP;
	for (int e = threadIdx.x; e < LP * px; e += blockDim.x) {
		const int b = e / px, x = e % px;
		const int ra = 2 * (line0 + b), rb = ra + 1;
		T a = 0, bb = 0;
		if (x < nx) {
			if (ra < rows) {
				a = M[(size_t)ra * nx + x];
				if (SCALE) a *= ms_tab[reg ? reg[(size_t)(ra % nyz) * nx + x] : 0];
			}
			if (rb < rows) {
				bb = M[(size_t)rb * nx + x];
				if (SCALE) bb *= ms_tab[reg ? reg[(size_t)(rb % nyz) * nx + x] : 0];
			}
		}
		b0[e] = C{a, bb};
	}
	__syncthreads();
	C *res = fft_lines<T, false>(b0, b1, px, 1, LP, rad, tw);
	for (int e = threadIdx.x; e < LP * hx; e += blockDim.x) {
		const int b = e / hx, k = e % hx;
		const int ra = 2 * (line0 + b), rb = ra + 1;
		const C zk = res[b * px + k];
		const C zn = res[b * px + (px - k) % px];
		const T h = T(0.5);
		if (ra < rows) {
			const int c = ra / nyz, rem = ra % nyz;
			const size_t srow = (size_t)(c * nz + rem / ny) * py + rem % ny;
			S[srow * lx + k] = C{h * (zk.x + zn.x), h * (zk.y - zn.y)};
		}
		if (rb < rows) {
			const int c = rb / nyz, rem = rb % nyz;
			const size_t srow = (size_t)(c * nz + rem / ny) * py + rem % ny;
			S[srow * lx + k] = C{h * (zk.y + zn.y), h * (zn.x - zk.x)};
		}
	}
}

// ---- x inverse: half spectra -> real rows ------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(NT) k_x_inv(const cplx<T> *__restrict__ S, T *__restrict__ H,
                                             int nx, int ny, int nz, int py, int hx, int lx, FftRadices rad,
                                             const cplx<T> *__restrict__ tw_g, int LP)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int px = rad.n;
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + px;
	C *b1 = b0 + (size_t)LP * px;
	load_twiddles<T>(tw, tw_g, px);
	const int rows = 3 * ny * nz;
	const int nyz = ny * nz;
	const int line0 = blockIdx.x * LP;
	const bool even = (px % 2) == 0;
	for (int e = threadIdx.x; e < LP * px; e += blockDim.x) {
		const int b = e / px, k = e % px;
		const int ra = 2 * (line0 + b), rb = ra + 1;
		const bool mirror = k >= hx;
		const int kk = mirror ? px - k : k;
		// the imaginary parts at kx = 0 and at the Nyquist frequency of a real row are zero
		const bool realonly = (kk == 0) || (even && kk == px / 2);
		C A = {0, 0}, B = {0, 0};
		if (ra < rows) {
			const int c = ra / nyz, rem = ra % nyz;
			A = S[((size_t)(c * nz + rem / ny) * py + rem % ny) * lx + kk];
		}
		if (rb < rows) {
			const int c = rb / nyz, rem = rb % nyz;
			B = S[((size_t)(c * nz + rem / ny) * py + rem % ny) * lx + kk];
		}
		if (realonly) { A.y = 0; B.y = 0; }
		if (mirror) { A.y = -A.y; B.y = -B.y; }
		b0[e] = C{A.x - B.y, A.y + B.x};
	}
	__syncthreads();
	C *res = fft_lines<T, true>(b0, b1, px, 1, LP, rad, tw);
	for (int e = threadIdx.x; e < LP * nx; e += blockDim.x) {
		const int b = e / nx, x = e % nx;
		const int ra = 2 * (line0 + b), rb = ra + 1;
		const C z = res[b * px + x];
		if (ra < rows) H[(size_t)ra * nx + x] = z.x;
		if (rb < rows) H[(size_t)rb * nx + x] = z.y;
	}
}

// ---- y pass (3-D): column tiles, forward pads ny -> py, inverse crops py -> ny -----------------
template <typename T, bool INV>
__global__ void __launch_bounds__(NT) k_y(cplx<T> *__restrict__ S, int n_in, int n_out, int nz,
                                         int py, int hx, int lx, FftRadices rad,
                                         const cplx<T> *__restrict__ tw_g, int TB)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + py;
	C *b1 = b0 + (size_t)TB * py;
	load_twiddles<T>(tw, tw_g, py);
	const int kx0 = blockIdx.x * TB;
	const int z = blockIdx.y, c = blockIdx.z;
	C *base = S + (size_t)(c * nz + z) * py * lx;
	for (int e = threadIdx.x; e < TB * py; e += blockDim.x) {
		const int y = e / TB, b = e % TB;
		b0[e] = (y < n_in && kx0 + b < hx) ? base[(size_t)y * lx + kx0 + b] : C{0, 0};
	}
	__syncthreads();
	C *res = fft_lines<T, INV>(b0, b1, 1, TB, TB, rad, tw);
	for (int e = threadIdx.x; e < TB * n_out; e += blockDim.x) {
		const int y = e / TB, b = e % TB;
		if (kx0 + b < hx) base[(size_t)y * lx + kx0 + b] = res[e];
	}
}

// Real tensor spectrum with parity signs restored.  t points at component 0 of
// (kz', ky', kx); cs = component stride.
template <typename T, typename C>
__device__ __forceinline__ void tensor_apply(const T *__restrict__ t, size_t cs, T sy, T sz, C &m0,
                                             C &m1, C &m2)
{
	const T nxx = t[0], nxy = sy * t[cs], nxz = sz * t[2 * cs];
	const T nyy = t[3 * cs], nyz = sy * sz * t[4 * cs], nzz = t[5 * cs];
	const C a = m0, b = m1, c = m2;
	m0 = C{nxx * a.x + nxy * b.x + nxz * c.x, nxx * a.y + nxy * b.y + nxz * c.y};
	m1 = C{nxy * a.x + nyy * b.x + nyz * c.x, nxy * a.y + nyy * b.y + nyz * c.y};
	m2 = C{nxz * a.x + nyz * b.x + nzz * c.x, nxz * a.y + nyz * b.y + nzz * c.y};
}

// ---- z pass (3-D): forward FFT along z, tensor multiply, inverse FFT, all three components ----
template <typename T>
__global__ void __launch_bounds__(NT) k_z_mul(cplx<T> *__restrict__ S, const T *__restrict__ Nt,
                                             int nz, int py, int hx, int lx, int qy, int qz, FftRadices rad,
                                             const cplx<T> *__restrict__ tw_g, int TB)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int pz = rad.n;
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + pz;
	C *b1 = b0 + (size_t)3 * TB * pz;
	load_twiddles<T>(tw, tw_g, pz);
	const int kx0 = blockIdx.x * TB;
	const int ky = blockIdx.y;
	const int L = 3 * TB;
	const size_t cstride = (size_t)nz * py * lx;
	for (int e = threadIdx.x; e < L * pz; e += blockDim.x) {
		const int zz = e / L, l = e % L, c = l / TB, b = l % TB;
		b0[e] = (zz < nz && kx0 + b < hx) ? S[c * cstride + ((size_t)zz * py + ky) * lx + kx0 + b] : C{0, 0};
	}
	__syncthreads();
	C *res = fft_lines<T, false>(b0, b1, 1, L, L, rad, tw);
	C *other = (res == b0) ? b1 : b0;
	const bool fy = ky > py / 2;
	const int kyr = fy ? py - ky : ky;
	const T sy = fy ? T(-1) : T(1);
	const size_t cs = (size_t)qz * qy * hx;
	for (int e = threadIdx.x; e < pz * TB; e += blockDim.x) {
		const int kz = e / TB, b = e % TB;
		if (kx0 + b >= hx) continue;
		const bool fz = kz > pz / 2;
		const int kzr = fz ? pz - kz : kz;
		const T sz = fz ? T(-1) : T(1);
		const T *t = Nt + ((size_t)kzr * qy + kyr) * hx + kx0 + b;
		C &m0 = res[kz * L + b], &m1 = res[kz * L + TB + b], &m2 = res[kz * L + 2 * TB + b];
		tensor_apply<T, C>(t, cs, sy, sz, m0, m1, m2);
	}
	__syncthreads();
	C *out = fft_lines<T, true>(res, other, 1, L, L, rad, tw);
	for (int e = threadIdx.x; e < L * nz; e += blockDim.x) {
		const int zz = e / L, l = e % L, c = l / TB, b = l % TB;
		if (kx0 + b < hx) S[c * cstride + ((size_t)zz * py + ky) * lx + kx0 + b] = out[e];
	}
}

// ---- y pass with multiply (2-D problems): forward y FFT, tensor multiply, inverse y FFT -------
template <typename T>
__global__ void __launch_bounds__(NT) k_y_mul2d(cplx<T> *__restrict__ S, const T *__restrict__ Nt,
                                               int ny, int hx, int lx, int qy, FftRadices rad,
                                               const cplx<T> *__restrict__ tw_g, int TB)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int py = rad.n;
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + py;
	C *b1 = b0 + (size_t)3 * TB * py;
	load_twiddles<T>(tw, tw_g, py);
	const int kx0 = blockIdx.x * TB;
	const int L = 3 * TB;
	const size_t cstride = (size_t)py * lx;
	for (int e = threadIdx.x; e < L * py; e += blockDim.x) {
		const int y = e / L, l = e % L, c = l / TB, b = l % TB;
		b0[e] = (y < ny && kx0 + b < hx) ? S[c * cstride + (size_t)y * lx + kx0 + b] : C{0, 0};
	}
	__syncthreads();
	C *res = fft_lines<T, false>(b0, b1, 1, L, L, rad, tw);
	C *other = (res == b0) ? b1 : b0;
	const size_t cs = (size_t)qy * hx;  // qz == 1
	for (int e = threadIdx.x; e < py * TB; e += blockDim.x) {
		const int ky = e / TB, b = e % TB;
		if (kx0 + b >= hx) continue;
		const bool fy = ky > py / 2;
		const int kyr = fy ? py - ky : ky;
		const T sy = fy ? T(-1) : T(1);
		const T *t = Nt + (size_t)kyr * hx + kx0 + b;
		C &m0 = res[ky * L + b], &m1 = res[ky * L + TB + b], &m2 = res[ky * L + 2 * TB + b];
		tensor_apply<T, C>(t, cs, sy, T(1), m0, m1, m2);
	}
	__syncthreads();
	C *out = fft_lines<T, true>(res, other, 1, L, L, rad, tw);
	for (int e = threadIdx.x; e < L * ny; e += blockDim.x) {
		const int y = e / L, l = e % L, c = l / TB, b = l % TB;
		if (kx0 + b < hx) S[c * cstride + (size_t)y * lx + kx0 + b] = out[e];
	}
}

// ---- set-up: the tensor's spectrum, one axis at a time, on one octant ----------------------------
// Every component of the tensor is even or odd along each axis, so its transform along an axis is
// real (even) or imaginary (odd, the stored value is its imaginary part) and is known from half of
// it, in space and in frequency.  A pass therefore reads offsets k < m of real lines, extends them by
// their parity in shared memory, and keeps the frequencies f <= len/2 as real numbers; two
// components of equal parity share one complex FFT (their spectra come out as its real and
// imaginary part).  All passes in FP64.  Against complex FFTs of the whole padded array, component by
// component, that is a sixteenth of the bytes of a 3-D box: 0.19 ms against 1.6 at 240x120x10 cells.
struct SpecPass {
	const double *in;            // in[c ic + o io + k ik + i ii]: component, outer, along the axis, inner
	size_t ic, io, ik, ii;
	size_t oc, oo, ok, oi;       // the output's strides
	int m, inner;                // offsets given along the axis, inner lines per outer index
	int a[3], b[3], odd[3];      // the pairs of components and their parity along this axis
	int part;                    // the tensor's part (0, or 3, 5, 6: tensor_mixed_parity)
	bool add;                    // adds to the output
	double scale;                // of the outputs; with signs, the components odd along two axes get -scale (i * i)
	bool signs;
};

// One CTA: TB lines of one outer index (blockIdx.y) and one pair (blockIdx.z).  KFAST: the axis is the
// contiguous one, so a warp loads along it; else along the inner lines.
template <typename OUT, bool KFAST>
__global__ void __launch_bounds__(NT) k_spec_axis(SpecPass s, OUT *__restrict__ out, FftRadices rad,
                                                 const double2 *__restrict__ tw_g, int TB)
{
	using C = double2;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int len = rad.n, q = len / 2 + 1;
	C *tw = reinterpret_cast<C *>(smem_raw);
	C *b0 = tw + len;
	C *b1 = b0 + (size_t)TB * len;
	load_twiddles<double>(tw, tw_g, len);
	const int i0 = blockIdx.x * TB, pr = blockIdx.z;
	const bool odd = s.odd[pr];
	const double *ina = s.in + (size_t)s.a[pr] * s.ic + blockIdx.y * s.io;
	const double *inb = s.in + (size_t)s.b[pr] * s.ic + blockIdx.y * s.io;
	for (int e = threadIdx.x; e < TB * len; e += blockDim.x) {
		const int k = KFAST ? e % len : e / TB, b = KFAST ? e / len : e % TB;
		const bool back = k >= s.m;
		const int src = back ? len - k : k;
		C v{0, 0};
		// (an odd component vanishes where an offset is its own mirror)
		if (i0 + b < s.inner && src < s.m && !(odd && (k == 0 || 2 * k == len))) {
			const size_t at = src * s.ik + (size_t)(i0 + b) * s.ii;
			v = C{ina[at], inb[at]};
			if (back && odd) v = C{-v.x, -v.y};
		}
		b0[e] = v;
	}
	__syncthreads();
	C *res = KFAST ? fft_lines<double, false>(b0, b1, len, 1, TB, rad, tw) : fft_lines<double, false>(b0, b1, 1, TB, TB, rad, tw);
	OUT *oa = out + (size_t)s.a[pr] * s.oc + blockIdx.y * s.oo, *ob = out + (size_t)s.b[pr] * s.oc + blockIdx.y * s.oo;
	const double sa = s.signs && component_parity(s.a[pr]) != s.part ? -s.scale : s.scale;
	const double sb = s.signs && component_parity(s.b[pr]) != s.part ? -s.scale : s.scale;
	for (int e = threadIdx.x; e < TB * q; e += blockDim.x) {
		const int k = KFAST ? e % q : e / TB, b = KFAST ? e / q : e % TB;
		if (i0 + b >= s.inner) continue;
		const C z = res[KFAST ? b * len + k : k * TB + b];
		const size_t at = k * s.ok + (size_t)(i0 + b) * s.oi;
		const double va = sa * (odd ? z.y : z.x), vb = sb * (odd ? -z.x : z.y);  // odd: z = i A - B
		oa[at] = (OUT)(s.add ? (double)oa[at] + va : va);
		ob[at] = (OUT)(s.add ? (double)ob[at] + vb : vb);
	}
}

int pick_tile(int len, int ncomp, size_t elem, int cap)
{
	int tb = cap;
	while (tb > 1 && (size_t)(2 * ncomp * tb + 1) * len * elem > SMEM_TARGET) tb >>= 1;
	return tb;
}

// Lets fn take `bytes` of dynamic shared memory.  The attribute belongs to the kernel, not to a plan, and plans of
// different lengths share kernels, so it is always set to all that the device allows: set to each plan's
// own need, a later plan with less would have an earlier one's launches refused.
template <typename T>
mm_status set_smem(const void *fn, size_t bytes)
{
	if (bytes <= 48 * 1024) return MM_OK;
	int dev = 0, most = 0;
	MM_CUDA(cudaGetDevice(&dev));
	MM_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
	cudaFuncAttributes a{};
	MM_CUDA(cudaFuncGetAttributes(&a, fn));
	most -= (int)a.sharedSizeBytes;
	if (bytes > (size_t)most) return fail(MM_ERR_UNSUPPORTED, "conv: more shared memory than a block can have");
	MM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
	return MM_OK;
}

// ---- CTA-Stockham passes (cta_fft, radix 16 in registers, shared-memory passes) -----------------
__host__ __device__ constexpr int ct_radix(int n) { return fft_is_pow2(n) ? (n < 16 ? n : 16) : n < 24 ? n : 24; }
__host__ __device__ constexpr int ct_radix8(int n) { return n < 8 ? n : 8; }
__host__ __device__ constexpr int ct_tb(int n, int csize)
{
	int tb = 32;
	while (tb > 1 && ((long)n * tb * csize > 65536 || tb * (n / ct_radix(n)) > 512)) tb >>= 1;
	return tb;
}
__host__ __device__ constexpr int ct_lpb(int n, int csize)
{
	int l = 256 / (n / ct_radix(n));
	if (l < 1) l = 1;
	while (l > 1 && (long)(l * n + (l * n >> 5) + 1) * csize > 65536) l >>= 1;
	return l;
}

// Tiles of a grid that would not fill the device with the sizes above: one warp's worth of lines,
// and rows of at least 32 bytes in the y pass.  A 128x32 film has 48 lines in its x passes, 3 CTAs of
// 16 lines, each waiting on its own passes: 24 CTAs of 2 lines take 12.8 us forward, FP64, against
// 14.0 (event-timed, about 6 us of it the timing).
__host__ __device__ constexpr int ct_lpb_narrow(int n)
{
	const int l = 32 / (n / ct_radix(n));
	return l < 1 ? 1 : l;
}
__host__ __device__ constexpr int ct_tb_narrow(int n, int csize)
{
	int tb = 32 / csize;
	while (tb * (n / ct_radix(n)) < 32) tb <<= 1;
	return tb < ct_tb(n, csize) ? tb : ct_tb(n, csize);
}

// y pass (3-D): TB columns per CTA; forward pads rows n_in -> N, inverse crops N -> n_out.
// (bx: column tile, plane = c nz + z; shared by the single-grid and the grouped kernels)
template <typename T, int N, int TB, bool INV, int R = ct_radix(N)>
__device__ __forceinline__ void y_ct_body(cplx<T> *__restrict__ S, int n_in, int n_out, int hx, int lx,
                                          const cplx<T> *__restrict__ twN, int bx, int plane)
{
	using C = cplx<T>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int line = tid & (TB - 1), j0 = tid / TB;  // N / R threads per column
	const int kx = bx * TB + line;
	const bool ok = kx < hx;
	C *base = S + (size_t)plane * N * lx + (ok ? kx : 0);
	auto ld = [&](int, int k) -> C { return (ok && k < n_in) ? base[(size_t)k * lx] : C{0, 0}; };
	auto st = [&](int, int k, C v) {
		if (ok && k < n_out) base[(size_t)k * lx] = v;
	};
	cta_fft<T, N, R, TB, INV, SmCols<N, TB>>(sm, twN, line, j0, ld, st);
}

template <typename T, int N, int TB, bool INV>
__global__ void __launch_bounds__(TB * (N / ct_radix(N)), 2) k_y_ct(cplx<T> *__restrict__ S, int n_in, int n_out, int nz,
                                                                 int hx, int lx, const cplx<T> *__restrict__ twN, Gate gate)
{
	if (gate.skip()) return;
	y_ct_body<T, N, TB, INV>(S, n_in, n_out, hx, lx, twN, blockIdx.x, blockIdx.z * nz + blockIdx.y);
}

__device__ const uint8_t g_region0 = 0;

// Spectrum rows of the real rows ra and ra + 1 (row (c nz + z) ny + y has row (c nz + z) py + y); row 0 for
// one that does not exist.
__device__ __forceinline__ void spec_rows(int ra, bool va, bool vb, int ny, int py, size_t &sa, size_t &sb)
{
	const int plane = (va ? ra : 0) / ny, y = (va ? ra : 0) - plane * ny;
	sa = (size_t)plane * py + y;
	sb = !vb ? 0 : y + 1 < ny ? sa + 1 : (size_t)(plane + 1) * py;
}

// x pass forward: LPB complex lines per CTA (line q packs real rows 2q, 2q+1).
template <typename T, int N, int LPB, bool SCALE, int R = ct_radix(N), bool H0 = false, bool PK = true>
__device__ __forceinline__ void x_fwd_ct_body(const T *__restrict__ M, const uint8_t *__restrict__ reg,
                                              const T *__restrict__ ms_tab, cplx<T> *__restrict__ S, int nx, int ny,
                                              int nz, int py, int hx, int lx, const cplx<T> *__restrict__ twN, int blk)
{
	using C = cplx<T>;
	constexpr int TPL = N / R;
	using SI = SmRows<N, LPB>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int line = tid / TPL, j0 = tid % TPL;
	const int rows = 3 * ny * nz, nyz = ny * nz;
	const int ra = 2 * (blk * LPB + line), rb = ra + 1;
	const bool va = ra < rows, vb = rb < rows;
	const int qa = va ? ra : 0, qb = vb ? rb : 0;
	const T *Ma = M + (size_t)qa * nx, *Mb = M + (size_t)qb * nx;
	// a box without a region map reads region 0 at every x
	const uint8_t *Ra = reg ? reg + (size_t)(qa % nyz) * nx : &g_region0;
	const uint8_t *Rb = reg ? reg + (size_t)(qb % nyz) * nx : &g_region0;
	const int rstep = reg ? 1 : 0;
	// Loads first and selects afterwards: behind branches the compiler issued the 2 R loads (and the scale
	// lookups that follow them) one after another, a memory latency each: 20 steps of a 128x32 film,
	// FP64, took 3.15 ms, against 2.77 this way.
	auto ld = [&](int, int x) -> C {
		const bool in = x < nx;
		const int xx = in ? x : 0;
		T a = Ma[xx], b = Mb[xx];
		if (SCALE) {
			a *= ms_tab[Ra[xx * rstep]];
			b *= ms_tab[Rb[xx * rstep]];
		}
		return C{in && va ? a : T(0), in && vb ? b : T(0)};
	};
	auto st = [&](int l, int k, C v) { sm[SI::at(l, k)] = v; };
	if constexpr (H0) cta_fft_h0<T, N, R, LPB, SI, false, PK>(sm, twN, line, j0, ld, st);
	else cta_fft<T, N, R, LPB, false, SI, false, PK>(sm, twN, line, j0, ld, st);
	__syncthreads();
	size_t sa, sb;
	spec_rows(ra, va, vb, ny, py, sa, sb);
	C *Sa = S + sa * lx, *Sb = S + sb * lx;
	const T h = T(0.5);
	auto out = [&](int k) {
		const C zk = sm[SI::at(line, k)], zn = sm[SI::at(line, k == 0 ? 0 : N - k)];
		if (va) Sa[k] = C{h * (zk.x + zn.x), h * (zk.y - zn.y)};
		if (vb) Sb[k] = C{h * (zk.y + zn.y), h * (zn.x - zk.x)};
	};
#pragma unroll
	for (int i = 0; i < R / 2; ++i) out(j0 + i * TPL);  // k < N/2, then the last stored frequency
	if (j0 == 0) out(N / 2);
}

// H0: at most N/2 samples, the upper half of the inputs is zero padding (not along a periodic axis).
template <typename T, int N, int LPB, bool SCALE, bool H0>
__global__ void __launch_bounds__(LPB * (N / ct_radix(N))) k_x_fwd_ct(const T *__restrict__ M,
                                                                     const uint8_t *__restrict__ reg,
                                                                     const T *__restrict__ ms_tab,
                                                                     cplx<T> *__restrict__ S, int nx, int ny, int nz,
                                                                     int py, int hx, int lx, const cplx<T> *__restrict__ twN, Gate gate)
{
	if (gate.skip()) return;
	x_fwd_ct_body<T, N, LPB, SCALE, ct_radix(N), H0, LPB != ct_lpb_narrow(N)>(M, reg, ms_tab, S, nx, ny, nz, py, hx, lx, twN, blockIdx.x);
}

// x pass inverse: half spectra of rows 2q, 2q+1 -> real rows.
template <typename T, int N, int LPB, int R = ct_radix(N), bool PK = true>
__device__ __forceinline__ void x_inv_ct_body(const cplx<T> *__restrict__ S, T *__restrict__ H, int nx, int ny,
                                              int nz, int py, int hx, int lx, const cplx<T> *__restrict__ twN, int blk)
{
	using C = cplx<T>;
	constexpr int TPL = N / R;
	using SI = SmRows<N, LPB>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int line = tid / TPL, j0 = tid % TPL;
	const int rows = 3 * ny * nz;
	const int ra = 2 * (blk * LPB + line), rb = ra + 1;
	const bool va = ra < rows, vb = rb < rows;
	const int qa = va ? ra : 0, qb = vb ? rb : 0;
	size_t sa, sb;
	spec_rows(ra, va, vb, ny, py, sa, sb);
	const C *Sa = S + sa * lx, *Sb = S + sb * lx;
	T *Ha = H + (size_t)qa * nx, *Hb = H + (size_t)qb * nx;
	auto ld = [&](int, int f) -> C {
		const bool mirror = 2 * f > N;
		const int ff = mirror ? N - f : f;
		C A = Sa[ff], B = Sb[ff];
		if (!vb) B = C{0, 0};
		if (ff == 0 || 2 * ff == N) { A.y = 0; B.y = 0; }
		if (mirror) { A.y = -A.y; B.y = -B.y; }
		return C{A.x - B.y, A.y + B.x};
	};
	auto st = [&](int, int x, C v) {
		if (x < nx) {
			if (va) Ha[x] = v.x;
			if (vb) Hb[x] = v.y;
		}
	};
	cta_fft<T, N, R, LPB, true, SI, false, PK>(sm, twN, line, j0, ld, st);
}

template <typename T, int N, int LPB>
__global__ void __launch_bounds__(LPB * (N / ct_radix(N))) k_x_inv_ct(const cplx<T> *__restrict__ S, T *__restrict__ H,
                                                                     int nx, int ny, int nz, int py, int hx, int lx,
                                                                     const cplx<T> *__restrict__ twN, Gate gate)
{
	if (gate.skip()) return;
	x_inv_ct_body<T, N, LPB, ct_radix(N), LPB != ct_lpb_narrow(N)>(S, H, nx, ny, nz, py, hx, lx, twN, blockIdx.x);
}

// y pass with the tensor multiply for 2-D problems (CTA-Stockham form): a CTA takes TB columns of
// x-frequencies of all three components (lines c * TB + b), transforms them along y into shared
// memory, and the inverse transform's first pass reads its inputs through the tensor (three
// components and three tensor entries per value), so the y spectrum never leaves the SM.  Bound by
// the latency of its passes for films of up to a few ten thousand cells: 128x32 cells, FP64, 8.6 us
// against 18.7 in the mixed-radix form (5 CTAs of 32 columns), 500x125 cells 14.7 against 27.2
// (event-timed, about 6 us of it the timing).  A CTA has at most 384 threads, which leaves each the 168
// registers that a radix-16 butterfly and its twiddles need: at 768 threads the FP32 passes spilled over a
// kilobyte a thread and an evaluation of 1024x1024 cells took 307 us (mixed radix: 278), against 148 with
// single columns; 640x480 133 (131), 62 with two; 512x512 51 (78), 42; 2000x400 395 (264), 221.  192
// threads are no better (640x480: 74, 700x700: 99 against 77).
__host__ __device__ constexpr int y2d_tb(int n, int csize)
{
	int tb = 8;
	while (tb > 1 && (3L * tb * n * csize > 100 * 1024 || 3 * tb * (n / ct_radix(n)) > 384)) tb >>= 1;
	return tb;
}

template <typename T, int N, int TB>
__global__ void __launch_bounds__(3 * TB * (N / ct_radix(N)))
    k_y2d_ct(cplx<T> *__restrict__ S, const T *__restrict__ Nt, int ny, int hx, int lx, int qy,
             const cplx<T> *__restrict__ twN)
{
	using C = cplx<T>;
	constexpr int R = ct_radix(N), LANES = 3 * TB;
	using SI = SmCols<N, LANES>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int line = tid % LANES, j0 = tid / LANES;
	const int c = line / TB, b = line % TB;
	const int kx = blockIdx.x * TB + b;
	const bool ok = kx < hx;
	C *col = S + (size_t)c * N * lx + (ok ? kx : 0);
	{
		auto ld = [&](int, int y) -> C { return (ok && y < ny) ? col[(size_t)y * lx] : C{0, 0}; };
		auto st = [&](int l, int k, C v) { sm[SI::at(l, k)] = v; };
		cta_fft<T, N, R, LANES, false, SI, false, TB != 1>(sm, twN, line, j0, ld, st);
	}
	__syncthreads();
	// row c of the symmetric tensor (components xx, xy, xz, yy, yz, zz); xy and yz are odd in ky
	const size_t cs = (size_t)qy * hx;
	const T *t0 = Nt + (size_t)c * cs + (ok ? kx : 0);
	const T *t1 = Nt + (size_t)(c == 0 ? 1 : c + 2) * cs + (ok ? kx : 0);
	const T *t2 = Nt + (size_t)(c == 0 ? 2 : c + 3) * cs + (ok ? kx : 0);
	auto ld = [&](int, int k) -> C {
		const bool f = 2 * k > N;
		const size_t r = (size_t)(f ? N - k : k) * hx;
		const T s = f ? T(-1) : T(1);
		T n0 = t0[r], n1 = t1[r], n2 = t2[r];
		if (c == 0) n1 = s * n1;
		else if (c == 1) { n0 = s * n0; n2 = s * n2; }
		else n1 = s * n1;
		const C m0 = sm[SI::at(b, k)], m1 = sm[SI::at(TB + b, k)], m2 = sm[SI::at(2 * TB + b, k)];
		return C{n0 * m0.x + n1 * m1.x + n2 * m2.x, n0 * m0.y + n1 * m1.y + n2 * m2.y};
	};
	auto st = [&](int, int y, C v) {
		if (ok && y < ny) col[(size_t)y * lx] = v;
	};
	cta_fft<T, N, R, LANES, true, SI, true, TB != 1>(sm, twN, line, j0, ld, st);
}

// z pass with the tensor multiply (CTA-Stockham form): lines (c, b) = c * TB + b hold the z
// column of component c at x-frequency kx0 + b; forward transform into shared memory, multiply by
// the real symmetric tensor (three components meet in shared memory), inverse transform to HBM.
template <typename T, int PZ, int TB>
__global__ void __launch_bounds__(3 * TB * (PZ / ct_radix8(PZ))) k_z_ct(cplx<T> *__restrict__ S,
                                                                        const T *__restrict__ Nt, int nz, int py,
                                                                        int hx, int lx, int qy, int qz,
                                                                        const cplx<T> *__restrict__ twN)
{
	using C = cplx<T>;
	constexpr int R = ct_radix8(PZ);
	constexpr int LANES = 3 * TB;
	using SI = SmCols<PZ, LANES>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);
	const int tid = threadIdx.x;
	const int line = tid % LANES, j0 = tid / LANES;
	const int c = line / TB, b = line % TB;
	const int ky = blockIdx.y;
	const size_t cstride = (size_t)nz * py * lx, zstride = (size_t)py * lx;
	{
		const int kx = blockIdx.x * TB + b;
		const bool ok = kx < hx;
		C *col = S + c * cstride + (size_t)ky * lx + (ok ? kx : 0);
		auto ld = [&](int, int z) -> C { return (ok && z < nz) ? col[z * zstride] : C{0, 0}; };
		auto st = [&](int l, int k, C v) { sm[SI::at(l, k)] = v; };
		cta_fft<T, PZ, R, LANES, false, SI>(sm, twN, line, j0, ld, st);
	}
	__syncthreads();
	const bool fy = ky > py / 2;
	const int kyr = fy ? py - ky : ky;
	const T sy = fy ? T(-1) : T(1);
	const size_t cs = (size_t)qz * qy * hx, kzs = (size_t)qy * hx;
	for (int idx = tid; idx < PZ * TB; idx += LANES * (PZ / R)) {
		const int kz = idx / TB, bb = idx % TB;
		const int kx = blockIdx.x * TB + bb;
		if (kx >= hx) continue;
		const bool fz = kz > PZ / 2;
		const int kzr = fz ? PZ - kz : kz;
		const T sz = fz ? T(-1) : T(1);
		const T *t = Nt + (size_t)kzr * kzs + (size_t)kyr * hx + kx;
		C &m0 = sm[SI::at(bb, kz)], &m1 = sm[SI::at(TB + bb, kz)], &m2 = sm[SI::at(2 * TB + bb, kz)];
		tensor_apply<T, C>(t, cs, sy, sz, m0, m1, m2);
	}
	{
		const int kx = blockIdx.x * TB + b;
		const bool ok = kx < hx;
		C *col = S + c * cstride + (size_t)ky * lx + (ok ? kx : 0);
		auto ld = [&](int l, int k) -> C { return sm[SI::at(l, k)]; };
		auto st = [&](int, int z, C v) {
			if (ok && z < nz) col[z * zstride] = v;
		};
		__syncthreads();
		cta_fft<T, PZ, R, LANES, true, SI, true>(sm, twN, line, j0, ld, st);
	}
}

// Asynchronous copy of one real value global -> shared (LDGSTS, 4 or 8 bytes).
template <typename T>
__device__ __forceinline__ void cp_async_t(T *dst, const T *src)
{
	const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
	if constexpr (sizeof(T) == 4)
		asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
	else
		asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all_t() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shared memory of the register z pass: the spectrum of two rows (2 PZ kz x 3 components x 32 kx)
// and the block's tensor entries ((PZ/2 + 1) x 6 x 32).
template <typename T>
constexpr size_t zr_smem(int pz) { return (size_t)2 * pz * 96 * 2 * sizeof(T) + (size_t)(pz / 2 + 1) * 192 * sizeof(T); }

// ---- z pass in registers ------------------------------------------------------------------------
// One thread per (kx, component, ky) column holds the whole length-PZ column in registers: the
// forward DFT (upper half zero padding, nz <= PZ/2), the tensor multiply through shared memory,
// and the inverse DFT, of which only the outputs z < nz are formed and stored.  A block covers
// 32 consecutive kx (one warp per component and row: coalesced 256-byte loads and stores) and the
// ky pair {b, py - b}, b = blockIdx.y <= py/2, whose tensor entries agree up to parity signs: each
// tensor value is read once per block and applied to up to four (ky, kz) combinations.
constexpr int ZR_THREADS = 192;  // 32 kx x 3 components x 2 rows

template <typename T, int PZ>
__device__ __forceinline__ void z_reg_body(cplx<T> *__restrict__ S, const T *__restrict__ Nt, int nz, int py, int hx,
                                           int lx, int qy, int qz, int bx, int b)
{
	using C = cplx<T>;
	constexpr int H = PZ / 2;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *sm = reinterpret_cast<C *>(smem_raw);  // [row][kz][component][32 kx]
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int c = w % 3, r = w / 3;
	const int b1 = py - b;
	const bool two = b > 0 && b1 != b;
	const int kx = bx * 32 + lane;
	const bool ok = (r == 0 || two) && kx < hx;
	const size_t zstride = (size_t)py * lx;
	C *col = S + ((size_t)c * nz * py + (size_t)(r == 0 ? b : b1)) * lx + kx;
	// the block's tensor entries (kz' <= pz/2, 6 components, 32 kx at ky' = b) come in by
	// asynchronous copies while the columns are loaded and transformed
	T *tens = reinterpret_cast<T *>(sm + 2 * PZ * 96);
	static_assert(ZR_THREADS == 192, "one thread per (tensor component, kx) of a kz plane");
	{
		// thread (warp w, lane) copies component w at kx for every kz' (one pointer step per plane)
		const size_t kzs = (size_t)qy * hx;
		const T *src = Nt + (size_t)w * qz * kzs + (size_t)b * hx + kx;
		if (kx < hx) {
#pragma unroll
			for (int kzr = 0; kzr <= H; ++kzr, src += kzs) cp_async_t(&tens[kzr * 192 + threadIdx.x], src);
		}
	}
	C v[PZ];
#pragma unroll
	for (int z = 0; z < H; ++z) v[z] = (ok && z < nz) ? col[z * zstride] : C{0, 0};
	dft_reg_halfzero<T, PZ>(v);
	C *mine = sm + (r * PZ * 3 + c) * 32 + lane;
#pragma unroll
	for (int k = 0; k < PZ; ++k) mine[k * 96] = v[dft_pos<PZ>(k)];
	cp_async_wait_all_t();
	__syncthreads();
	if (kx < hx) {
		for (int kzr = w; kzr <= H; kzr += ZR_THREADS / 32) {
			const T *t = tens + kzr * 192 + lane;
			const T nxx = t[0], nxy = t[32], nxz = t[64], nyy = t[96], nyz = t[128], nzz = t[160];
			const int nk = (kzr == 0 || kzr == H) ? 1 : 2;
			const C xx{nxx, nxx}, yy{nyy, nyy}, zz{nzz, nzz};
#pragma unroll
			for (int rr = 0; rr < 2; ++rr) {
				if (rr && !two) break;
#pragma unroll
				for (int q = 0; q < 2; ++q) {
					if (q && nk < 2) break;
					const int kz = q ? PZ - kzr : kzr;
					C *e = sm + ((rr * PZ + kz) * 3) * 32 + lane;
					const C m0 = e[0], m1 = e[32], m2 = e[64];
					const T sxy = rr ? -nxy : nxy, sxz = q ? -nxz : nxz, syz = rr != q ? -nyz : nyz;
					const C xy{sxy, sxy}, xz{sxz, sxz}, yz{syz, syz};
					e[0] = cfma2(xz, m2, cfma2(xy, m1, cscale2(xx, m0)));
					e[32] = cfma2(yz, m2, cfma2(yy, m1, cscale2(xy, m0)));
					e[64] = cfma2(zz, m2, cfma2(yz, m1, cscale2(xz, m0)));
				}
			}
		}
	}
	__syncthreads();
#pragma unroll
	for (int k = 0; k < PZ; ++k) v[k] = mine[k * 96];
	dft_reg<T, PZ, true>(v);
	if (ok) {
#pragma unroll
		for (int z = 0; z < H; ++z)
			if (z < nz) col[z * zstride] = v[dft_pos<PZ>(z)];
	}
}

template <typename T, int PZ>
__global__ void __launch_bounds__(ZR_THREADS, 2) k_z_reg(cplx<T> *__restrict__ S, const T *__restrict__ Nt, int nz,
                                                        int py, int hx, int lx, int qy, int qz, Gate gate)
{
	if (gate.skip()) return;
	z_reg_body<T, PZ>(S, Nt, nz, py, hx, lx, qy, qz, blockIdx.x, blockIdx.y);
}

template <typename T, int PZ>
void fs_z_reg(ConvPlan *p, cudaStream_t st, Gate gate)
{
	const dim3 grid((p->hx + 31) / 32, p->qy);
	k_z_reg<T, PZ><<<grid, ZR_THREADS, zr_smem<T>(PZ), st>>>(
	    (cplx<T> *)p->spec, (const T *)p->tensor, p->nz, p->py, p->hx, p->lx, p->qy, p->qz, gate);
}

// ---- y pass through TMA-staged tiles -------------------------------------------------------------
// Persistent CTAs walk tiles (TB columns of one (component, z) plane).  Each tile's input rows
// (the ny < N/2 data rows padded to N/2 by the TMA unit's zero fill going forward, all N rows
// going back) arrive by cp.async.bulk.tensor in one of two stage buffers while the previous tile is
// transformed; pass 0 reads the stage buffer, the later passes work in a skewed shared-memory
// buffer, and the last pass stores straight to HBM.  Thread 0 issues the loads; a bounded wait that
// runs out sets *err and ends the kernel instead of hanging.
template <int N, int TB, bool INV, class C>
struct YTmaGeom {
	static constexpr int ROWS = INV ? N : N / 2;
	static constexpr int BR = ROWS < 256 ? ROWS : ROWS % 256 == 0 ? 256 : 192;  // rows of a box
	static_assert(ROWS % BR == 0, "a tile is whole boxes");
	static constexpr int NBOX = ROWS / BR;
	static constexpr int E = (int)(sizeof(C) / 8);
	static constexpr uint32_t TILE_BYTES = (uint32_t)(TB * ROWS * sizeof(C));
	static constexpr size_t WORK = ((size_t)SmCols<N, TB, 4>::SIZE * sizeof(C) + 15) / 16 * 16;
	static constexpr size_t SMEM = 2 * (size_t)TILE_BYTES + WORK + 16;
	// the single-instance pass keeps its pass twiddles in shared memory behind the barriers
	static constexpr size_t TW = SMEM;
	static constexpr size_t SMEM_TW = SMEM + (size_t)N * sizeof(C);
};

// Columns per CTA of the single-instance TMA y pass: 32-byte rows, at most 256 threads, so that
// two CTAs (and their barriers) interleave on an SM.
__host__ __device__ constexpr int y_tma_tb(int n, int csize)
{
	int tb = ct_tb(n, csize);
	while (tb * csize > 32 && (tb * (n / ct_radix(n)) > 256 || (!fft_is_pow2(n) && 3L * n * tb * csize > 110 * 1024)))
		tb >>= 1;
	return tb;
}

template <typename T, int N, int TB, bool INV>
__global__ void __launch_bounds__(TB * (N / ct_radix(N)), 2)
    k_y_tma(const __grid_constant__ CUtensorMap tmap, cplx<T> *__restrict__ S, int n_out, int hx, int lx,
            int tiles_x, int ntiles, const cplx<T> *__restrict__ twN, int *err, Gate gate)
{
	if (gate.skip()) return;
	using C = cplx<T>;
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
	C *tws = reinterpret_cast<C *>(smem_tma + G::TW);
	for (int q = tid; q < N; q += blockDim.x) tws[q] = twN[q];
	auto issue = [&](int t, int b) {
		const int tx = t % tiles_x, plane = t / tiles_x;
		C *dst = b ? stage1 : stage0;
		mbar_expect_tx(&bar[b], G::TILE_BYTES);
#pragma unroll
		for (int q = 0; q < G::NBOX; ++q)
			tma_load_3d(dst + q * G::BR * TB, &tmap, tx * TB * G::E, q * G::BR, plane, &bar[b]);
	};
	if (tid == 0) {
		mbar_init(&bar[0], 1);
		mbar_init(&bar[1], 1);
		fence_proxy_async();
	}
	__syncthreads();
	if (tid == 0) {
		if ((int)blockIdx.x < ntiles) issue(blockIdx.x, 0);
		if ((int)(blockIdx.x + gridDim.x) < ntiles) issue(blockIdx.x + gridDim.x, 1);
	}
	uint32_t parity = 0;  // bit b: phase parity expected next on bar[b]
	int k = 0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
		const int b = k & 1;
		const bool late = !mbar_wait(&bar[b], (parity >> b) & 1u);
		if (__syncthreads_or(late)) {
			if (tid == 0) {
				atomicExch(err, 1);
				mbar_drain2(bar, parity, b, t + (int)gridDim.x < ntiles);
			}
			return;
		}
		parity ^= 1u << b;
		const int tx = t % tiles_x, plane = t / tiles_x;
		const int kx = tx * TB + line;
		const bool ok = kx < hx;
		C *base = S + (size_t)plane * N * lx + (ok ? kx : 0);
		const C *sb = b ? stage1 : stage0;
		auto ld = [&](int, int r) -> C { return r < G::ROWS ? sb[r * TB + line] : C{0, 0}; };
		auto st = [&](int, int r, C v) {
			if (ok && r < n_out) base[(size_t)r * lx] = v;
		};
		const int next = t + 2 * (int)gridDim.x;
		auto release = [&]() {
			__syncthreads();  // every thread has read stage buffer b
			if (tid == 0 && next < ntiles) {
				fence_proxy_async();
				issue(next, b);
			}
		};
		if constexpr (INV) cta_fft<T, N, R, TB, INV, SI>(work, tws, line, j0, ld, st, release);
		else cta_fft_h0<T, N, R, TB, SI>(work, tws, line, j0, ld, st, release);  // rows >= N/2 are zero
	}
}

// ---- x passes through TMA-staged tiles -----------------------------------------------------------
// Persistent CTAs walk tiles of LPB complex lines (2 LPB real rows).  A tile's rows arrive by
// cp.async.bulk.tensor in a ring of stage buffers (xbox_n boxes of xbox_w 8-byte elements per row,
// so the staged rows are dense: real rows of nx values going forward, spectrum rows of lx complex
// values going back); pass 0 reads the stage buffer and writes a separate skewed work buffer, after
// which the stage is refilled with the tile STG strides ahead, so that up to STG tiles are loading
// while one is transformed.  Two CTAs share an SM.
template <int N, class C>
struct XTmaGeom {
	static constexpr int R = ct_radix(N);
	static constexpr int LPB = ct_lpb(N, sizeof(C));
	static constexpr int THREADS = LPB * (N / R);
	static constexpr size_t WORK = (size_t)SmRows<N, LPB, 4>::SIZE * sizeof(C);
	static constexpr size_t BUF = (WORK + 127) / 128 * 128;
	static constexpr size_t PER_SM = 228 * 1024;  // shared memory per SM (1 KB of it reserved per CTA)
	// forward stage: 2 LPB real rows of at most N/2 values and their region bytes
	static constexpr size_t SB_F = ((size_t)LPB * N * (sizeof(C) / 2 + 1) + 127) / 128 * 128;
	// forward extras: barriers, the 256-entry Ms table, the pass twiddles
	static constexpr size_t EXTRA_F = 64 + 256 * (sizeof(C) / 2) + (size_t)N * sizeof(C);
	static constexpr int STG_F = 2 * (3 * SB_F + BUF + EXTRA_F + 1024) <= PER_SM ? 3 : 2;
	static constexpr size_t SMEM_F = STG_F * SB_F + BUF + EXTRA_F;
	static constexpr int MINB_F = 2 * (SMEM_F + 1024) <= PER_SM ? 2 : 1;
	// inverse stage: 2 LPB spectrum rows of lx complex values (lx * sizeof(C) * 2 LPB <= BUF,
	// checked at set-up); behind the work buffer the barriers and the pass twiddles
	static constexpr size_t SB_I = BUF;
	static constexpr size_t EXTRA_I = 64 + (size_t)N * sizeof(C);
	static constexpr int STG_I = 2 * (3 * SB_I + BUF + EXTRA_I + 1024) <= PER_SM ? 3 : 2;
	static constexpr size_t SMEM_I = STG_I * SB_I + BUF + EXTRA_I;
	static constexpr int MINB_I = 2 * (SMEM_I + 1024) <= PER_SM ? 2 : 1;
};

// After a bounded wait gave up in a ring of STG stage buffers on the tile t of local index k:
// waits (bounded again) for every load still in flight (tiles t, t + G, ..., t + (STG - 1) G
// that exist), so that no copy lands in shared memory after the CTA has exited.
template <int STG>
__device__ __forceinline__ void mbar_drain_ring(uint64_t *bar, uint32_t parity, int k, int t, int G, int ntiles)
{
	for (int i = 0; i < STG; ++i) {
		const int s = (k + i) % STG;
		if (t + i * G < ntiles) mbar_wait(&bar[s], (parity >> s) & 1u);
	}
}

// Forward: with SCALE the tile's region bytes (rows r % (ny nz), contiguous within a tile) ride
// along in the same stage behind the real rows, and the 256-entry Ms table sits in shared memory,
// so that pass 0 reads nothing but shared memory.
template <typename T, int N, bool SCALE>
__global__ void __launch_bounds__(XTmaGeom<N, cplx<T>>::THREADS, XTmaGeom<N, cplx<T>>::MINB_F)
    k_x_fwd_tma(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap rmap,
                const T *__restrict__ ms_tab, cplx<T> *__restrict__ S, int nx, int ny, int nz, int py, int hx,
                int lx, int ntiles, const cplx<T> *__restrict__ twN, int *err, Gate gate)
{
	if (gate.skip()) return;
	using C = cplx<T>;
	using G = XTmaGeom<N, C>;
	constexpr int LPB = G::LPB, TPL = N / G::R, STG = G::STG_F;
	using SI = SmRows<N, LPB, 4>;
	extern __shared__ __align__(128) unsigned char smem_tma[];
	C *work = reinterpret_cast<C *>(smem_tma + STG * G::SB_F);
	unsigned char *extra = smem_tma + STG * G::SB_F + G::BUF;
	uint64_t *bar = reinterpret_cast<uint64_t *>(extra);
	T *msr = reinterpret_cast<T *>(extra + 64);
	C *tws = reinterpret_cast<C *>(extra + 64 + 256 * sizeof(T));
	const int tid = threadIdx.x;
	const int line = tid / TPL, j0 = tid % TPL;
	const int rows = 3 * ny * nz, nyz = ny * nz;
	const int G_ = (int)gridDim.x;
	const uint32_t row_bytes = (uint32_t)(2 * LPB * (size_t)nx * sizeof(T));
	const uint32_t tile_bytes = row_bytes + (SCALE ? (uint32_t)(2 * LPB * nx) : 0u);
	auto issue = [&](int t, int s) {
		unsigned char *dst = smem_tma + s * G::SB_F;
		mbar_expect_tx(&bar[s], tile_bytes);
		tma_load_3d(dst, &tmap, 0, 0, t * 2 * LPB, &bar[s]);
		if (SCALE) tma_load_2d(dst + row_bytes, &rmap, 0, (t * 2 * LPB) % nyz, &bar[s]);
	};
	if (SCALE)
		for (int r = tid; r < 256; r += blockDim.x) msr[r] = ms_tab[r];
	for (int q = tid; q < N; q += blockDim.x) tws[q] = twN[q];
	if (tid == 0) {
		for (int s = 0; s < STG; ++s) mbar_init(&bar[s], 1);
		fence_proxy_async();
	}
	__syncthreads();
	if (tid == 0)
		for (int s = 0; s < STG; ++s)
			if ((int)blockIdx.x + s * G_ < ntiles) issue(blockIdx.x + s * G_, s);
	uint32_t parity = 0;  // bit s: phase parity expected next on bar[s]
	int k = 0, s = 0;
	for (int t = blockIdx.x; t < ntiles; t += G_, ++k, s = s + 1 == STG ? 0 : s + 1) {
		// (this barrier also orders the previous tile's reads of the work buffer before pass 0)
		const bool late = !mbar_wait(&bar[s], (parity >> s) & 1u);
		if (__syncthreads_or(late)) {
			if (tid == 0) {
				atomicExch(err, 1);
				mbar_drain_ring<STG>(bar, parity, k, t, G_, ntiles);
			}
			return;
		}
		parity ^= 1u << s;
		const unsigned char *stage = smem_tma + s * G::SB_F;
		const T *rowa = reinterpret_cast<const T *>(stage) + (size_t)(2 * line) * nx;
		const T *rowb = rowa + nx;
		const uint8_t *rga = stage + row_bytes + (size_t)(2 * line) * nx;
		const uint8_t *rgb = rga + nx;
		const int ra = 2 * (t * LPB + line), rb = ra + 1;
		const bool va = ra < rows, vb = rb < rows;
		// loads first, selects afterwards (as x_fwd_ct_body); x < N/2 stays inside the stage buffer, and
		// whatever byte lies there is an index of the 256-entry table
		auto ld = [&](int, int x) -> C {
			T a = rowa[x], bb = rowb[x];
			if (SCALE) {
				a *= msr[rga[x]];
				bb *= msr[rgb[x]];
			}
			return C{x < nx && va ? a : T(0), x < nx && vb ? bb : T(0)};
		};
		auto st = [&](int l, int kk, C v) { work[SI::at(l, kk)] = v; };
		const int next = t + STG * G_;
		auto release = [&]() {
			__syncthreads();  // every thread has read stage s
			if (tid == 0 && next < ntiles) {
				fence_proxy_async();
				issue(next, s);
			}
		};
		cta_fft_h0<T, N, G::R, LPB, SI>(work, tws, line, j0, ld, st, release);  // x >= nx, N/2 <= x: zero
		__syncthreads();
		size_t sa, sb;
		spec_rows(ra, va, vb, ny, py, sa, sb);
		C *Sa = S + sa * lx, *Sb = S + sb * lx;
		const T h = T(0.5);
		auto out = [&](int kk) {
			const C zk = work[SI::at(line, kk)], zn = work[SI::at(line, kk == 0 ? 0 : N - kk)];
			if (va) Sa[kk] = C{h * (zk.x + zn.x), h * (zk.y - zn.y)};
			if (vb) Sb[kk] = C{h * (zk.y + zn.y), h * (zn.x - zk.x)};
		};
#pragma unroll
		for (int i = 0; i < G::R / 2; ++i) out(j0 + i * TPL);  // k < N/2, then the last stored frequency
		if (j0 == 0) out(N / 2);
	}
}

// x inverse: the 2 LPB spectrum rows of a tile lie in one (component, z) plane (ny a multiple of
// 2 LPB); the 4-D tensor map addresses them as (box element, box, y, plane).
template <typename T, int N>
__global__ void __launch_bounds__(XTmaGeom<N, cplx<T>>::THREADS, XTmaGeom<N, cplx<T>>::MINB_I)
    k_x_inv_tma(const __grid_constant__ CUtensorMap tmap, T *__restrict__ H, int nx, int ny, int hx, int lx,
                int ntiles, const cplx<T> *__restrict__ twN, int *err, Gate gate)
{
	if (gate.skip()) return;
	using C = cplx<T>;
	using G = XTmaGeom<N, C>;
	constexpr int LPB = G::LPB, TPL = N / G::R, STG = G::STG_I;
	using SI = SmRows<N, LPB, 4>;
	extern __shared__ __align__(128) unsigned char smem_tma[];
	C *work = reinterpret_cast<C *>(smem_tma + STG * G::SB_I);
	uint64_t *bar = reinterpret_cast<uint64_t *>(smem_tma + STG * G::SB_I + G::BUF);
	C *tws = reinterpret_cast<C *>(smem_tma + STG * G::SB_I + G::BUF + 64);
	const int tid = threadIdx.x;
	const int line = tid / TPL, j0 = tid % TPL;
	const int G_ = (int)gridDim.x;
	const uint32_t tile_bytes = (uint32_t)(2 * LPB * (size_t)lx * sizeof(C));
	auto issue = [&](int t, int s) {
		const int row0 = t * 2 * LPB;
		mbar_expect_tx(&bar[s], tile_bytes);
		tma_load_4d(smem_tma + s * G::SB_I, &tmap, 0, 0, row0 % ny, row0 / ny, &bar[s]);
	};
	for (int q = tid; q < N; q += blockDim.x) tws[q] = twN[q];
	if (tid == 0) {
		for (int s = 0; s < STG; ++s) mbar_init(&bar[s], 1);
		fence_proxy_async();
	}
	__syncthreads();
	if (tid == 0)
		for (int s = 0; s < STG; ++s)
			if ((int)blockIdx.x + s * G_ < ntiles) issue(blockIdx.x + s * G_, s);
	uint32_t parity = 0;
	int k = 0, s = 0;
	for (int t = blockIdx.x; t < ntiles; t += G_, ++k, s = s + 1 == STG ? 0 : s + 1) {
		// (this barrier also orders the previous tile's last-pass reads of the work buffer before
		// this tile's pass 0 writes)
		const bool late = !mbar_wait(&bar[s], (parity >> s) & 1u);
		if (__syncthreads_or(late)) {
			if (tid == 0) {
				atomicExch(err, 1);
				mbar_drain_ring<STG>(bar, parity, k, t, G_, ntiles);
			}
			return;
		}
		parity ^= 1u << s;
		const C *Sa = reinterpret_cast<const C *>(smem_tma + s * G::SB_I) + (size_t)(2 * line) * lx;
		const C *Sb = Sa + lx;
		const size_t ra = 2 * ((size_t)t * LPB + line);
		T *Ha = H + ra * nx, *Hb = Ha + nx;
		auto ld = [&](int, int f) -> C {
			const bool mirror = 2 * f > N;
			const int ff = mirror ? N - f : f;
			C A = Sa[ff], B = Sb[ff];
			if (ff == 0 || 2 * ff == N) { A.y = 0; B.y = 0; }
			if (mirror) { A.y = -A.y; B.y = -B.y; }
			return C{A.x - B.y, A.y + B.x};
		};
		auto st = [&](int, int x, C v) {
			if (x < nx) {
				Ha[x] = v.x;
				Hb[x] = v.y;
			}
		};
		const int next = t + STG * G_;
		auto release = [&]() {
			__syncthreads();  // every thread has read stage s
			if (tid == 0 && next < ntiles) {
				fence_proxy_async();
				issue(next, s);
			}
		};
		cta_fft<T, N, G::R, LPB, true, SI>(work, tws, line, j0, ld, st, release);
	}
}

// ---- fast-path geometry and dispatch ---------------------------------------------------------------


// Lengths with compile-time passes: powers of two and three times powers of two.
template <typename T>
bool fs_len_ok(int n)
{
	if (fft_is_pow2(n)) return n >= 4 && n <= 2048;
	return n % 3 == 0 && fft_is_pow2(n / 3) && n >= 12 && n <= 1536;
}

// z lengths with compile-time passes: whole columns in registers (zero-padded axes), or through
// shared memory (powers of two, padded or not).
template <typename T>
bool fz_reg_ok(int pz, int nz)
{
	if (2 * nz > pz) return false;
	if (fft_is_pow2(pz)) return pz >= 2 && pz <= (sizeof(T) == 4 ? 32 : 16);
	return pz == 6 || pz == 12 || pz == 24;
}
template <typename T>
bool fz_len_ok(int pz, int nz)
{
	return fz_reg_ok<T>(pz, nz) || (fft_is_pow2(pz) && pz >= 2 && pz <= 64);
}

// FFT length of one axis of n cells whose tensor layout has length e.  With e >= 2n - 1 the axis is
// zero padded and any length >= 2n - 1 gives the same convolution, so it takes the shortest length
// with compile-time passes (2n or more, whose upper half of inputs is zero) instead of the
// mixed-radix passes at e; otherwise the convolution is circular and e is its length.  The
// run-time radices of the mixed-radix passes cost an integer division per index and one barrier
// per small radix: 200x150x6 cells, FP32, took 27 + 52 + 29 us in the y, z and y passes at 300 and 12
// points and 24 + 27 us in the x passes at 400; at 384, 12 and 512 points the compile-time passes
// take 15 + 13 + 15 and 15 + 11 us (event-timed, about 6 us of each is the timing).  A length with a large
// prime factor gained most (796 points: 980 us a pass, against 15 at 1024).
template <typename T>
int fit_length(int n, int e, bool z)
{
	if (n < 2 || e < 2 * n - 1) return e;
	int best = 0;
	for (int base : {1, 3})
		for (int len = base == 3 ? 6 : 2; len <= 2048; len *= 2)
			if (len >= 2 * n && (z ? fz_len_ok<T>(len, n) : fs_len_ok<T>(len)) && (best == 0 || len < best)) best = len;
	return best ? best : e;
}

// Relative cost of one axis's transforms per point: with compile-time passes, or in the mixed-radix ones, where
// a pass of a radix up to 8 costs about the same whatever the radix and a larger prime factor in proportion to it.
// (Fitted to evaluations of 60 boxes of 33 to 128 layers, mixed-radix and compile-time along x and y: 5% rms
// in FP64, 11% in FP32.)
inline double axis_cost(int len, bool ct)
{
	if (ct) return 0.35;
	double c = 0;
	const FftRadices f = fft_factor(len);
	for (int p = 0; p < f.count; ++p) c += f.r[p] <= 8 ? 1.0 : 0.42 * f.r[p];
	return c;
}

// FFT lengths of a box of n cells whose tensor has layout e.  An axis takes fit_length, with two exceptions for
// boxes whose z passes are of the mixed-radix form (more than 32 layers, or a periodic axis of no such length), which
// pay for every column that longer x and y lengths add:
// - x and y take those lengths only unless the whole gets an eighth cheaper without: 140x140x64 cells, FP32, take
//   598 us at 280x280x128 points and 733 at 384x384x128; 260x260x40 1977 at 520x520x80 and 1650 at 768x768x80;
// - a zero-padded z axis whose length has a prime factor above 7 takes a near length that has none: 100x100x34 cells,
//   FP32, 363 us at 200x200x68 points, 435 at 256x256x68, 201 at 256x256x80.
template <typename T>
void choose_lengths(const int (&n)[3], const int (&e)[3], int (&p)[3])
{
	for (int a = 0; a < 3; ++a) p[a] = fit_length<T>(n[a], e[a], a == 2);
	if (p[2] == 1 || fz_len_ok<T>(p[2], n[2])) return;
	if (n[2] > 1 && e[2] >= 2 * n[2] - 1) {
		// (Multiples of 8 with a factor 5 or 7: 34 and 37 layers take 80 points, 65 take 160.  Lengths of 2s and 3s
		// alone, like those of x and y, repeat their constants' rounding along every axis: FP32 errors of 35x35x129 cells
		// were 1.4 times those at 260 points with 288, 0.8 with 280.)
		const FftRadices own = fft_factor(e[2]);
		double least = axis_cost(e[2], false) * e[2];
		if (own.r[own.count - 1] > 7)
			for (int len = (2 * n[2] + 6) / 8 * 8; len <= e[2] + e[2] / 4; len += 8) {
				const FftRadices f = fft_factor(len);
				const double c = axis_cost(len, false) * len;
				if (f.r[f.count - 1] <= 7 && (len % 5 == 0 || len % 7 == 0) && c < least && 7 * sizeof(cplx<T>) * len <= 227 * 1024) {
					least = c;
					p[2] = len;
				}
			}
	}
	const double rows_z = (double)n[2] / p[2], rows_yz = rows_z * n[1] / e[1];  // lines that carry data
	auto cost = [&](int px, int py) {
		return (double)px * py * (rows_yz * axis_cost(px, fs_len_ok<T>(px)) + rows_z * axis_cost(py, fs_len_ok<T>(py)) +
		                          axis_cost(p[2], false));
	};
	const int fx = p[0], fy = p[1];
	double least = 0.87 * cost(fx, fy);
	for (int own = 1; own < 4; ++own) {  // bit a: axis a keeps the tensor's length
		const int px = own & 1 ? e[0] : fx, py = own & 2 ? e[1] : fy;
		if (cost(px, py) < least) {
			least = cost(px, py);
			p[0] = px;
			p[1] = py;
		}
	}
}

template <typename T, int N>
mm_status fs_setup_len()
{
	using C = cplx<T>;
	constexpr int TB = ct_tb(N, sizeof(C)), LPB = ct_lpb(N, sizeof(C)), T2 = y2d_tb(N, sizeof(C));
	const size_t sx = (size_t)SmRows<N, LPB>::SIZE * sizeof(C), sy = (size_t)SmCols<N, TB>::SIZE * sizeof(C);
	MM_TRY(set_smem<T>((const void *)k_y2d_ct<T, N, T2>, (size_t)SmCols<N, 3 * T2>::SIZE * sizeof(C)));
	MM_TRY(set_smem<T>((const void *)k_y2d_ct<T, N, 1>, (size_t)SmCols<N, 3>::SIZE * sizeof(C)));
	MM_TRY(set_smem<T>((const void *)k_x_fwd_ct<T, N, LPB, false, false>, sx));
	MM_TRY(set_smem<T>((const void *)k_x_fwd_ct<T, N, LPB, true, false>, sx));
	MM_TRY(set_smem<T>((const void *)k_x_fwd_ct<T, N, LPB, false, true>, sx));
	MM_TRY(set_smem<T>((const void *)k_x_fwd_ct<T, N, LPB, true, true>, sx));
	MM_TRY(set_smem<T>((const void *)k_x_inv_ct<T, N, LPB>, sx));
	MM_TRY(set_smem<T>((const void *)k_y_ct<T, N, TB, false>, sy));
	MM_TRY(set_smem<T>((const void *)k_y_ct<T, N, TB, true>, sy));
	return MM_OK;
}

// Whether the usual tiles of the x or y passes leave SMs without work: then narrow tiles spread the
// lines over the device (and the staged passes, whose CTAs walk several tiles each, are not used).
template <typename T, int N>
bool fs_narrow_x(const ConvPlan *p)
{
	constexpr int LPB = ct_lpb(N, sizeof(cplx<T>));
	return ((3 * p->ny * p->nz + 1) / 2 + LPB - 1) / LPB < num_sms();
}
template <typename T, int N>
bool fs_narrow_y(const ConvPlan *p)
{
	constexpr int TB = ct_tb(N, sizeof(cplx<T>));
	return (p->hx + TB - 1) / TB * 3 * p->nz < num_sms();
}

// TMA-staged y passes: tensor maps over the spectrum, shared-memory size, persistent grid size.
// Used when the inverse pass's stage buffers fit in shared memory and the forward input is at
// most half the padded length (ny <= py/2, the zero padding the first pass relies on).
template <typename T, int N>
mm_status fs_setup_y_tma(ConvPlan *p)
{
	using C = cplx<T>;
	constexpr int TB = y_tma_tb(N, sizeof(C)), THREADS = TB * (N / ct_radix(N));
	using GF = YTmaGeom<N, TB, false, C>;
	using GI = YTmaGeom<N, TB, true, C>;
	p->tma_y = false;
	if (fs_narrow_y<T, N>(p)) return MM_OK;
	if (GI::SMEM_TW > 227 * 1024 || 2 * p->ny > p->py || TB * sizeof(C) < 16) return MM_OK;
	constexpr int E = GF::E;
	const uint64_t d0 = (uint64_t)p->lx * E, rowb = (uint64_t)p->lx * sizeof(C), planeb = rowb * p->py;
	MM_TRY(tma_encode_3d(&p->tm_yf, p->spec, d0, (uint64_t)p->ny, 3ull * p->nz, rowb, planeb, TB * E, GF::BR, 1));
	MM_TRY(tma_encode_3d(&p->tm_yi, p->spec, d0, (uint64_t)p->py, 3ull * p->nz, rowb, planeb, TB * E, GI::BR, 1));
	MM_TRY(set_smem<T>((const void *)k_y_tma<T, N, TB, false>, GF::SMEM_TW));
	MM_TRY(set_smem<T>((const void *)k_y_tma<T, N, TB, true>, GI::SMEM_TW));
	int bf = 0, bi = 0;
	MM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bf, k_y_tma<T, N, TB, false>, THREADS, GF::SMEM_TW));
	MM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bi, k_y_tma<T, N, TB, true>, THREADS, GI::SMEM_TW));
	if (bf < 1 || bi < 1) return MM_OK;
	p->grid_yf = bf * num_sms();
	p->grid_yi = bi * num_sms();
	if (!p->err) {
		MM_CUDA(cudaMalloc(&p->err, sizeof(int)));
		MM_CUDA(cudaMemset(p->err, 0, sizeof(int)));
	}
	p->tma_y = true;
	return MM_OK;
}

template <typename T, int N, bool INV>
void fs_y_tma(ConvPlan *p, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	constexpr int TB = y_tma_tb(N, sizeof(C)), THREADS = TB * (N / ct_radix(N));
	using G = YTmaGeom<N, TB, INV, C>;
	const int tiles_x = (p->hx + TB - 1) / TB, ntiles = tiles_x * 3 * p->nz;
	const int grid = std::min(ntiles, INV ? p->grid_yi : p->grid_yf);
	k_y_tma<T, N, TB, INV><<<grid, THREADS, G::SMEM_TW, st>>>(INV ? p->tm_yi : p->tm_yf, (C *)p->spec,
	                                                       INV ? p->ny : N, p->hx, p->lx, tiles_x, ntiles,
	                                                       tw_of((const C *)p->tw_y, N, ct_radix(N)), p->err, gate);
}

// TMA-staged x passes.  The inverse pass's tensor map (over the spectrum) is fixed; the forward
// pass reads the state the caller passes, so its map is encoded per input pointer (a small cache
// keeps the solver's few state buffers).
template <typename T, int N>
mm_status fs_setup_x_tma(ConvPlan *p)
{
	using C = cplx<T>;
	using G = XTmaGeom<N, C>;
	constexpr int LPB = G::LPB;
	p->tma_xf = p->tma_xi = false;
	if (fs_narrow_x<T, N>(p)) return MM_OK;
	// the forward pass's half-zero first butterflies need nx <= N/2 (non-periodic zero padding)
	if (G::SMEM_F > 227 * 1024 || G::SMEM_I > 227 * 1024 || N < 64 || 2 * p->nx > N) return MM_OK;
	int occ = 0;
	// forward: dense real rows split into boxes of even width
	const size_t wf = (size_t)p->nx * sizeof(T) / 8;
	const size_t nbf = (wf + 255) / 256;
	if ((p->nx * sizeof(T)) % 16 == 0 && wf % (2 * nbf) == 0 && 2 * LPB * p->nx * sizeof(T) <= G::SB_F) {
		// region bytes ride behind the rows when a tile's rows are contiguous in the region map
		p->tma_xf_scale = p->nx % 16 == 0 && (p->ny * p->nz) % (2 * LPB) == 0 && p->nx / 8 <= 256 &&
		                  2 * LPB * p->nx * (sizeof(T) + 1) <= G::SB_F;
		MM_TRY(set_smem<T>((const void *)k_x_fwd_tma<T, N, false>, G::SMEM_F));
		MM_TRY(set_smem<T>((const void *)k_x_fwd_tma<T, N, true>, G::SMEM_F));
		MM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_x_fwd_tma<T, N, true>, G::THREADS, G::SMEM_F));
		if (occ >= 1) {
			p->grid_xf = occ * num_sms();
			p->xf_box_n = (int)nbf;
			p->xf_box_w = (int)(wf / nbf);
			p->tma_xf = true;
		}
	}
	// inverse: spectrum rows of a tile within one plane
	if (p->ny % (2 * LPB) == 0 && (size_t)2 * LPB * p->lx * sizeof(C) <= G::SB_I) {
		const uint64_t rowb = (uint64_t)p->lx * sizeof(C);
		const uint64_t dims[4] = {(uint64_t)p->xbox_w, (uint64_t)p->xbox_n, (uint64_t)p->ny, 3ull * p->nz};
		const uint64_t strides[3] = {(uint64_t)p->xbox_w * 8, rowb, rowb * p->py};
		const uint32_t box[4] = {(uint32_t)p->xbox_w, (uint32_t)p->xbox_n, (uint32_t)(2 * LPB), 1};
		MM_TRY(tma_encode(&p->tm_xi, p->spec, 4, dims, strides, box));
		MM_TRY(set_smem<T>((const void *)k_x_inv_tma<T, N>, G::SMEM_I));
		MM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_x_inv_tma<T, N>, G::THREADS, G::SMEM_I));
		if (occ >= 1) {
			p->grid_xi = occ * num_sms();
			p->tma_xi = true;
		}
	}
	if ((p->tma_xf || p->tma_xi) && !p->err) {
		MM_CUDA(cudaMalloc(&p->err, sizeof(int)));
		MM_CUDA(cudaMemset(p->err, 0, sizeof(int)));
	}
	return MM_OK;
}

// Tensor map of the forward x pass over the real rows at M (NULL when M is not 16-byte aligned).
// Tensor map of the region bytes of the forward x pass (NULL when not usable for `reg`).
const CUtensorMap *x_reg_map(ConvPlan *p, const uint8_t *reg, int lpb)
{
	if (!p->tma_xf_scale || !reg || (reinterpret_cast<uintptr_t>(reg) & 15)) return nullptr;
	if (p->xr_ptr == reg) return &p->xr_map;
	const uint64_t dims[2] = {(uint64_t)p->nx / 8, (uint64_t)p->ny * p->nz};
	const uint64_t strides[1] = {(uint64_t)p->nx};
	const uint32_t box[2] = {(uint32_t)(p->nx / 8), (uint32_t)(2 * lpb)};
	if (tma_encode(&p->xr_map, reg, 2, dims, strides, box) != MM_OK) {
		clear_error();
		return nullptr;
	}
	p->xr_ptr = reg;
	return &p->xr_map;
}

template <typename T>
const CUtensorMap *x_fwd_map(ConvPlan *p, const T *M, int lpb)
{
	if (reinterpret_cast<uintptr_t>(M) & 15) return nullptr;
	for (int i = 0; i < ConvPlan::XF_CACHE; ++i)
		if (p->xf_ptr[i] == M) return &p->xf_map[i];
	const int slot = p->xf_next;
	const uint64_t rows = 3ull * p->ny * p->nz;
	const uint64_t dims[3] = {(uint64_t)p->xf_box_w, (uint64_t)p->xf_box_n, rows};
	const uint64_t strides[2] = {(uint64_t)p->xf_box_w * 8, (uint64_t)p->nx * sizeof(T)};
	const uint32_t box[3] = {(uint32_t)p->xf_box_w, (uint32_t)p->xf_box_n, (uint32_t)(2 * lpb)};
	if (tma_encode(&p->xf_map[slot], M, 3, dims, strides, box) != MM_OK) {
		clear_error();
		return nullptr;
	}
	p->xf_ptr[slot] = M;
	p->xf_next = (slot + 1) % ConvPlan::XF_CACHE;
	return &p->xf_map[slot];
}

template <typename T, int N>
bool fs_x_fwd_tma(ConvPlan *p, const T *M, const uint8_t *reg, const T *ms_tab, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	using G = XTmaGeom<N, C>;
	const CUtensorMap *map = x_fwd_map<T>(p, M, G::LPB);
	if (!map) return false;
	const CUtensorMap *rmap = map;
	if (ms_tab) {
		// a missing region map means region 0 everywhere: the staged kernel needs real bytes
		rmap = reg ? x_reg_map(p, reg, G::LPB) : nullptr;
		if (!rmap) return false;
	}
	const int lines = (3 * p->ny * p->nz + 1) / 2;
	const int ntiles = (lines + G::LPB - 1) / G::LPB;
	const int grid = std::min(ntiles, p->grid_xf);
	if (ms_tab)
		k_x_fwd_tma<T, N, true><<<grid, G::THREADS, G::SMEM_F, st>>>(*map, *rmap, ms_tab, (C *)p->spec, p->nx, p->ny,
		                                                            p->nz, p->py, p->hx, p->lx, ntiles,
		                                                            tw_of((const C *)p->tw_x, N, ct_radix(N)), p->err, gate);
	else
		k_x_fwd_tma<T, N, false><<<grid, G::THREADS, G::SMEM_F, st>>>(*map, *rmap, ms_tab, (C *)p->spec, p->nx, p->ny,
		                                                             p->nz, p->py, p->hx, p->lx, ntiles,
		                                                             tw_of((const C *)p->tw_x, N, ct_radix(N)), p->err, gate);
	return true;
}

template <typename T, int N>
void fs_x_inv_tma(ConvPlan *p, T *H, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	using G = XTmaGeom<N, C>;
	const int ntiles = 3 * p->ny * p->nz / (2 * G::LPB);
	const int grid = std::min(ntiles, p->grid_xi);
	k_x_inv_tma<T, N><<<grid, G::THREADS, G::SMEM_I, st>>>(p->tm_xi, H, p->nx, p->ny, p->hx, p->lx, ntiles,
	                                                     tw_of((const C *)p->tw_x, N, ct_radix(N)), p->err, gate);
}

template <typename T, int N>
void fs_x_fwd(ConvPlan *p, const T *M, const uint8_t *reg, const T *ms_tab, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	constexpr int TPL = N / ct_radix(N);
	const int lines = (3 * p->ny * p->nz + 1) / 2;
	auto go = [&](auto lpb, auto half) {
		constexpr int LPB = decltype(lpb)::value;
		constexpr bool H0 = decltype(half)::value;
		const dim3 grid((lines + LPB - 1) / LPB), block(LPB * TPL);
		const size_t smem = (size_t)SmRows<N, LPB>::SIZE * sizeof(C);
		if (ms_tab)
			k_x_fwd_ct<T, N, LPB, true, H0><<<grid, block, smem, st>>>(M, reg, ms_tab, (C *)p->spec, p->nx, p->ny, p->nz,
		                                                       p->py, p->hx, p->lx, tw_of((const C *)p->tw_x, N, ct_radix(N)), gate);
		else
			k_x_fwd_ct<T, N, LPB, false, H0><<<grid, block, smem, st>>>(M, reg, ms_tab, (C *)p->spec, p->nx, p->ny, p->nz,
			                                                        p->py, p->hx, p->lx, tw_of((const C *)p->tw_x, N, ct_radix(N)), gate);
	};
	auto pick = [&](auto half) {
		if (fs_narrow_x<T, N>(p)) go(std::integral_constant<int, ct_lpb_narrow(N)>(), half);
		else go(std::integral_constant<int, ct_lpb(N, sizeof(C))>(), half);
	};
	if (2 * p->nx <= N) pick(std::true_type());
	else pick(std::false_type());
}

template <typename T, int N>
void fs_x_inv(ConvPlan *p, T *H, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	constexpr int TPL = N / ct_radix(N);
	const int lines = (3 * p->ny * p->nz + 1) / 2;
	auto go = [&](auto lpb) {
		constexpr int LPB = decltype(lpb)::value;
		const dim3 grid((lines + LPB - 1) / LPB), block(LPB * TPL);
		k_x_inv_ct<T, N, LPB><<<grid, block, (size_t)SmRows<N, LPB>::SIZE * sizeof(C), st>>>(
		    (const C *)p->spec, H, p->nx, p->ny, p->nz, p->py, p->hx, p->lx, tw_of((const C *)p->tw_x, N, ct_radix(N)), gate);
	};
	if (fs_narrow_x<T, N>(p)) go(std::integral_constant<int, ct_lpb_narrow(N)>());
	else go(std::integral_constant<int, ct_lpb(N, sizeof(C))>());
}

template <typename T, int N, bool INV>
void fs_y(ConvPlan *p, cudaStream_t st, Gate gate)
{
	using C = cplx<T>;
	constexpr int TPL = N / ct_radix(N);
	auto go = [&](auto tb) {
		constexpr int TB = decltype(tb)::value;
		const dim3 grid((p->hx + TB - 1) / TB, p->nz, 3), block(TB * TPL);
		k_y_ct<T, N, TB, INV><<<grid, block, (size_t)SmCols<N, TB>::SIZE * sizeof(C), st>>>(
		    (C *)p->spec, INV ? N : p->ny, INV ? p->ny : N, p->nz, p->hx, p->lx,
		    tw_of((const C *)p->tw_y, N, ct_radix(N)), gate);
	};
	if (fs_narrow_y<T, N>(p)) go(std::integral_constant<int, ct_tb_narrow(N, sizeof(C))>());
	else go(std::integral_constant<int, ct_tb(N, sizeof(C))>());
}

// The fused y pass of a 2-D problem: tiles of several columns where they fill the device, else single
// columns.
template <typename T, int N>
void fs_y2d(ConvPlan *p, cudaStream_t st)
{
	using C = cplx<T>;
	constexpr int TPL = N / ct_radix(N), WIDE = y2d_tb(N, sizeof(C));
	auto go = [&](auto tb) {
		constexpr int TB = decltype(tb)::value;
		k_y2d_ct<T, N, TB><<<(p->hx + TB - 1) / TB, 3 * TB * TPL, (size_t)SmCols<N, 3 * TB>::SIZE * sizeof(C), st>>>(
		    (C *)p->spec, (const T *)p->tensor, p->ny, p->hx, p->lx, p->qy, tw_of((const C *)p->tw_y, N, ct_radix(N)));
	};
	if (p->hx >= WIDE * num_sms()) go(std::integral_constant<int, WIDE>());
	else go(std::integral_constant<int, 1>());
}

constexpr int CT_ZTB = 32;

template <typename T, int PZ>
void fs_z(ConvPlan *p, cudaStream_t st)
{
	using C = cplx<T>;
	const dim3 grid((p->hx + CT_ZTB - 1) / CT_ZTB, p->py), block(3 * CT_ZTB * (PZ / ct_radix8(PZ)));
	k_z_ct<T, PZ, CT_ZTB><<<grid, block, (size_t)SmCols<PZ, 3 * CT_ZTB>::SIZE * sizeof(C), st>>>(
	    (C *)p->spec, (const T *)p->tensor, p->nz, p->py, p->hx, p->lx, p->qy, p->qz, tw_of((const C *)p->tw_z, PZ, ct_radix8(PZ)));
}

#define MM_FS_SWITCH(n, CALL)                                                                    \
	switch (n) {                                                                                 \
	case 4: CALL(4); break;                                                                      \
	case 8: CALL(8); break;                                                                      \
	case 16: CALL(16); break;                                                                    \
	case 32: CALL(32); break;                                                                    \
	case 64: CALL(64); break;                                                                    \
	case 128: CALL(128); break;                                                                  \
	case 256: CALL(256); break;                                                                  \
	case 512: CALL(512); break;                                                                  \
	case 1024: CALL(1024); break;                                                                \
	case 2048: if constexpr (sizeof(T) == 4) { CALL(2048); } break;                               \
	default: break;                                                                              \
	}

// The lengths of fs_len_ok: the single-instance passes (grouped members have power-of-two lengths).
#define MM_FS_SWITCH3(n, CALL)                                                                   \
	switch (n) {                                                                                 \
	case 12: CALL(12); break;                                                                    \
	case 24: CALL(24); break;                                                                    \
	case 48: CALL(48); break;                                                                    \
	case 96: CALL(96); break;                                                                    \
	case 192: CALL(192); break;                                                                  \
	case 384: CALL(384); break;                                                                  \
	case 768: CALL(768); break;                                                                  \
	case 1536: CALL(1536); break;                                                                \
	case 2048: CALL(2048); break;                                                                \
	default: MM_FS_SWITCH(n, CALL)                                                               \
	}

template <typename T>
mm_status fs_setup(ConvPlan *p)
{
	// (the staged and register passes skip the zero upper half of a forward transform; an axis without
	// zero padding, a periodic one of padded length n, takes those that load every input)
	p->fast_x = fs_len_ok<T>(p->px);
	p->fast_y = fs_len_ok<T>(p->py);
	p->fast_z = !p->is2d && fz_len_ok<T>(p->pz, p->nz);
	mm_status r = MM_OK;
#define MM_SETUP(N) r = fs_setup_len<T, N>()
	if (p->fast_x) { MM_FS_SWITCH3(p->px, MM_SETUP); MM_TRY(r); }
	if (p->fast_y) { MM_FS_SWITCH3(p->py, MM_SETUP); MM_TRY(r); }
#undef MM_SETUP
#define MM_XTSETUP(N) r = fs_setup_x_tma<T, N>(p)
	if (p->fast_x) { MM_FS_SWITCH3(p->px, MM_XTSETUP); MM_TRY(r); }
#undef MM_XTSETUP
#define MM_YTSETUP(N) r = fs_setup_y_tma<T, N>(p)
	if (p->fast_y && !p->is2d) { MM_FS_SWITCH3(p->py, MM_YTSETUP); MM_TRY(r); }
#undef MM_YTSETUP
	p->reg_z = p->fast_z && fz_reg_ok<T>(p->pz, p->nz);
	if (p->reg_z) {
		const size_t sz = zr_smem<T>(p->pz);
		switch (p->pz) {
		case 2: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 2>, sz)); break;
		case 6: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 6>, sz)); break;
		case 12: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 12>, sz)); break;
		case 24: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 24>, sz)); break;
		case 4: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 4>, sz)); break;
		case 8: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 8>, sz)); break;
		case 16: MM_TRY(set_smem<T>((const void *)k_z_reg<T, 16>, sz)); break;
		case 32: if constexpr (sizeof(T) == 4) { MM_TRY(set_smem<T>((const void *)k_z_reg<T, 32>, sz)); } break;
		}
	} else if (p->fast_z) {
		const size_t sz = (size_t)(p->pz * 3 * CT_ZTB + (p->pz * 3 * CT_ZTB >> 5) + 1) * sizeof(cplx<T>);
		switch (p->pz) {
		case 2: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 2, CT_ZTB>, sz)); break;
		case 4: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 4, CT_ZTB>, sz)); break;
		case 8: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 8, CT_ZTB>, sz)); break;
		case 16: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 16, CT_ZTB>, sz)); break;
		case 32: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 32, CT_ZTB>, sz)); break;
		case 64: MM_TRY(set_smem<T>((const void *)k_z_ct<T, 64, CT_ZTB>, sz)); break;
		}
	}
	return MM_OK;
}

template <typename T>
__global__ void __launch_bounds__(NT) k_round(const double *__restrict__ in, T *__restrict__ out, size_t n)
{
	for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = (T)in[i];
}

// The three passes over one part of the tensor, octant [m2][m1][m0][6] -> out (OUT = T, or double to add up).
template <typename OUT>
mm_status spectrum_passes(const ConvPlan *p, const double *octant, int part, const int (&m)[3], double *A, double *B,
                          const double2 *const (&tw)[3], OUT *out, cudaStream_t st)
{
	const int p3[3] = {p->px, p->py, p->pz};
	const FftRadices rads[3] = {p->rx, p->ry, p->rz};
	const size_t hx = p->hx, qy = p->qy, qz = p->qz;
	mm_status r = MM_OK;
	for (int ax = 0; ax < 3 && r == MM_OK; ++ax) {
		SpecPass s{};
		// pairs of equal parity; xy, xz, yz (components 1, 2, 4) are odd along their two axes
		const int pairs[3][3][3] = {{{0, 3, 0}, {5, 4, 0}, {1, 2, 1}}, {{0, 3, 0}, {5, 2, 0}, {1, 4, 1}}, {{0, 3, 0}, {5, 1, 0}, {2, 4, 1}}};
		for (int q = 0; q < 3; ++q) {
			s.a[q] = pairs[ax][q][0];
			s.b[q] = pairs[ax][q][1];
			s.odd[q] = pairs[ax][q][2] ^ (part >> ax & 1);
		}
		s.part = part;
		s.scale = 1.0;
		s.m = m[ax];
		int outer = 1;
		if (ax == 0) {
			s.in = octant; s.ic = 1; s.ik = 6; s.ii = 6 * (size_t)m[0]; s.io = 6 * (size_t)m[0] * m[1];
			s.ok = 1; s.oi = hx; s.oo = hx * m[1]; s.oc = hx * m[1] * m[2];
			s.inner = m[1];
			outer = m[2];
		} else if (ax == 1) {
			s.in = A; s.ic = hx * m[1] * m[2]; s.ik = hx; s.ii = 1; s.io = hx * m[1];
			s.ok = hx; s.oi = 1; s.oo = hx * qy; s.oc = hx * qy * m[2];
			s.inner = (int)hx;
			outer = m[2];
		} else {
			s.in = B; s.ic = hx * qy * m[2]; s.ik = hx * qy; s.ii = 1; s.io = 0;
			s.ok = hx * qy; s.oi = 1; s.oo = 0; s.oc = hx * qy * qz;
			s.inner = (int)(hx * qy);
		}
		const int len = p3[ax], TB = pick_tile(len, 1, sizeof(double2), ax == 0 ? 4 : 16);
		const size_t smem = (size_t)(2 * TB + 1) * len * sizeof(double2);
		const dim3 grid((s.inner + TB - 1) / TB, outer, 3);
		if (ax == 0) {
			r = set_smem<double>((const void *)k_spec_axis<double, true>, smem);
			if (r == MM_OK) k_spec_axis<double, true><<<grid, NT, smem, st>>>(s, A, rads[ax], tw[ax], TB);
		} else if (ax == 1) {
			r = set_smem<double>((const void *)k_spec_axis<double, false>, smem);
			if (r == MM_OK) k_spec_axis<double, false><<<grid, NT, smem, st>>>(s, B, rads[ax], tw[ax], TB);
		} else {
			s.scale = 1.0 / ((double)p3[0] * p3[1] * p3[2]);  // the inverse transforms'
			s.signs = true;
			s.add = part != 0;
			r = set_smem<double>((const void *)k_spec_axis<OUT, false>, smem);
			if (r == MM_OK) k_spec_axis<OUT, false><<<grid, NT, smem, st>>>(s, out, rads[ax], tw[ax], TB);
		}
		if (r == MM_OK) r = after_launch("k_spec_axis");
	}
	return r;
}

// N: the octant [nz][ny][nx][6] (octant), or a tensor that was handed in, whose part of the components' own
// parities is taken (of one that has no other: the tensor itself) and, of mixed parity, the others behind it.
template <typename T>
mm_status tensor_spectrum(ConvPlan *p, const double *N, bool octant, cudaStream_t st)
{
	const int n3[3] = {p->nx, p->ny, p->nz}, e3[3] = {p->ex, p->ey, p->ez}, p3[3] = {p->px, p->py, p->pz};
	int m[3];  // offsets of an axis that matter: those of the box, or half a period
	for (int a = 0; a < 3; ++a) m[a] = e3[a] >= 2 * n3[a] - 1 && !p->mixed_parity ? n3[a] : e3[a] / 2 + 1;
	const size_t hx = p->hx, qy = p->qy, qz = p->qz;
	const size_t sizeA = 6 * hx * m[1] * m[2], sizeB = 6 * hx * qy * m[2], sizeS = p->mixed_parity ? 6 * hx * qy * qz : 0;
	std::vector<double2> tw;
	size_t tw_at[3];
	for (int a = 0; a < 3; ++a) {
		tw_at[a] = tw.size();
		for (int k = 0; k < p3[a]; ++k) {
			const long double w = -2.0L * 3.14159265358979323846264338327950288L * (long double)k / (long double)p3[a];
			tw.push_back(double2{(double)cosl(w), (double)sinl(w)});
		}
	}
	double *work = nullptr;  // the x spectrum, the x-y spectrum (and before it the part's octant), the sum of parts, the twiddles
	MM_TRY(setup_alloc((void **)&work, (sizeA + sizeB + sizeS) * sizeof(double) + tw.size() * sizeof(double2), st));
	double *A = work, *B = work + sizeA, *S = B + sizeB;
	double2 *twd = reinterpret_cast<double2 *>(S + sizeS);
	const double2 *const tws[3] = {twd + tw_at[0], twd + tw_at[1], twd + tw_at[2]};
	mm_status r = cuda_status(cudaMemcpyAsync(twd, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice, st),
	                          "cudaMemcpyAsync");
	for (int part : {0, 3, 5, 6}) {
		if (r != MM_OK || (part && !p->mixed_parity)) break;
		if (!octant) r = tensor_part(N, e3, m, part, B, st);  // (m <= hx, qy along x, y)
		if (r != MM_OK) break;
		r = p->mixed_parity ? spectrum_passes<double>(p, B, part, m, A, B, tws, S, st)
		                    : spectrum_passes<T>(p, octant ? N : B, part, m, A, B, tws, (T *)p->tensor, st);
	}
	if (r == MM_OK && p->mixed_parity) {
		k_round<T><<<num_sms() * 8, NT, 0, st>>>(S, (T *)p->tensor, sizeS);
		r = after_launch("k_round");
	}
	setup_free(work, st);
	if (r == MM_OK) r = cuda_status(cudaStreamSynchronize(st), "cudaStreamSynchronize");
	return r;
}

template <typename T>
mm_status plan_setup(ConvPlan *p, const double *N, bool octant, cudaStream_t st)
{
	using C = cplx<T>;
	MM_TRY(make_twiddles<T>(p->px, &p->tw_x));
	MM_TRY(make_twiddles<T>(p->py, &p->tw_y));
	MM_TRY(make_twiddles<T>(p->pz, &p->tw_z));
	MM_CUDA(cudaMalloc(&p->tensor, sizeof(T) * 6 * (size_t)p->qz * p->qy * p->hx));
	MM_CUDA(cudaMalloc(&p->spec, p->spec_bytes()));
	MM_CUDA(cudaMemsetAsync(p->spec, 0, p->spec_bytes(), st));
	// launch geometry
	{
		int lp = 8;
		while (lp > 1 && (size_t)(2 * lp + 1) * p->px * sizeof(C) > SMEM_TARGET) lp >>= 1;
		p->lp_x = lp;
		p->smem_x = (size_t)(2 * lp + 1) * p->px * sizeof(C);
	}
	if (p->is2d) {
		p->tb_y = pick_tile(p->py, 3, sizeof(C), 32);
		p->smem_y = (size_t)(6 * p->tb_y + 1) * p->py * sizeof(C);
	} else {
		p->tb_y = pick_tile(p->py, 1, sizeof(C), 32);
		p->smem_y = (size_t)(2 * p->tb_y + 1) * p->py * sizeof(C);
		p->tb_z = pick_tile(p->pz, 3, sizeof(C), 32);
		p->smem_z = (size_t)(6 * p->tb_z + 1) * p->pz * sizeof(C);
	}
	MM_TRY(fs_setup<T>(p));
	// the mixed-radix passes of the axes without compile-time ones
	if ((!p->fast_x && p->smem_x > 227 * 1024) || (!p->fast_y && p->smem_y > 227 * 1024) ||
	    (!p->is2d && !p->fast_z && p->smem_z > 227 * 1024))
		return fail(MM_ERR_UNSUPPORTED, "conv: FFT length too large for one CTA");
	if (!p->fast_x) {
		MM_TRY(set_smem<T>((const void *)k_x_fwd<T, false>, p->smem_x));
		MM_TRY(set_smem<T>((const void *)k_x_fwd<T, true>, p->smem_x));
		MM_TRY(set_smem<T>((const void *)k_x_inv<T>, p->smem_x));
	}
	if (!p->fast_y && p->is2d) {
		MM_TRY(set_smem<T>((const void *)k_y_mul2d<T>, p->smem_y));
	} else if (!p->fast_y) {
		MM_TRY(set_smem<T>((const void *)k_y<T, false>, p->smem_y));
		MM_TRY(set_smem<T>((const void *)k_y<T, true>, p->smem_y));
	}
	if (!p->is2d && !p->fast_z) MM_TRY(set_smem<T>((const void *)k_z_mul<T>, p->smem_z));
	return tensor_spectrum<T>(p, N, octant, st);
}

template <typename T>
mm_status execute(ConvPlan *p, const T *M, const uint8_t *reg, const T *ms_tab, T *H, cudaStream_t st, Gate gate = Gate())
{
	using C = cplx<T>;
	C *S = (C *)p->spec;
	const int rows = 3 * p->ny * p->nz;
	const int lines = (rows + 1) / 2;
	const int gx = (lines + p->lp_x - 1) / p->lp_x;
	// algorithmic bytes of each pass (every array element crossing HBM once)
	const double n = (double)p->nx * p->ny * p->nz, s = sizeof(T), c = sizeof(C);
	const double half = 3.0 * p->hx * p->ny * p->nz * c;      // x-transformed rows y < ny, z < nz
	const double ypad = 3.0 * p->hx * p->py * p->nz * c;      // y-transformed, z < nz
	const double tens = 6.0 * p->hx * p->qy * p->qz * s;
	ProfToken tk = gate.flags ? ProfToken() : prof_begin(st);
	bool staged = false;
	if (p->tma_xf) {
#define MM_XTF(N) staged = fs_x_fwd_tma<T, N>(p, M, reg, ms_tab, st, gate)
		MM_FS_SWITCH3(p->px, MM_XTF);
#undef MM_XTF
	}
	if (staged) {
	} else if (p->fast_x) {
#define MM_XF(N) fs_x_fwd<T, N>(p, M, reg, ms_tab, st, gate)
		MM_FS_SWITCH3(p->px, MM_XF);
#undef MM_XF
	} else if (ms_tab)
		k_x_fwd<T, true><<<gx, NT, p->smem_x, st>>>(M, reg, ms_tab, S, p->nx, p->ny, p->nz, p->py, p->hx, p->lx,
		                                            p->rx, (const C *)p->tw_x, p->lp_x);
	else
		k_x_fwd<T, false><<<gx, NT, p->smem_x, st>>>(M, reg, ms_tab, S, p->nx, p->ny, p->nz, p->py, p->hx, p->lx,
		                                             p->rx, (const C *)p->tw_x, p->lp_x);
	const char *xf_name = staged ? "k_x_fwd_tma" : p->fast_x ? "k_x_fwd_ct" : "k_x_fwd";
	MM_TRY(after_launch(xf_name));
	prof_end(tk, xf_name, 3 * n * s + (reg ? n : 0.0) + half, st);
	if (p->is2d) {
		const int gy = (p->hx + p->tb_y - 1) / p->tb_y;
		tk = gate.flags ? ProfToken() : prof_begin(st);
		if (p->fast_y) {
#define MM_Y2(N) fs_y2d<T, N>(p, st)
			MM_FS_SWITCH3(p->py, MM_Y2);
#undef MM_Y2
		} else
			k_y_mul2d<T><<<gy, NT, p->smem_y, st>>>(S, (const T *)p->tensor, p->ny, p->hx, p->lx, p->qy, p->ry,
			                                        (const C *)p->tw_y, p->tb_y);
		const char *y2_name = p->fast_y ? "k_y2d_ct" : "k_y_mul2d";
		MM_TRY(after_launch(y2_name));
		prof_end(tk, y2_name, 2 * half + tens, st);
	} else {
		dim3 gy((p->hx + p->tb_y - 1) / p->tb_y, p->nz, 3);
		tk = gate.flags ? ProfToken() : prof_begin(st);
		if (p->tma_y) {
#define MM_YTF(N) fs_y_tma<T, N, false>(p, st, gate)
			MM_FS_SWITCH3(p->py, MM_YTF);
#undef MM_YTF
		} else if (p->fast_y) {
#define MM_YF(N) fs_y<T, N, false>(p, st, gate)
			MM_FS_SWITCH3(p->py, MM_YF);
#undef MM_YF
		} else
			k_y<T, false><<<gy, NT, p->smem_y, st>>>(S, p->ny, p->py, p->nz, p->py, p->hx, p->lx, p->ry,
			                                         (const C *)p->tw_y, p->tb_y);
		const char *yf_name = p->tma_y ? "k_y_tma (forward)" : p->fast_y ? "k_y_ct (forward)" : "k_y (forward)";
		MM_TRY(after_launch(yf_name));
		prof_end(tk, yf_name, half + ypad, st);
		dim3 gz((p->hx + p->tb_z - 1) / p->tb_z, p->py, 1);
		tk = gate.flags ? ProfToken() : prof_begin(st);
		if (p->reg_z) {
			switch (p->pz) {
			case 2: fs_z_reg<T, 2>(p, st, gate); break;
			case 6: fs_z_reg<T, 6>(p, st, gate); break;
			case 12: fs_z_reg<T, 12>(p, st, gate); break;
			case 24: fs_z_reg<T, 24>(p, st, gate); break;
			case 4: fs_z_reg<T, 4>(p, st, gate); break;
			case 8: fs_z_reg<T, 8>(p, st, gate); break;
			case 16: fs_z_reg<T, 16>(p, st, gate); break;
			case 32: if constexpr (sizeof(T) == 4) { fs_z_reg<T, 32>(p, st, gate); } break;
			}
		} else if (p->fast_z) {
			switch (p->pz) {
			case 2: fs_z<T, 2>(p, st); break;
			case 4: fs_z<T, 4>(p, st); break;
			case 8: fs_z<T, 8>(p, st); break;
			case 16: fs_z<T, 16>(p, st); break;
			case 32: fs_z<T, 32>(p, st); break;
			case 64: fs_z<T, 64>(p, st); break;
			}
		} else
			k_z_mul<T><<<gz, NT, p->smem_z, st>>>(S, (const T *)p->tensor, p->nz, p->py, p->hx, p->lx, p->qy, p->qz,
			                                      p->rz, (const C *)p->tw_z, p->tb_z);
		const char *z_name = p->reg_z ? "k_z_reg" : p->fast_z ? "k_z_ct" : "k_z_mul";
		MM_TRY(after_launch(z_name));
		prof_end(tk, z_name, 2 * ypad + tens, st);
		tk = gate.flags ? ProfToken() : prof_begin(st);
		if (p->tma_y) {
#define MM_YTI(N) fs_y_tma<T, N, true>(p, st, gate)
			MM_FS_SWITCH3(p->py, MM_YTI);
#undef MM_YTI
		} else if (p->fast_y) {
#define MM_YI(N) fs_y<T, N, true>(p, st, gate)
			MM_FS_SWITCH3(p->py, MM_YI);
#undef MM_YI
		} else
			k_y<T, true><<<gy, NT, p->smem_y, st>>>(S, p->py, p->ny, p->nz, p->py, p->hx, p->lx, p->ry,
			                                        (const C *)p->tw_y, p->tb_y);
		const char *yi_name = p->tma_y ? "k_y_tma (inverse)" : p->fast_y ? "k_y_ct (inverse)" : "k_y (inverse)";
		MM_TRY(after_launch(yi_name));
		prof_end(tk, yi_name, half + ypad, st);
	}
	tk = gate.flags ? ProfToken() : prof_begin(st);
	if (p->tma_xi) {
#define MM_XTI(N) fs_x_inv_tma<T, N>(p, H, st, gate)
		MM_FS_SWITCH3(p->px, MM_XTI);
#undef MM_XTI
	} else if (p->fast_x) {
#define MM_XI(N) fs_x_inv<T, N>(p, H, st, gate)
		MM_FS_SWITCH3(p->px, MM_XI);
#undef MM_XI
	} else
		k_x_inv<T><<<gx, NT, p->smem_x, st>>>(S, H, p->nx, p->ny, p->nz, p->py, p->hx, p->lx, p->rx,
		                                      (const C *)p->tw_x, p->lp_x);
	const char *xi_name = p->tma_xi ? "k_x_inv_tma" : p->fast_x ? "k_x_inv_ct" : "k_x_inv";
	MM_TRY(after_launch(xi_name));
	prof_end(tk, xi_name, half + 3 * n * s, st);
	return MM_OK;
}

} // namespace

} // namespace mm
