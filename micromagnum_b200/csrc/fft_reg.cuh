// Register-resident FFT building blocks for lengths 2^k and 3 * 2^k (included by conv_passes.cuh).
//
// dft_reg<T, N, INV>: an N-point DFT (N up to 64, or 3 * 2^k up to 48) held entirely in one thread's
// registers, radix-4 decimation in frequency (a radix-2 stage last where 4 does not divide, after one
// radix-3 stage for N = 3 * 2^k), fully unrolled, output k in register dft_pos<N>(k).  Its twiddles are
// compile-time constants.
//
// Longer transforms are CTA-wide Stockham passes over shared memory (cta_fft below).  No index
// arithmetic depends on run-time values except the tile offsets, so the inner work is straight-line code.
#pragma once

#include "fft.cuh"

namespace mm {

// cos(2 pi r / n) - 1 and sin(2 pi r / n) for n = 64 or 48, 0 < r < n / 8.  Called with constants after
// unrolling, so the values are operands in the instruction stream: from __constant__ tables they were
// fetched anew by every SM in every launch, which the short launches waited for.
__host__ __device__ constexpr double cosm1_of(int r, int n)
{
	switch (n == 64 ? r : 8 + r) {
	case 1: return -0.004815273327803113755;
	case 2: return -0.019214719596769550874;
	case 3: return -0.043059664267791135064;
	case 4: return -0.076120467488713243872;
	case 5: return -0.118078735651644970287;
	case 6: return -0.168530387697454762921;
	case 7: return -0.226989546637263039189;
	case 9: return -0.008555138626189588855;
	case 10: return -0.034074173710931713250;
	case 11: return -0.076120467488713243872;
	case 12: return -0.133974596215561353236;
	case 13: return -0.206646659708764835420;
	default: return 0.0;
	}
}
__host__ __device__ constexpr double sin_of(int r, int n)
{
	switch (n == 64 ? r : 8 + r) {
	case 1: return 0.098017140329560601994;
	case 2: return 0.195090322016128267848;
	case 3: return 0.290284677254462367636;
	case 4: return 0.382683432365089771728;
	case 5: return 0.471396736825997648556;
	case 6: return 0.555570233019602224743;
	case 7: return 0.634393284163645498215;
	case 9: return 0.130526192220051591548;
	case 10: return 0.258819045102520762349;
	case 11: return 0.382683432365089771728;
	case 12: return 0.5;
	case 13: return 0.608761429008720639416;
	default: return 0.0;
	}
}

__host__ __device__ constexpr bool fft_is_pow2(int n) { return (n & (n - 1)) == 0; }

__host__ __device__ constexpr int brev_c(int k, int n)
{
	int r = 0;
	for (int m = n >> 1; m > 0; m >>= 1, k >>= 1) r = (r << 1) | (k & 1);
	return r;
}

template <int N>
__device__ __forceinline__ int brev(int k) { return brev_c(k, N); }

// Register that holds output k of an N-point register transform: bit-reversed for a power of two;
// for N = 3 M the outputs 3 k' + r are the r-th M-point transform's output k' (dft_reg3).
template <int N>
__device__ __forceinline__ constexpr int dft_pos(int k)
{
	if (fft_is_pow2(N)) return brev_c(k, N);
	return (k % 3) * (N / 3) + brev_c(k / 3, N / 3);
}

// v (hi + lo), a constant in two parts; packed (PK) it is as many instructions as a plain constant.
template <bool PK, typename T>
__device__ __forceinline__ cplx<T> mul_parts(cplx<T> v, T hi, T lo)
{
	using C = cplx<T>;
	if constexpr (PK) return cfma2(C{hi, hi}, v, cscale2(C{lo, lo}, v));
	else return {fma(v.x, hi, v.x * lo), fma(v.y, hi, v.y * lo)};
}
template <bool PK, typename T>
__device__ __forceinline__ cplx<T> mul_sqrt_half(cplx<T> v)
{
	constexpr double c = 0.70710678118654752440;
	constexpr T hi = (T)c, lo = sizeof(T) == 4 ? (T)(c - (double)hi) : (T)-4.8336466567264565e-17;
	return mul_parts<PK, T>(v, hi, lo);
}
template <bool PK, typename T>
__device__ __forceinline__ cplx<T> mul_sin60(cplx<T> v)
{
	constexpr double c = 0.86602540378443864676;
	constexpr T hi = (T)c, lo = sizeof(T) == 4 ? (T)(c - (double)hi) : (T)5.0175421109034514e-17;
	return mul_parts<PK, T>(v, hi, lo);
}

// v W_n^q (conjugated for the inverse), n = 64 or 48, q a compile-time constant after unrolling.  The
// constants are the same in every line and in both directions of a convolution, so a constant whose
// modulus is off by its rounding scales what it touches twice, coherently: with W rounded to T they were
// more than half of the FP32 field's error at lengths 2^k and 3 * 2^k.  So W is a number of quarter turns
// (exact) and a turn of at most n / 8: 1 + (cos - 1) - i sin, whose rounding is relative to the small
// parts, in four operations like the plain product; an eighth turn multiplies by sqrt(1/2) in two parts.
// Against direct sums in 80 bits, 128x32 cells, FP32: 1.14e-7, against 1.47e-7 with rounded twiddles
// and 1.62e-7 in the mixed-radix passes that these took over; 33x30x3: 0.98e-7, 1.34e-7, 1.36e-7; FP64, 128x32:
// 2.7e-16, 3.0e-16, 3.3e-16.  An evaluation of a 128x32 film takes about 1% longer, a larger box less.
template <typename T, bool INV, int n, bool PK>
__device__ __forceinline__ cplx<T> mul_w(cplx<T> v, int q)
{
	const int k = (8 * q / n + 1) / 2, r = q - k * (n / 4);
	const bool minus = (r > 0) != INV;  // the turn is 1 - i tan
	if (r == n / 8 || r == -n / 8) {
		v = minus ? cplx<T>{v.x + v.y, v.y - v.x} : cplx<T>{v.x - v.y, v.y + v.x};
		v = mul_sqrt_half<PK, T>(v);
	} else if (r != 0) {
		const T c = (T)cosm1_of(r < 0 ? -r : r, n), s = (T)(minus ? -sin_of(r < 0 ? -r : r, n) : sin_of(r < 0 ? -r : r, n));
		v = {fma(v.x, c, fma(-v.y, s, v.x)), fma(v.x, s, fma(v.y, c, v.y))};
	}
#pragma unroll
	for (int i = 0; i < k; ++i) v = mul_mi<INV>(v);
	return v;
}

// Decimation-in-frequency stages over v[0..N): a radix-4 stage stands for the radix-2 stages of spans
// SPAN0 and SPAN0/2 (and leaves its outputs where they would), so a value passes one twiddle
// multiplication where two radix-2 stages have two (8 instead of 10 in a 16-point transform, and the
// smaller rounding error); SPAN0 = N/2 is the full transform.
template <typename T, int N, bool INV, int SPAN0, bool PK = true>
__device__ __forceinline__ void dif_stages(cplx<T> (&v)[N])
{
	using C = cplx<T>;
	if constexpr (SPAN0 >= 2) {
		constexpr int Q = SPAN0 / 2;  // a butterfly's inputs are Q apart, its transform has 4 Q points
#pragma unroll
		for (int b = 0; b < N; b += 4 * Q) {
#pragma unroll
			for (int j = 0; j < Q; ++j) {
				const C x0 = v[b + j], x1 = v[b + j + Q], x2 = v[b + j + 2 * Q], x3 = v[b + j + 3 * Q];
				const C s0 = cadd_pk<PK>(x0, x2), d0 = csub_pk<PK>(x0, x2), s1 = cadd_pk<PK>(x1, x3), d1 = csub_pk<PK>(x1, x3);
				const int q = j * (64 / (4 * Q));  // W_4Q^j = W_64^q
				v[b + j] = cadd_pk<PK>(s0, s1);
				v[b + j + Q] = mul_w<T, INV, 64, PK>(csub_pk<PK>(s0, s1), 2 * q);
				v[b + j + 2 * Q] = mul_w<T, INV, 64, PK>(cadd_mi<INV>(d0, d1), q);
				v[b + j + 3 * Q] = mul_w<T, INV, 64, PK>(csub_mi<INV>(d0, d1), 3 * q);
			}
		}
		if constexpr (Q >= 2) dif_stages<T, N, INV, Q / 2, PK>(v);
	} else if constexpr (SPAN0 == 1) {
#pragma unroll
		for (int b = 0; b < N; b += 2) {
			const C a = v[b], c = v[b + 1];
			v[b] = cadd_pk<PK>(a, c);
			v[b + 1] = csub_pk<PK>(a, c);
		}
	}
}

// N = 3 M points (M a power of two, N <= 48): one radix-3 stage over the inputs M apart, the
// twiddles W_N^(r j), then three M-point transforms in place.  Outputs at dft_pos<N>.
template <typename T, int N, bool INV, bool PK = true>
__device__ __forceinline__ void dft_reg3(cplx<T> (&v)[N])
{
	using C = cplx<T>;
	constexpr int M = N / 3;
	static_assert(3 * M == N && fft_is_pow2(M) && 48 % N == 0, "3 * 2^k points, at most 48");
	C y[3][M];
#pragma unroll
	for (int j = 0; j < M; ++j) {
		const C a = v[j], b = v[j + M], c = v[j + 2 * M];
		const C s = cadd_pk<PK>(b, c), d = csub_pk<PK>(b, c);
		const C t = C{a.x - T(0.5) * s.x, a.y - T(0.5) * s.y};
		const C r = mul_mi<INV>(mul_sin60<PK, T>(d));
		y[0][j] = cadd_pk<PK>(a, s);
		C y1 = cadd(t, r), y2 = csub(t, r);
		if (j > 0) {
			y1 = mul_w<T, INV, 48, PK>(y1, j * (48 / N));
			y2 = mul_w<T, INV, 48, PK>(y2, 2 * j * (48 / N));
		}
		y[1][j] = y1;
		y[2][j] = y2;
	}
#pragma unroll
	for (int r = 0; r < 3; ++r) {
		if constexpr (M > 1) dif_stages<T, M, INV, M / 2, PK>(y[r]);
#pragma unroll
		for (int j = 0; j < M; ++j) v[r * M + j] = y[r][j];
	}
}

template <typename T, int N, bool INV, bool PK = true>
__device__ __forceinline__ void dft_reg(cplx<T> (&v)[N])
{
	if constexpr (fft_is_pow2(N)) dif_stages<T, N, INV, N / 2, PK>(v);
	else dft_reg3<T, N, INV, PK>(v);
}

// Forward DFT of a column whose upper half v[N/2..N) is zero padding: the first stage's butterflies
// have two inputs.  Output at dft_pos<N>, like dft_reg.
template <typename T, int N, bool PK = true>
__device__ __forceinline__ void dft_reg_halfzero(cplx<T> (&v)[N])
{
	using C = cplx<T>;
	if constexpr (!fft_is_pow2(N)) {
#pragma unroll
		for (int j = N / 2; j < N; ++j) v[j] = C{T(0), T(0)};
		dft_reg3<T, N, false, PK>(v);
	} else if constexpr (N >= 4) {
		constexpr int Q = N / 4;
#pragma unroll
		for (int j = 0; j < Q; ++j) {
			const C x0 = v[j], x1 = v[j + Q];
			const int q = j * (64 / N);
			v[j] = cadd_pk<PK>(x0, x1);
			v[j + Q] = mul_w<T, false, 64, PK>(csub_pk<PK>(x0, x1), 2 * q);
			v[j + 2 * Q] = mul_w<T, false, 64, PK>(cadd_mi<false>(x0, x1), q);
			v[j + 3 * Q] = mul_w<T, false, 64, PK>(csub_mi<false>(x0, x1), 3 * q);
		}
		if constexpr (Q >= 2) dif_stages<T, N, false, Q / 2, PK>(v);
	} else if constexpr (N == 2) {
		v[1] = v[0];
	}
}

} // namespace mm

namespace mm {

// ---- CTA-wide Stockham FFT with compile-time length and radix -----------------------------------
// LANES independent lines of length N live in shared memory; each of the N/R threads of a line
// performs R/Rp radix-Rp butterflies per pass (Rp: fft_radix).  Pass 0
// reads its inputs through `ld(line, k)` (global memory, with zero padding), the last pass hands
// its outputs to `st(line, k, value)`; intermediate passes go through shared memory at
// `SmIdx::at(line, k)`.  All strides are compile-time powers of two.
__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n / 2); }
// Radices: a power of two takes passes of radix R and a smaller last one; N = 3 * 2^k (R = 24, or
// N itself below 24) takes radix 8 until at most 24 points are left, which are the last pass (so
// the factor 3 comes last and every earlier stride stays a power of two).
__host__ __device__ constexpr int fft_npasses(int N, int R)
{
	if (!fft_is_pow2(N)) {
		int p = 1;
		for (; N > 24; N /= 8) ++p;
		return p;
	}
	return (ilog2c(N) + ilog2c(R) - 1) / ilog2c(R);
}
__host__ __device__ constexpr int fft_radix(int N, int R, int p)
{
	if (!fft_is_pow2(N)) {
		for (; p > 0; --p) N /= 8;
		return N > 24 ? 8 : N;
	}
	return ilog2c(N) - p * ilog2c(R) >= ilog2c(R) ? R : (1 << (ilog2c(N) - p * ilog2c(R)));
}

// Twiddles of the passes p >= 1, one block per pass: entry (q, jm), 1 <= q < Rp, jm < Ns, at
// fft_tw_off(N, R, p) + (q - 1) Ns + jm holds W_(Ns Rp)^(q jm).  The threads of a warp work on
// consecutive butterflies, so for each q they read consecutive entries: one coalesced line from
// global memory, or a conflict-free shared-memory access.  (Reading the same values from a plain
// table W_N^k, at multiples of q N / (Ns Rp), put up to 16 lanes of a warp on one bank: the y pass
// of 1024 points spent 84 us on the 512x512x16 slab, FP32, against 78 us with this layout,
// the forward x pass 74 against 59.)  Fewer than N entries in all.
__host__ __device__ constexpr int fft_tw_off(int N, int R, int p)
{
	int off = 0, ns = fft_radix(N, R, 0);
	for (int i = 1; i < p; ++i) {
		off += (fft_radix(N, R, i) - 1) * ns;
		ns *= fft_radix(N, R, i);
	}
	return off;
}

// Shared-memory layouts.  One padding slot per 2^SH elements skews the Stockham pass-0 writes
// (stride R) and the column tiles across the banks.  SH = 4 makes the radix-16 pass-0 writes of
// 8-byte elements conflict-free (consecutive butterflies 17 elements = 34 words apart, so a
// half-warp's 16 stores cover all 32 banks once); SH = 5 halves the padding.
template <int SH = 5>
__host__ __device__ constexpr int sm_pad(int raw) { return raw + (raw >> SH); }
template <int N, int LANES, int SH = 5>
struct SmCols {  // element (line, k) at k * LANES + line: lines are adjacent columns
	static constexpr int SIZE = N * LANES + (N * LANES >> SH) + 1;
	__device__ __forceinline__ static int at(int line, int k) { return sm_pad<SH>(k * LANES + line); }
};
template <int N, int LANES, int SH = 5>
struct SmRows {  // element (line, k) at line * N + k
	static constexpr int SIZE = N * LANES + (N * LANES >> SH) + 1;
	__device__ __forceinline__ static int at(int line, int k) { return sm_pad<SH>(line * N + k); }
};

// Hook run by every thread after pass 0 has stored its outputs (a no-op unless a kernel stages
// its inputs and can release their buffer once pass 0 has read them).
struct NoHook {
	__device__ __forceinline__ void operator()() const {}
};

// H0: the inputs at k >= N/2 are zero (a forward transform of zero-padded data), so pass 0 loads
// only the lower half of each butterfly's inputs and runs the half-zero register DFT.
template <typename T, int N, int R, int LANES, bool INV, class SmIdx, bool LD_SM, int p, bool H0, bool PK, class LD,
          class ST, class HK = NoHook>
__device__ __forceinline__ void cta_fft_pass(cplx<T> *sm, const cplx<T> *__restrict__ twp, int line, int j0,
                                             LD &ld, ST &st, HK hk = HK())
{
	using C = cplx<T>;
	constexpr int P = fft_npasses(N, R);
	constexpr int Rp = fft_radix(N, R, p);
	constexpr int Ns = 1 << (p * (fft_is_pow2(N) ? ilog2c(R) : 3));  // product of the radices of earlier passes
	constexpr int TPL = N / R;
	constexpr int BPT = R / Rp;
	constexpr int M = N / Rp;                  // butterflies per line, input stride
	constexpr bool HALF = H0 && p == 0;
	static_assert(!HALF || (!INV && Rp % 2 == 0), "half-zero pass 0: forward, an even radix");
	static_assert(R % Rp == 0, "a thread takes whole butterflies");
	C v[BPT][Rp];
	if constexpr (p > 0) __syncthreads();
#pragma unroll
	for (int u = 0; u < BPT; ++u) {
		const int j = j0 + u * TPL;
#pragma unroll
		for (int q = 0; q < (HALF ? Rp / 2 : Rp); ++q) {
			if constexpr (p == 0) v[u][q] = ld(line, j + q * M);
			else v[u][q] = sm[SmIdx::at(line, j + q * M)];
		}
	}
	if constexpr (p > 0 || LD_SM) __syncthreads();  // all inputs read before any output lands
#pragma unroll
	for (int u = 0; u < BPT; ++u) {
		const int j = j0 + u * TPL;
		const int jm = j & (Ns - 1);
		if constexpr (Ns > 1) {
			const C *tw = twp + fft_tw_off(N, R, p) + jm;
#pragma unroll
			for (int q = 1; q < Rp; ++q) {
				C w = tw[(q - 1) * Ns];
				if (INV) w = conjc(w);
				v[u][q] = cmul(v[u][q], w);
			}
		}
		if constexpr (HALF) dft_reg_halfzero<T, Rp, PK>(v[u]);
		else dft_reg<T, Rp, INV, PK>(v[u]);
		const int base = (j / Ns) * Ns * Rp + jm;
#pragma unroll
		for (int k = 0; k < Rp; ++k) {
			const C val = v[u][dft_pos<Rp>(k)];
			if constexpr (p == P - 1) st(line, base + k * Ns, val);
			else sm[SmIdx::at(line, base + k * Ns)] = val;
		}
	}
	if constexpr (p == 0) hk();
	if constexpr (p + 1 < P)
		cta_fft_pass<T, N, R, LANES, INV, SmIdx, LD_SM, p + 1, false, PK>(sm, twp, line, j0, ld, st, hk);
}

// LD_SM: the loader reads the same shared memory the passes write (adds a barrier after pass 0's
// reads).
template <typename T, int N, int R, int LANES, bool INV, class SmIdx, bool LD_SM = false, bool PK = true, class LD,
          class ST, class HK = NoHook>
__device__ __forceinline__ void cta_fft(cplx<T> *sm, const cplx<T> *__restrict__ twp, int line, int j0, LD &ld,
                                        ST &st, HK hk = HK())
{
	cta_fft_pass<T, N, R, LANES, INV, SmIdx, LD_SM, 0, false, PK>(sm, twp, line, j0, ld, st, hk);
}

// Forward transform whose inputs at k >= N/2 are zero (ld is not called for them).
template <typename T, int N, int R, int LANES, class SmIdx, bool LD_SM = false, bool PK = true, class LD,
          class ST, class HK = NoHook>
__device__ __forceinline__ void cta_fft_h0(cplx<T> *sm, const cplx<T> *__restrict__ twp, int line, int j0, LD &ld,
                                           ST &st, HK hk = HK())
{
	cta_fft_pass<T, N, R, LANES, false, SmIdx, LD_SM, 0, true, PK>(sm, twp, line, j0, ld, st, hk);
}

} // namespace mm
