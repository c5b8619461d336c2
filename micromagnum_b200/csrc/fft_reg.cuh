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

// cos(2 pi q / 64) and cos(2 pi q / 48) for the first quarter, and the rest by symmetry.  Called with
// constants after unrolling, so the values are operands in the instruction stream: from __constant__
// tables they were fetched anew by every SM in every launch, which the short launches waited for.
__host__ __device__ constexpr double cos_q64(int q)
{
	switch (q) {
	case 0: return 1.0;
	case 1: return 0.99518472667219688624;
	case 2: return 0.98078528040323044913;
	case 3: return 0.95694033573220886494;
	case 4: return 0.92387953251128675613;
	case 5: return 0.88192126434835502971;
	case 6: return 0.83146961230254523708;
	case 7: return 0.77301045336273696081;
	case 8: return 0.70710678118654752440;
	case 9: return 0.63439328416364549822;
	case 10: return 0.55557023301960222474;
	case 11: return 0.47139673682599764856;
	case 12: return 0.38268343236508977173;
	case 13: return 0.29028467725446236764;
	case 14: return 0.19509032201612826785;
	case 15: return 0.09801714032956060199;
	default: return 0.0;
	}
}
__host__ __device__ constexpr double cos_q48(int q)
{
	switch (q) {
	case 0: return 1.0;
	case 1: return 0.99144486137381041114;
	case 2: return 0.96592582628906828675;
	case 3: return 0.92387953251128675613;
	case 4: return 0.86602540378443864676;
	case 5: return 0.79335334029123516458;
	case 6: return 0.70710678118654752440;
	case 7: return 0.60876142900872063942;
	case 8: return 0.5;
	case 9: return 0.38268343236508977173;
	case 10: return 0.25881904510252076235;
	case 11: return 0.13052619222005159155;
	default: return 0.0;
	}
}
// cos(2 pi q / n) for n = 64 or 48, any q >= 0
__host__ __device__ constexpr double cos_of(int q, int n)
{
	q %= n;
	if (2 * q > n) q = n - q;
	const bool neg = 4 * q > n;
	if (neg) q = n / 2 - q;
	const double c = n == 64 ? cos_q64(q) : cos_q48(q);
	return neg ? -c : c;
}
// W_n^q = exp(-2 pi i q / n): sin(2 pi q / n) = cos(2 pi (q - n / 4) / n)
template <typename T>
__device__ __forceinline__ cplx<T> w64(int q)
{
	return {(T)cos_of(q, 64), (T)-cos_of(q + 48, 64)};
}
template <typename T>
__device__ __forceinline__ cplx<T> w48(int q)
{
	return {(T)cos_of(q, 48), (T)-cos_of(q + 36, 48)};
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

// v W_64^q (conjugated for the inverse), q a compile-time constant after unrolling.
template <typename T, bool INV>
__device__ __forceinline__ cplx<T> mul_w64(cplx<T> v, int q)
{
	if (q == 0) return v;
	if (q == 16) return mul_mi<INV>(v);
	cplx<T> w = w64<T>(q);
	if (INV) w = conjc(w);
	return cmul(v, w);
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
				v[b + j + Q] = mul_w64<T, INV>(csub_pk<PK>(s0, s1), 2 * q);
				v[b + j + 2 * Q] = mul_w64<T, INV>(cadd_mi<INV>(d0, d1), q);
				v[b + j + 3 * Q] = mul_w64<T, INV>(csub_mi<INV>(d0, d1), 3 * q);
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
	const T s60 = T(0.86602540378443864676372317075293618);  // sin(60 deg)
	C y[3][M];
#pragma unroll
	for (int j = 0; j < M; ++j) {
		const C a = v[j], b = v[j + M], c = v[j + 2 * M];
		const C s = cadd_pk<PK>(b, c), d = csub_pk<PK>(b, c);
		const C t = C{a.x - T(0.5) * s.x, a.y - T(0.5) * s.y};
		const C r = mul_mi<INV>(C{s60 * d.x, s60 * d.y});
		y[0][j] = cadd_pk<PK>(a, s);
		C y1 = cadd(t, r), y2 = csub(t, r);
		if (j > 0) {
			C w1 = w48<T>(j * (48 / N)), w2 = w48<T>(2 * j * (48 / N));
			if (INV) {
				w1 = conjc(w1);
				w2 = conjc(w2);
			}
			y1 = cmul(y1, w1);
			y2 = cmul(y2, w2);
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
			v[j + Q] = mul_w64<T, false>(csub_pk<PK>(x0, x1), 2 * q);
			v[j + 2 * Q] = mul_w64<T, false>(cadd_mi<false>(x0, x1), q);
			v[j + 3 * Q] = mul_w64<T, false>(csub_mi<false>(x0, x1), 3 * q);
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
