// cpic_fft.cuh -- periodic FFT Poisson solver for any grid (radix-4/2
// passes for power-of-two sides, mixed-radix passes otherwise), templated
// on the real type (double for the FP64 form, float for the mixed form).
//
// Replaces MFT_solve (src/solver.c:465-509): phi = IFFT(G * FFT(rho)) / (nx
// ny) with G(kx,ky) = 1 / (2 (cos(2 pi kx/nx) + cos(2 pi ky/ny)) - 4) and
// G(0,0) = 0 (solver.c:269-280).  Three kernels, all working in shared
// memory with Stockham passes (self-sorting, no bit reversal):
//   rows_fwd : two real rows packed as one complex row, FFT along x, split
//              into the two half spectra (nx/2+1 bins each; the last row
//              of an odd ny alone);
//   cols     : a few spectrum columns per block, FFT along y, multiply by G,
//              inverse FFT along y (the Green's function never leaves
//              shared memory);
//   rows_inv : two half spectra packed into one Hermitian-extended row,
//              inverse FFT, real and imaginary parts are the two phi rows,
//              divided by nx*ny as MFT_normalize does (solver.c:366).
//
// What bounds them, and the split that follows.  An FP64 instruction of one
// warp takes 67 clocks whatever its lanes or its independence of the next,
// and an SM starts one every 20 clocks (measured), so the FP64 transforms
// are bound by the chain of FP64 instructions of one warp on small grids and
// by their number per SM on large ones: columns go one (or two) to a block
// so that every SM has its share, and each lane computes one component (real
// or imaginary) of a butterfly, which halves the chain without adding work.
// The FP32 transforms are bound by the latency of their passes: columns
// are spread over blocks until every SM has one.
#pragma once
#include <cuda_runtime.h>
#include "cpic_common.cuh"

namespace cpic {

template <typename T> struct Cx;
template <> struct Cx<double> { typedef double2 t; };
template <> struct Cx<float> { typedef float2 t; };

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C>
__device__ __forceinline__ C cmul(C a, C b)
{
	C r;
	r.x = a.x * b.x - a.y * b.y;
	r.y = a.x * b.y + a.y * b.x;
	return r;
}

// Twiddle exp(-2 pi i m / n) for 0 <= m < n from the half table
// tw[m] (m < n/2): exp(-2 pi i (m + n/2) / n) = -exp(-2 pi i m / n).
template <typename C>
__device__ __forceinline__ C twiddle(const C *tw, int m, int half, int sign)
{
	C w = m < half ? tw[m] : tw[m - half];
	if(m >= half) { w.x = -w.x; w.y = -w.y; }
	if(sign > 0) w.y = -w.y;
	return w;
}

// The passes of a transform of any length: radix r after sub-transforms of
// length Ns (the product of the radices before it), 4s first, then 2, then
// the odd primes in increasing order.  Power-of-two lengths use npass = 0
// and the radix-4 passes below.
struct FftPlan {
	int n, log2n;             // log2n: exponent of the power of two >= n
	int npass;
	int r[14];
	int Ns[14];
	uint32_t mul_ns[14], mul_m[14];   // division by Ns and by n / r (bits::div_q)
	int sh_ns[14], sh_m[14];
	uint32_t mul_n;           // division by n
	int sh_n;
};

inline FftPlan fft_plan(int n)
{
	FftPlan p;
	memset(&p, 0, sizeof(p));
	p.n = n;
	while((1 << p.log2n) < n) p.log2n++;
	if((1 << p.log2n) == n)
		return p;
	bits::div_init((uint32_t) n, p.mul_n, p.sh_n);
	int rem = n, Ns = 1;
	while(rem > 1)
	{
		int r = 3;
		if(rem % 4 == 0) r = 4;
		else if(rem % 2 == 0) r = 2;
		else while(rem % r) r += 2;
		const int k = p.npass++;
		p.r[k] = r;
		p.Ns[k] = Ns;
		bits::div_init((uint32_t) Ns, p.mul_ns[k], p.sh_ns[k]);
		bits::div_init((uint32_t) (n / r), p.mul_m[k], p.sh_m[k]);
		Ns *= r;
		rem /= r;
	}
	return p;
}

// Elements between the starts of consecutive sequences in shared memory: the
// 4 spare ones keep the transposing loads and stores of several columns off
// each other's banks.
__host__ __device__ inline int fft_pitch(int n, int nb) { return nb > 1 ? n + 4 : n; }

// ------------------------------------------------ power-of-two lengths
//
// nb independent length-n sequences, `pitch` elements apart, in `a`; `b` is
// scratch of the same size.  tw[k] = exp(-2 pi i k / n), k < n/2.
// sign -1 forward, +1 inverse (unnormalised).  Returns the buffer holding
// the result.  Must be called by the whole block; blockDim.x a multiple of
// 32.
//
// Stockham autosort passes (no bit reversal): one radix-2 pass first when
// log2 n is odd (sub-transforms of length 1: unit twiddles), then radix-4
// passes.  A radix-4 pass with sub-transform length Ns takes x[j + q n/4],
// q = 0..3, twiddles them by exp(sign 2 pi i q k / (4 Ns)) (k = j mod Ns)
// and writes their 4-point DFT to y[4 (j - k) + k + p Ns], p = 0..3: half
// as many passes and block barriers as radix 2.
template <typename C>
__device__ C *fft_smem(C *a, C *b, int n, int log2n, int nb, int pitch, int sign, const C *tw)
{
	const int half = n >> 1;
	int Ns = 1, s = 0;
	if(log2n & 1)
	{
		const int total = half * nb;
		for(int idx = threadIdx.x; idx < total; idx += blockDim.x)
		{
			int seq = idx >> (log2n - 1);
			int j = idx & (half - 1);
			const C *x = a + seq * pitch;
			C *y = b + seq * pitch;
			C a0 = x[j], a1 = x[j + half];
			y[2 * j] = cadd(a0, a1);
			y[2 * j + 1] = csub(a0, a1);
		}
		__syncthreads();
		C *t = a; a = b; b = t;
		Ns = 2;
		s = 1;
	}
	const int q4 = n >> 2;
	for(; Ns < n; Ns <<= 2, s += 2)
	{
		const int total = q4 * nb;
		const int sh = log2n - 2 - s;        // n / (4 Ns) = 2^sh
		for(int idx = threadIdx.x; idx < total; idx += blockDim.x)
		{
			int seq = idx >> (log2n - 2);
			int j = idx & (q4 - 1);
			const C *x = a + seq * pitch;
			C *y = b + seq * pitch;
			int k = j & (Ns - 1);
			C v0 = x[j];
			C v1 = cmul(x[j + q4], twiddle(tw, k << sh, half, sign));
			C v2 = cmul(x[j + 2 * q4], twiddle(tw, (2 * k) << sh, half, sign));
			C v3 = cmul(x[j + 3 * q4], twiddle(tw, (3 * k) << sh, half, sign));
			C t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3), t3 = csub(v1, v3);
			// t3 times -i (forward) or +i (inverse)
			C r3;
			if(sign < 0) { r3.x = t3.y; r3.y = -t3.x; }
			else { r3.x = -t3.y; r3.y = t3.x; }
			int o = ((j - k) << 2) + k;
			y[o] = cadd(t0, t2);
			y[o + Ns] = cadd(t1, r3);
			y[o + 2 * Ns] = csub(t0, t2);
			y[o + 3 * Ns] = csub(t1, r3);
		}
		__syncthreads();
		C *t = a; a = b; b = t;
	}
	return a;
}

// One component of a complex value, and of its product with a twiddle
// (conjugated for the inverse): two FP64 instructions instead of four.
__device__ __forceinline__ double comp(double2 v, bool im) { return im ? v.y : v.x; }
__device__ __forceinline__ double neg_if(double v, bool neg)
{
	return __longlong_as_double(__double_as_longlong(v) ^ (neg ? (long long) 0x8000000000000000ull : 0ll));
}
__device__ __forceinline__ double cmul_comp(double2 x, double2 w, bool im)
{
	// re: x.x w.x - x.y w.y     im: x.x w.y + x.y w.x
	return __fma_rn(x.y, im ? w.x : neg_if(w.y, true), __dmul_rn(x.x, im ? w.y : w.x));
}
__device__ __forceinline__ double other_comp(double v)
{
	return __shfl_xor_sync(0xffffffffu, v, 1);
}

// The FP64 transform: the passes of fft_smem with each butterfly shared by
// two neighbouring lanes, one per component (the 4-point DFT crosses
// components once, in t3, by a shuffle).  Products are fused
// multiply-adds: 14 FP64 instructions per lane and butterfly, 8 in the
// first pass (unit twiddles), against 34 for one lane doing both without
// fusing.
__device__ inline double2 *fft_smem(double2 *a, double2 *b, int n, int log2n, int nb, int pitch,
		int sign, const double2 *tw)
{
	const int half = n >> 1;
	const bool im = threadIdx.x & 1;
	int Ns = 1, s = 0;
	if(log2n & 1)
	{
		const int total = n * nb;                // half n butterflies, two lanes each
		for(int idx = threadIdx.x; idx < total; idx += blockDim.x)
		{
			const int seq = idx >> log2n;
			const int j = (idx & (n - 1)) >> 1;
			const double *x = reinterpret_cast<const double *>(a + seq * pitch) + im;
			double *y = reinterpret_cast<double *>(b + seq * pitch) + im;
			const double a0 = x[2 * j], a1 = x[2 * (j + half)];
			y[4 * j] = a0 + a1;
			y[4 * j + 2] = a0 - a1;
		}
		__syncthreads();
		double2 *t = a; a = b; b = t;
		Ns = 2;
		s = 1;
	}
	const int q4 = n >> 2;
	for(; Ns < n; Ns <<= 2, s += 2)
	{
		const int total = half * nb;             // n/4 butterflies, two lanes each
		const int sh = log2n - 2 - s;
		for(int base = 0; base < total; base += blockDim.x)
		{
			// every lane takes part in the shuffle; lanes past the end repeat
			// the last butterfly and store nothing
			const int idx = base + (int) threadIdx.x;
			const bool on = idx < total;
			const int i = on ? idx : total - 2 + im;
			const int seq = i >> (log2n - 1);
			const int j = (i & (half - 1)) >> 1;
			const double2 *x = a + seq * pitch;
			const int k = j & (Ns - 1);
			const double v0 = comp(x[j], im);
			double v1, v2, v3;
			if(Ns == 1)
			{
				v1 = comp(x[j + q4], im);
				v2 = comp(x[j + 2 * q4], im);
				v3 = comp(x[j + 3 * q4], im);
			}
			else
			{
				const int m = k << sh;
				double2 w1 = tw[m];
				double2 w2 = tw[2 * m];                // 2 m < n/2
				const bool far = 3 * m >= half;
				double2 w3 = tw[far ? 3 * m - half : 3 * m];
				if(far) { w3.x = neg_if(w3.x, true); w3.y = neg_if(w3.y, true); }
				w1.y = neg_if(w1.y, sign > 0);
				w2.y = neg_if(w2.y, sign > 0);
				w3.y = neg_if(w3.y, sign > 0);
				v1 = cmul_comp(x[j + q4], w1, im);
				v2 = cmul_comp(x[j + 2 * q4], w2, im);
				v3 = cmul_comp(x[j + 3 * q4], w3, im);
			}
			const double t0 = v0 + v2, t1 = v0 - v2, t2 = v1 + v3, t3 = v1 - v3;
			// t3 times -i (forward: re = t3.im, im = -t3.re) or +i
			const double r3 = neg_if(other_comp(t3), im == (sign < 0));
			if(on)
			{
				double *y = reinterpret_cast<double *>(b + seq * pitch) + im;
				const int o = ((j - k) << 2) + k;
				y[2 * o] = t0 + t2;
				y[2 * (o + Ns)] = t1 + r3;
				y[2 * (o + 2 * Ns)] = t0 - t2;
				y[2 * (o + 3 * Ns)] = t1 - r3;
			}
		}
		__syncthreads();
		double2 *t = a; a = b; b = t;
	}
	return a;
}

// ------------------------------------------------------- other lengths
//
// Mixed-radix Stockham passes.  A pass of radix r after sub-transforms of
// length Ns writes
//   y[(j - k) r + k + p Ns] = sum_q x[j + q n/r] exp(sign 2 pi i q (k + p Ns) / (r Ns))
// for j < n/r, k = j mod Ns, p < r.  The FP32 form computes every output
// directly from its r inputs, the twiddle and the r-point DFT in one
// exponent read from the full table tw[m] = exp(-2 pi i m / n), m < n
// (conjugated for the inverse): O(n r) work per pass, so a length with a
// large prime factor transforms correctly but slowly.
template <typename C>
__device__ C *fft_smem_any(C *a, C *b, const FftPlan &pl, int nb, int pitch, int sign, const C *tw)
{
	const int n = pl.n;
	for(int ps = 0; ps < pl.npass; ps++)
	{
		const int r = pl.r[ps], Ns = pl.Ns[ps];
		const int m = n / r;                 // outputs per output digit p
		const int step0 = m / Ns;            // table stride of one unit of k + p Ns
		const int total = n * nb;
		for(int idx = threadIdx.x; idx < total; idx += blockDim.x)
		{
			const int seq = nb == 1 ? 0 : (int) bits::div_q((uint32_t) idx, pl.mul_n, pl.sh_n);
			const int o = idx - seq * n;
			const int p = (int) bits::div_q((uint32_t) o, pl.mul_m[ps], pl.sh_m[ps]), j = o - p * m;
			const int k = j - (int) bits::div_q((uint32_t) j, pl.mul_ns[ps], pl.sh_ns[ps]) * Ns;
			const C *x = a + (size_t) seq * pitch;
			const int step = (k + p * Ns) * step0;   // < n
			C acc = x[j];
			int t = 0;
			for(int q = 1; q < r; q++)
			{
				t += step;
				if(t >= n) t -= n;
				C w = tw[t];
				if(sign > 0) w.y = -w.y;
				acc = cadd(acc, cmul(x[j + q * m], w));
			}
			b[(size_t) seq * pitch + (j - k) * r + k + p * Ns] = acc;
		}
		__syncthreads();
		C *t = a; a = b; b = t;
	}
	return a;
}

// The FP64 form: radices 2 to 5 as butterflies (the inputs twiddled once,
// then the r-point DFT from its constants), two lanes per butterfly, one
// component each.  Per lane and output 4 to 5.2 FP64 instructions, where
// the direct sum takes 4 (r - 1).  Larger primes take the direct sum, one
// component of one output per lane.
__device__ inline double2 *fft_smem_any(double2 *a, double2 *b, const FftPlan &pl, int nb, int pitch,
		int sign, const double2 *tw)
{
	const int n = pl.n;
	const bool im = threadIdx.x & 1;
	// cos and sin of 2 pi / 3, 2 pi / 5 and 4 pi / 5
	const double s3 = 0.86602540378443864676;
	const double c51 = 0.30901699437494742410, c52 = -0.80901699437494742410;
	const double s51 = 0.95105651629515357212, s52 = 0.58778525229247312917;
	for(int ps = 0; ps < pl.npass; ps++)
	{
		const int r = pl.r[ps], Ns = pl.Ns[ps];
		const int m = n / r;
		const int step0 = m / Ns;
		const bool direct = r > 5;
		const int per = direct ? n : m;          // items per sequence (x 2 lanes)
		const int total = 2 * per * nb;
		for(int base = 0; base < total; base += blockDim.x)
		{
			const int idx = base + (int) threadIdx.x;
			const bool on = idx < total;
			const int i = (on ? idx : total - 1) >> 1;
			int seq = 0, o = i;
			if(nb > 1)
			{
				// i / per: per is n (direct) or m
				seq = direct ? (int) bits::div_q((uint32_t) i, pl.mul_n, pl.sh_n)
					: (int) bits::div_q((uint32_t) i, pl.mul_m[ps], pl.sh_m[ps]);
				o = i - seq * per;
			}
			const int p0 = direct ? (int) bits::div_q((uint32_t) o, pl.mul_m[ps], pl.sh_m[ps]) : 0;
			const int j = o - p0 * m;
			const int k = j - (int) bits::div_q((uint32_t) j, pl.mul_ns[ps], pl.sh_ns[ps]) * Ns;
			const double2 *x = a + (size_t) seq * pitch;
			double *y = reinterpret_cast<double *>(b + (size_t) seq * pitch) + im
				+ 2 * ((j - k) * r + k);
			const double v0 = comp(x[j], im);
			if(direct)
			{
				const int step = (k + p0 * Ns) * step0;
				double acc = v0;
				int t = 0;
				for(int q = 1; q < r; q++)
				{
					t += step;
					if(t >= n) t -= n;
					double2 w = tw[t];
					w.y = neg_if(w.y, sign > 0);
					acc += cmul_comp(x[j + q * m], w, im);
				}
				if(on) y[2 * p0 * Ns] = acc;
				continue;
			}
			double v[5];
			#pragma unroll
			for(int q = 1; q < 5; q++)
			{
				v[q] = 0.0;
				if(q < r)
				{
					double2 w = tw[q * k * step0];       // q k step0 < n
					w.y = neg_if(w.y, sign > 0);
					v[q] = Ns == 1 ? comp(x[j + q * m], im) : cmul_comp(x[j + q * m], w, im);
				}
			}
			// (i times u).re = -u.im, .im = u.re; sgn(im) turns a lane's other
			// component into its own of sign i u
			const bool flip = im == (sign < 0);
			if(r == 4)
			{
				const double t0 = v0 + v[2], t1 = v0 - v[2], t2 = v[1] + v[3], t3 = v[1] - v[3];
				const double r3 = neg_if(other_comp(t3), flip);
				if(on)
				{
					y[0] = t0 + t2;
					y[2 * Ns] = t1 + r3;
					y[4 * Ns] = t0 - t2;
					y[6 * Ns] = t1 - r3;
				}
			}
			else if(r == 2)
			{
				if(on)
				{
					y[0] = v0 + v[1];
					y[2 * Ns] = v0 - v[1];
				}
			}
			else if(r == 3)
			{
				const double t = v[1] + v[2], h = __fma_rn(-0.5, t, v0);
				const double u = neg_if(other_comp(v[1] - v[2]), flip);
				if(on)
				{
					y[0] = v0 + t;
					y[2 * Ns] = __fma_rn(s3, u, h);
					y[4 * Ns] = __fma_rn(-s3, u, h);
				}
			}
			else
			{
				const double t1 = v[1] + v[4], t2 = v[2] + v[3], t3 = v[1] - v[4], t4 = v[2] - v[3];
				const double h1 = __fma_rn(c52, t2, __fma_rn(c51, t1, v0));
				const double h2 = __fma_rn(c51, t2, __fma_rn(c52, t1, v0));
				const double u1 = neg_if(other_comp(__fma_rn(s52, t4, s51 * t3)), flip);
				const double u2 = neg_if(other_comp(__fma_rn(-s51, t4, s52 * t3)), flip);
				if(on)
				{
					y[0] = (v0 + t1) + t2;
					y[2 * Ns] = h1 + u1;
					y[4 * Ns] = h2 + u2;
					y[6 * Ns] = h2 - u2;
					y[8 * Ns] = h1 - u1;
				}
			}
		}
		__syncthreads();
		double2 *t = a; a = b; b = t;
	}
	return a;
}

// The transform of any length (pl its plan).
template <typename C>
__device__ __forceinline__ C *fft_any(C *a, C *b, const FftPlan &pl, int nb, int pitch, int sign,
		const C *tw)
{
	if(pl.npass == 0)
		return fft_smem(a, b, pl.n, pl.log2n, nb, pitch, sign, tw);
	return fft_smem_any(a, b, pl, nb, pitch, sign, tw);
}

// Twiddles of a transform, in elements: the half table of a power-of-two
// length, the full one otherwise.
__host__ __device__ inline int fft_tw_elems(const FftPlan &pl) { return pl.npass ? pl.n : pl.n >> 1; }

// Shared-memory copy of the twiddles (each pass reads them with scattered
// indices; from global memory the first touch of every line stalls its
// pass).  kept: whether the launch reserved room for it behind the
// buffers.  tw may be the table of a length 2^twsh times larger (then kept
// is set).  The copy is complete at the block's next barrier.
template <typename C>
__device__ __forceinline__ const C *fft_tw_stage(C *dst, const C *tw, int n, bool kept, int twsh = 0)
{
	if(!kept) return tw;
	for(int i = threadIdx.x; i < n; i += blockDim.x)
		dst[i] = tw[i << twsh];
	return dst;
}

// The FP64 form keeps scalings by powers of two out of its transforms (their
// multiplications were 5 % of the row kernels, which the FP64 pipe bounds):
// the half of the row split, and 1 / (nx ny) where that is one, are folded
// into the Green's function, exactly.  FP32 multiplies where it always did.
template <typename T>
inline double green_scale(int nx, int ny)
{
	if(sizeof(T) == 4) return 1.0;
	const bool pow2 = (nx & (nx - 1)) == 0 && (ny & (ny - 1)) == 0;
	return pow2 ? 0.5 / ((double) nx * (double) ny) : 0.5;
}

// The number of grid nodes, to divide by: N, 1 / N (rounded) and whether N is
// a power of two (then v * r is v / N exactly).
template <typename T>
struct NodeCount { T n, r; bool pow2; };

template <typename T>
inline NodeCount<T> node_count(int nx, int ny)
{
	NodeCount<T> c;
	c.n = (T) ((double) nx * (double) ny);
	c.r = (T) (1.0 / (double) c.n);
	c.pow2 = (nx & (nx - 1)) == 0 && (ny & (ny - 1)) == 0;
	return c;
}

__device__ __forceinline__ float over(float v, const NodeCount<float> &c)
{
	return c.pow2 ? v * c.r : v / c.n;
}
// FP64: by the reciprocal and one correction (bits::div_by), three FP64
// instructions where the division takes about ten
__device__ __forceinline__ double over(double v, const NodeCount<double> &c)
{
	return c.pow2 ? v * c.r : bits::div_by(v, c.n, c.r);
}

// phi from the inverse transform (green_scale may have divided already)
__device__ __forceinline__ float phi_of(float v, const NodeCount<float> &c) { return over(v, c); }
__device__ __forceinline__ double phi_of(double v, const NodeCount<double> &c)
{
	return c.pow2 ? v : bits::div_by(v, c.n, c.r);
}

// The kernels below are static: the FP64 units (built without FMA
// contraction) and the mixed and adjoint units (built with it) each get their
// own copy, so a launch always runs the device code of the unit that makes
// it, and a kernel attribute set in one unit leaves the other units' kernels
// alone.

// The two half spectra of a transformed row pair, FP64: twice them
// (green_scale).
__device__ __forceinline__ float half_of(float v) { return v * 0.5f; }
__device__ __forceinline__ double half_of(double v) { return v; }
template <typename C>
__device__ __forceinline__ void split_rows(const C *Z, int nx, int nh, C *spec, int r0, bool two)
{
	for(int k = threadIdx.x; k < nh; k += blockDim.x)
	{
		C p = Z[k];
		C q = Z[k == 0 ? 0 : nx - k];
		q.y = -q.y;                          // conj(Z[-k])
		C A, B;
		A.x = half_of(p.x + q.x);
		A.y = half_of(p.y + q.y);
		// (p - q) / (2i) = -i (p - q) / 2
		B.x = half_of(p.y - q.y);
		B.y = half_of(-(p.x - q.x));
		spec[(int64_t) r0 * nh + k] = A;
		if(two) spec[(int64_t) (r0 + 1) * nh + k] = B;
	}
}

// rho (fixed point, ny x nx) -> spec (ny x (nx/2+1)).  One block per row
// pair.  value = (double) acc * qinv - mean, where the mean (the k = 0
// mode, removed in FP64 before the FP32 transform of the mixed form, so
// that the transform's rounding scales with the fluctuations, not with the
// total charge) comes from the exact integer sum rsum, or is mean0 when
// rsum is null.  G(0,0) = 0 discards whatever is left of the mode, so mean0
// may be the charge the particles carry (the deposit's weight rounding
// leaves a residue of ~2^-17 of it).  FP64 form: no removal (as the
// reference).
// rho_lo (FP64 form, may be null): the remainder word at scale qinv_lo.
template <typename T>
static __global__ void k_rows_fwd(const __grid_constant__ FftPlan px, int ny, const long long *rho,
		double qinv, const long long *rsum, typename Cx<T>::t *spec, const typename Cx<T>::t *tw,
		const long long *rho_lo, double qinv_lo, double mean0, bool tw_sm, const NodeCount<double> N)
{
	typedef typename Cx<T>::t C;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int nx = px.n;
	C *a = reinterpret_cast<C *>(smem_raw);
	C *b = a + nx;
	tw = fft_tw_stage(b + nx, tw, fft_tw_elems(px), tw_sm);
	pdl_wait();
	int r0 = 2 * blockIdx.x;
	const bool two = r0 + 1 < ny;            // an odd ny leaves the last row alone
	int nh = nx / 2 + 1;
	const double m = rsum ? over((double) *rsum * qinv, N) : mean0;
	for(int i = threadIdx.x; i < nx; i += blockDim.x)
	{
		int64_t ia = (int64_t) r0 * nx + i, ib = (int64_t) (r0 + 1) * nx + i;
		double va, vb;
		if(rho_lo)
		{
			// both words' products are exact (power-of-two scales): one
			// rounding, in the sum
			va = __fma_rn((double) rho[ia], qinv, (double) rho_lo[ia] * qinv_lo);
			vb = two ? __fma_rn((double) rho[ib], qinv, (double) rho_lo[ib] * qinv_lo) : 0.0;
			if(m != 0.0) { va -= m; vb -= two ? m : 0.0; }
		}
		else
		{
			va = (double) rho[ia] * qinv - m;
			vb = two ? (double) rho[ib] * qinv - m : 0.0;
		}
		C z; z.x = (T) va; z.y = (T) vb;
		a[i] = z;
	}
	__syncthreads();
	const C *Z = fft_any<C>(a, b, px, 1, nx, -1, tw);
	split_rows(Z, nx, nh, spec, r0, two);
}

// The Green's function G(kx, ky) = 1 / (2 (cos(2 pi kx/nx) + cos(2 pi
// ky/ny)) - 4), G(0, 0) = 0 (solver.c:269-280), stored once per context in
// column order Gt[kx * ny + ky] (the order k_cols reads it), as type T.
// Evaluated in FP64 from the cosine tables, times scale (green_scale).
template <typename T>
static __global__ void k_green(int nx, int ny, const double *cosx, const double *cosy, T *Gt, double scale)
{
	int nh = nx / 2 + 1;
	int64_t total = (int64_t) nh * ny;
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < total;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		int kx = (int) (i / ny), row = (int) (i - (int64_t) kx * ny);
		double G = (kx == 0 && row == 0) ? 0.0 : scale / (2.0 * (cosx[kx] + cosy[row]) - 4.0);
		Gt[i] = (T) G;
	}
}

// Columns [c0, c0 + cb) of spec, cb of this block: FFT along y, multiply by
// green(column of the block, row), inverse FFT.
template <typename T, class G>
__device__ __forceinline__ void cols_body(const FftPlan &py, int nh, int cb, typename Cx<T>::t *spec,
		const typename Cx<T>::t *tw, int twsh, bool tw_sm, unsigned char *smem_raw, const G &green)
{
	typedef typename Cx<T>::t C;
	const int ny = py.n;
	const int c0 = blockIdx.x * cb;
	const int ncol = min(cb, nh - c0);
	const int pitch = fft_pitch(ny, cb);
	C *a = reinterpret_cast<C *>(smem_raw);
	C *b = a + (size_t) cb * pitch;
	tw = fft_tw_stage(b + (size_t) cb * pitch, tw, fft_tw_elems(py), tw_sm, twsh);
	pdl_wait();
	// element idx of the block's columns: row idx / ncol, column idx % ncol
	// (cb is 1, 2 or 4; a last block with fewer columns divides)
	const int lg = (ncol & (ncol - 1)) == 0 ? __ffs(ncol) - 1 : -1;
	for(int idx = threadIdx.x; idx < ncol * ny; idx += blockDim.x)
	{
		int row = lg >= 0 ? idx >> lg : idx / ncol, c = idx - row * ncol;
		a[c * pitch + row] = spec[(int64_t) row * nh + c0 + c];
	}
	__syncthreads();
	C *X = fft_any<C>(a, b, py, ncol, pitch, -1, tw);
	for(int c = 0; c < ncol; c++)
		for(int row = threadIdx.x; row < ny; row += blockDim.x)
		{
			const T gv = green(c, row);
			C v = X[c * pitch + row];
			v.x = v.x * gv;
			v.y = v.y * gv;
			X[c * pitch + row] = v;
		}
	__syncthreads();
	C *Y = (X == a) ? b : a;
	const C *R = fft_any<C>(X, Y, py, ncol, pitch, +1, tw);
	for(int idx = threadIdx.x; idx < ncol * ny; idx += blockDim.x)
	{
		int row = lg >= 0 ? idx >> lg : idx / ncol, c = idx - row * ncol;
		spec[(int64_t) row * nh + c0 + c] = R[c * pitch + row];
	}
}

// The columns with the tabulated Green's function (k_green).
template <typename T>
static __global__ void k_cols(const __grid_constant__ FftPlan py, int nh, int cb, typename Cx<T>::t *spec,
		const typename Cx<T>::t *tw, const T *Gt, bool tw_sm)
{
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const T *Gc = Gt + (size_t) blockIdx.x * cb * py.n;    // columns are contiguous
	const int ny = py.n;
	cols_body<T>(py, nh, cb, spec, tw, 0, tw_sm, smem_raw,
			[=](int c, int row) { return Gc[c * ny + row]; });
}

// spec -> phi (ny x nx real).  One block per row pair.
template <typename T>
static __global__ void k_rows_inv(const __grid_constant__ FftPlan px, int ny,
		const typename Cx<T>::t *spec, const typename Cx<T>::t *tw, T *phi, bool tw_sm,
		const NodeCount<T> N, int twsh)
{
	typedef typename Cx<T>::t C;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int nx = px.n;
	C *a = reinterpret_cast<C *>(smem_raw);
	C *b = a + nx;
	tw = fft_tw_stage(b + nx, tw, fft_tw_elems(px), tw_sm, twsh);
	pdl_wait();
	int r0 = 2 * blockIdx.x;
	const bool two = r0 + 1 < ny;            // an odd ny leaves the last row alone
	int nh = nx / 2 + 1;
	for(int k = threadIdx.x; k < nh; k += blockDim.x)
	{
		C A = spec[(int64_t) r0 * nh + k];
		C B;
		if(two) B = spec[(int64_t) (r0 + 1) * nh + k];
		else { B.x = (T) 0; B.y = (T) 0; }
		if(k == 0 || 2 * k == nx)
		{
			// c2r uses only the real part of the DC and Nyquist bins
			C y; y.x = A.x; y.y = B.x;
			a[k] = y;
		}
		else
		{
			C y;
			y.x = A.x - B.y; y.y = A.y + B.x;     // A + iB
			a[k] = y;
			y.x = A.x + B.y; y.y = B.x - A.y;     // conj(A) + i conj(B)
			a[nx - k] = y;
		}
	}
	__syncthreads();
	const C *Y = fft_any<C>(a, b, px, 1, nx, +1, tw);
	for(int i = threadIdx.x; i < nx; i += blockDim.x)
	{
		C v = Y[i];
		phi[(int64_t) r0 * nx + i] = phi_of(v.x, N);
		if(two) phi[(int64_t) (r0 + 1) * nx + i] = phi_of(v.y, N);
	}
}

// Real-valued input (ny x nx of T) -> spec, otherwise as k_rows_fwd.  Used
// by the adjoint, whose source term (rho-bar) is not a charge sum, and by
// the solve on the caller's own buffers.
template <typename T>
static __global__ void k_rows_fwd_real(const __grid_constant__ FftPlan px, int ny, const T *in,
		typename Cx<T>::t *spec, const typename Cx<T>::t *tw, bool tw_sm, int twsh)
{
	typedef typename Cx<T>::t C;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	const int nx = px.n;
	C *a = reinterpret_cast<C *>(smem_raw);
	C *b = a + nx;
	tw = fft_tw_stage(b + nx, tw, fft_tw_elems(px), tw_sm, twsh);
	pdl_wait();
	int r0 = 2 * blockIdx.x;
	const bool two = r0 + 1 < ny;
	int nh = nx / 2 + 1;
	for(int i = threadIdx.x; i < nx; i += blockDim.x)
	{
		C z;
		z.x = in[(int64_t) r0 * nx + i];
		z.y = two ? in[(int64_t) (r0 + 1) * nx + i] : (T) 0;
		a[i] = z;
	}
	__syncthreads();
	const C *Z = fft_any<C>(a, b, px, 1, nx, -1, tw);
	split_rows(Z, nx, nh, spec, r0, two);
}

// ----------------------------------------------------------------- launch

// Dynamic shared memory the solver's kernels may be given.
constexpr int kFftMaxSmem = 200 * 1024;

// Launch shape of a kernel that transforms nb sequences of pl.n per block.
struct FftShape { int nb, threads; size_t smem; bool tw_sm; };

template <typename T>
inline FftShape fft_shape(const FftPlan &pl, int nb)
{
	typedef typename Cx<T>::t C;
	FftShape s;
	s.nb = nb;
	// a butterfly (FP32: half of one; FP64: one lane of its two) per thread
	// and pass, 512 threads at most; the FP32 loads convert in FP64, which
	// wants the warps of twice the butterflies
	const int64_t want = (int64_t) pl.n * nb / (pl.npass && sizeof(T) == 4 ? 1 : 2);
	s.threads = (int) (want < 64 ? 64 : want > 512 ? 512 : (want + 31) / 32 * 32);
	s.smem = 2 * (size_t) nb * fft_pitch(pl.n, nb) * sizeof(C);
	const size_t tws = (size_t) fft_tw_elems(pl) * sizeof(C);
	s.tw_sm = s.smem + tws <= (size_t) kFftMaxSmem;
	if(s.tw_sm) s.smem += tws;
	return s;
}

// Columns per block.  FP64 (bound by the FP64 pipe): one column per block
// until there are two for every SM, then two (whole 32-byte sectors).  FP32
// (bound by latency): as many of 4, 2, 1 as leave every SM a block.  A
// 64 x 64 solve's columns took 45 us in blocks of 32 columns (two SMs
// busy), a 512 x 512 one's 62 us in blocks of 8.  Two buffers stay within
// 64 KB so that several blocks share an SM.
template <typename T>
inline int cols_per_block(int nh, int ny)
{
	typedef typename Cx<T>::t C;
	int cb = sizeof(T) == 8 ? (nh > 2 * 152 ? 2 : 1) : 4;
	while(cb > 1 && ((sizeof(T) == 4 && (nh + cb - 1) / cb < 152)
				|| 2 * (size_t) cb * ny * sizeof(C) > 64 * 1024))
		cb >>= 1;
	return cb;
}

// spec (half spectra of the rows) -> phi
template <typename T>
static void poisson_tail(int nx, int ny, const FftPlan &px, const FftPlan &py, const FftShape &rs,
		typename Cx<T>::t *spec, const typename Cx<T>::t *twx, const typename Cx<T>::t *twy,
		const T *Gt, T *phi, cudaStream_t s)
{
	const int nh = nx / 2 + 1;
	const FftShape cs = fft_shape<T>(py, cols_per_block<T>(nh, ny));
	launch_pdl(k_cols<T>, (nh + cs.nb - 1) / cs.nb, cs.threads, cs.smem, s, py, nh, cs.nb, spec, twy, Gt,
			cs.tw_sm);
	launch_pdl(k_rows_inv<T>, (ny + 1) / 2, rs.threads, rs.smem, s, px, ny, spec, twx, phi, rs.tw_sm,
			node_count<T>(nx, ny), 0);
}

// rho (fixed point) -> phi.  Gt: the tabulated Green's function (k_green).
template <typename T>
static void poisson_launch(const Grid &g, const long long *rho, double qinv, const long long *mean,
		typename Cx<T>::t *spec, const typename Cx<T>::t *twx, const typename Cx<T>::t *twy,
		T *phi, cudaStream_t s, const T *Gt, const long long *rho_lo = nullptr, double qinv_lo = 0.0,
		double mean0 = 0.0)
{
	const FftPlan px = fft_plan(g.nx), py = fft_plan(g.ny);
	const FftShape rs = fft_shape<T>(px, 1);
	launch_pdl(k_rows_fwd<T>, (g.ny + 1) / 2, rs.threads, rs.smem, s, px, g.ny, rho, qinv, mean, spec, twx,
			rho_lo, qinv_lo, mean0, rs.tw_sm, node_count<double>(g.nx, g.ny));
	poisson_tail<T>(g.nx, g.ny, px, py, rs, spec, twx, twy, Gt, phi, s);
}

// out = IFFT(G FFT(in)) / (nx ny) for a real ny x nx input: the same linear
// operator as poisson_launch (symmetric, so it is also its own adjoint).
template <typename T>
static void poisson_launch_real(int nx, int ny, const T *in, typename Cx<T>::t *spec,
		const typename Cx<T>::t *twx, const typename Cx<T>::t *twy, const T *Gt, T *out,
		cudaStream_t s)
{
	const FftPlan px = fft_plan(nx), py = fft_plan(ny);
	const FftShape rs = fft_shape<T>(px, 1);
	launch_pdl(k_rows_fwd_real<T>, (ny + 1) / 2, rs.threads, rs.smem, s, px, ny, in, spec, twx, rs.tw_sm,
			0);
	poisson_tail<T>(nx, ny, px, py, rs, spec, twx, twy, Gt, out, s);
}

} // namespace cpic
