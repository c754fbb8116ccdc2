// cpic_noalloc.cu -- an FP64 periodic Poisson solve that allocates nothing.
//
// Some callers cannot allocate device memory: applications that have
// reserved the whole device up front for their own pool or run under a fixed
// memory budget, and latency-critical host threads on which cudaMalloc or
// cudaFree (which may synchronise the device) must not appear.  For them,
// cpic_poisson_noalloc solves the same periodic Poisson problem as the
// context's field stage (the MFT solve of the reference, solver.c:465-509)
// with its scratch, the half spectrum, in a file-scope __device__ array of fixed
// size.  The caller passes its own input and output device buffers.
//
// The array is held by every GPU that loads this library until the process
// exits (about 2.1 MB).  In host code the symbol is only a host-side
// stand-in, never a device address: its device address is obtained once per
// device with cudaGetSymbolAddress, on the first call made with that device
// current, and passed to the kernels.  All calls share the array and it keeps
// the last call's contents; each call rewrites everything it reads before
// reading it, so nothing carries over.  Calls that overlap on the GPU (for
// example from two streams at once) race on the array and must be
// serialised by the caller.
//
// The FFT twiddles, whose real parts are the Green's-function cosines, are
// constant data of the library, computed by the compiler, and never written
// (a kernel that filled tables of the call's own sizes took 9 us of every call).
#include <cmath>
#include <cstdio>
#include <mutex>

#include "../../include/cpic_gpu.h"
#include "cpic_common.cuh"
#include "cpic_fft.cuh"

namespace {

using namespace cpic;

constexpr int kMaxN = CPIC_NOALLOC_MAX_N;            // nx, ny <= kMaxN
constexpr int kLog2MaxN = 9;
static_assert(1 << kLog2MaxN == kMaxN, "");
constexpr size_t kSpecElems = (size_t) kMaxN * (kMaxN / 2 + 1);

static __device__ __align__(256) double2 g_noalloc_spec[kSpecElems];

// Pairs of doubles hi + lo for the twiddles: products by Dekker's splitting,
// sums by Knuth's two-sum, so that a sum of the power series is good to ~100 bits
// and its hi part is the correctly rounded value.
struct Pair { double hi, lo; };

constexpr Pair two_sum(double a, double b)
{
	const double s = a + b, t = s - a;
	return {s, (a - (s - t)) + (b - t)};
}

constexpr Pair add(Pair a, Pair b)
{
	const Pair s = two_sum(a.hi, b.hi);
	return two_sum(s.hi, s.lo + (a.lo + b.lo));
}

constexpr Pair mul(Pair a, Pair b)
{
	const double split = 134217729.0;              // 2^27 + 1
	const double ah = split * a.hi - (split * a.hi - a.hi), al = a.hi - ah;
	const double bh = split * b.hi - (split * b.hi - b.hi), bl = b.hi - bh;
	const double p = a.hi * b.hi;
	const double e = ((ah * bh - p) + ah * bl + al * bh) + al * bl;
	return two_sum(p, e + (a.hi * b.lo + a.lo * b.hi));
}

// 1/d to two doubles' precision (d a small whole number)
constexpr Pair recip(double d)
{
	const double q = 1.0 / d;
	const Pair r = mul({-q, 0.0}, {d, 0.0});
	return two_sum(q, ((1.0 + r.hi) + r.lo) / d);
}

// sin (odd) or cos (even) of t <= pi/4 by its power series
constexpr double series(Pair t, bool odd)
{
	const Pair t2 = mul({-t.hi, -t.lo}, t);        // -t^2
	Pair sum = {1.0, 0.0};
	for(int k = 2 * 14; k >= 2; k -= 2)            // terms beyond t^28 are below 2^-106
	{
		const double d = odd ? k * (k + 1.0) : k * (k - 1.0);
		sum = add({1.0, 0.0}, mul(mul(t2, recip(d)), sum));
	}
	return odd ? mul(t, sum).hi : sum.hi;
}

// exp(-2 pi i k / kMaxN), 0 <= k < kMaxN / 2.  A transform of any smaller
// power of two reads the table with a stride.
struct Twiddles { double2 v[kMaxN / 2]; };

constexpr Twiddles make_twiddles()
{
	constexpr int q = kMaxN / 4;                   // a quarter turn
	const Pair step = mul({3.141592653589793, 1.2246467991473532e-16}, {2.0 / kMaxN, 0.0});
	Twiddles t = {};
	for(int m = 0; m <= q / 2; m++)
	{
		const Pair a = mul(step, {(double) m, 0.0});
		const double c = series(a, false), s = m ? series(a, true) : 0.0;
		t.v[m].x = c;
		t.v[m].y = -s;
		t.v[m + q].x = -s;
		t.v[m + q].y = -c;
		if(m > 0)
		{
			t.v[q - m].x = s;
			t.v[q - m].y = -c;
			t.v[2 * q - m].x = -c;
			t.v[2 * q - m].y = -s;
		}
	}
	t.v[0].y = 0.0;
	t.v[q].x = 0.0;
	return t;
}

static __device__ const Twiddles g_noalloc_twiddles = make_twiddles();

constexpr int kMaxDevices = 64;
struct Scratch { double2 *spec; const double2 *tw; };
static Scratch g_scratch[kMaxDevices];
static std::mutex g_setup_lock;

// cos(2 pi j / n), 0 <= j < n, from the table
__device__ __forceinline__ double cos_of(const double2 *tw, int j, int log2n)
{
	const int m = j << (kLog2MaxN - log2n);
	return m < kMaxN / 2 ? tw[m].x : -tw[m - kMaxN / 2].x;
}

// The columns with the Green's function evaluated here (no room for its
// table): G(kx, ky) is even in ky, so each block divides for half of its
// rows, into shared memory behind the transform's buffers.
__global__ void k_noalloc_cols(const __grid_constant__ FftPlan py, int nh, int log2nx, double2 *spec,
		const double2 *tw, size_t buf_bytes, double scale)
{
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double *gs = reinterpret_cast<double *>(smem_raw + buf_bytes);
	const int kx = blockIdx.x, ny = py.n;
	const double cx = cos_of(tw, kx, log2nx);
	for(int row = threadIdx.x; row <= ny / 2; row += blockDim.x)
		gs[row] = (kx == 0 && row == 0) ? 0.0 : scale / (2.0 * (cx + cos_of(tw, row, py.log2n)) - 4.0);
	cols_body<double>(py, nh, 1, spec, tw, kLog2MaxN - py.log2n, true, smem_raw,
			[=](int, int row) { return gs[2 * row <= ny ? row : ny - row]; });
}

// Device addresses of the scratch array and the twiddles for the current
// device, looked up once per device, together with the kernels' shared-memory
// limits (a kernel attribute belongs to the device it was set on).  A device is
// marked ready only when every step succeeded, so a failed set-up is retried by
// the next call.
static int scratch_for_current_device(Scratch *out)
{
	int dev = -1;
	if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
		return CPIC_ENODEV;
	std::lock_guard<std::mutex> lk(g_setup_lock);
	if(!g_scratch[dev].spec)
	{
		void *p = nullptr, *tw = nullptr;
		cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_spec);
		if(e == cudaSuccess)
			e = cudaGetSymbolAddress(&tw, g_noalloc_twiddles);
		if(e == cudaSuccess && (!p || !tw))
			e = cudaErrorInvalidSymbol;
		if(e == cudaSuccess)
			e = set_max_dyn_smem({(const void *) k_rows_fwd_real<double>,
					(const void *) k_noalloc_cols, (const void *) k_rows_inv<double>}, 64 * 1024);
		if(e != cudaSuccess)
		{
			fprintf(stderr, "cpic_poisson_noalloc: set-up on device %d failed: %s\n", dev,
					cudaGetErrorString(e));
			return CPIC_ECUDA;
		}
		g_scratch[dev] = {(double2 *) p, (const double2 *) tw};
	}
	*out = g_scratch[dev];
	return CPIC_OK;
}

} // namespace

extern "C" CPIC_API int
cpic_poisson_noalloc(const double *rho, double *phi, int64_t nx, int64_t ny, void *stream)
{
	if(!rho || !phi) return CPIC_EINVAL;
	if(nx < 4 || ny < 4 || (nx & (nx - 1)) || (ny & (ny - 1)))
		return CPIC_EINVAL;
	if(nx > kMaxN || ny > kMaxN)
	{
		fprintf(stderr, "cpic_poisson_noalloc: grid %lldx%lld exceeds the %dx%d maximum of the "
				"built-in scratch array\n", (long long) nx, (long long) ny, kMaxN, kMaxN);
		return CPIC_EINVAL;
	}
	Scratch sc;
	cudaStream_t s = (cudaStream_t) stream;
	int r = scratch_for_current_device(&sc);
	if(r) return r;
	double2 *spec = sc.spec;
	const double2 *tw = sc.tw;
	const int nxi = (int) nx, nyi = (int) ny, nh = nxi / 2 + 1;
	const FftPlan px = fft_plan(nxi), py = fft_plan(nyi);
	const FftShape rs = fft_shape<double>(px, 1), cs = fft_shape<double>(py, 1);
	const int sx = kLog2MaxN - px.log2n;

	// one column per block, at most 257 of them
	// (each launch reports its own error, not an earlier one left pending on
	// the thread).  All three are dependent launches: the first waits on the
	// device for whatever the caller has queued.  In a capture, where its
	// predecessors may be any nodes, the first one is an ordinary launch.
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
	cudaError_t e = cudaStreamIsCapturing(s, &cap);
	if(e == cudaSuccess)
	{
		if(cap == cudaStreamCaptureStatusNone)
			e = launch_pdl(k_rows_fwd_real<double>, nyi / 2, rs.threads, rs.smem, s, px, nyi, rho, spec, tw,
					true, sx);
		else
		{
			double2 *spec0 = spec;
			bool kept = true;
			int nyarg = nyi, sharg = sx;
			FftPlan pxarg = px;
			void *argv[] = {&pxarg, &nyarg, (void *) &rho, &spec0, (void *) &tw, &kept, &sharg};
			e = cudaLaunchKernel((const void *) k_rows_fwd_real<double>, dim3(nyi / 2), dim3(rs.threads),
					argv, rs.smem, s);
		}
	}
	if(e == cudaSuccess)
		e = launch_pdl(k_noalloc_cols, nh, cs.threads, cs.smem + (nyi / 2 + 1) * sizeof(double), s, py, nh,
				px.log2n, spec, tw, cs.smem, green_scale<double>(nxi, nyi));
	if(e == cudaSuccess)
		e = launch_pdl(k_rows_inv<double>, nyi / 2, rs.threads, rs.smem, s, px, nyi, spec, tw, phi, true,
				node_count<double>(nxi, nyi), sx);
	if(e != cudaSuccess)
	{
		fprintf(stderr, "cpic_poisson_noalloc: launch failed: %s\n", cudaGetErrorString(e));
		return CPIC_ECUDA;
	}
	return CPIC_OK;
}
