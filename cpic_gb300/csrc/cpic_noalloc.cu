// cpic_noalloc.cu -- an FP64 periodic Poisson solve that allocates nothing.
//
// Some callers cannot allocate device memory: applications that have
// reserved the whole device up front for their own pool or run under a fixed
// memory budget, and latency-critical host threads on which cudaMalloc or
// cudaFree (which may synchronise the device) must not appear.  For them,
// cpic_poisson_noalloc solves the same periodic Poisson problem as the
// context's field stage (the MFT solve of the reference, solver.c:465-509)
// with every piece of scratch -- the half spectrum and the FFT twiddles, whose
// real parts are the Green's-function cosines -- in one file-scope __device__
// array of fixed size.  The caller passes its own input and output device buffers.
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
// layout: [spectrum kSpecElems double2][twiddles kMaxN/2 double2]
constexpr size_t kScratchBytes = (kSpecElems + kMaxN / 2) * sizeof(double2);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
static void *g_scratch_addr[kMaxDevices];
static bool g_tables_ready[kMaxDevices];
static std::mutex g_setup_lock;

// Twiddles exp(-2 pi i k / kMaxN), computed on the device (sincospi:
// correctly scaled, ~1 ulp).  A transform of any smaller power of two reads
// them with a stride, so one table, filled once per device, serves every
// grid (filling tables of the call's own sizes took 9 us of every call).
__global__ void k_noalloc_table(double2 *tw)
{
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if(k < kMaxN / 2)
	{
		double s, c;
		sincospi(-2.0 * k / kMaxN, &s, &c);
		tw[k] = make_double2(c, s);
	}
}

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

// Device address of the scratch array for the current device, looked up
// once per device, together with the kernels' shared-memory limits (a
// kernel attribute belongs to the device it was set on) and the twiddle
// table, filled on the caller's stream: later calls are ordered behind it,
// since calls that overlap on the GPU are the caller's to serialise.  A
// device is marked ready only when every step succeeded, so a failed set-up
// is retried by the next call; a table launch that was only recorded into a
// graph does not count.  *first: this call launched the table.
static int scratch_for_current_device(void **out, cudaStream_t s, bool *first)
{
	*first = false;
	int dev = -1;
	if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
		return CPIC_ENODEV;
	std::lock_guard<std::mutex> lk(g_setup_lock);
	if(!g_scratch_addr[dev])
	{
		void *p = nullptr;
		cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
		if(e == cudaSuccess && !p)
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
		g_scratch_addr[dev] = p;
	}
	if(!g_tables_ready[dev])
	{
		*first = true;
		cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
		double2 *tw = (double2 *) g_scratch_addr[dev] + kSpecElems;
		void *argv[] = {&tw};
		cudaError_t e = cudaLaunchKernel((const void *) k_noalloc_table, dim3(1), dim3(kMaxN / 2), argv,
				0, s);
		if(e == cudaSuccess)
			e = cudaStreamIsCapturing(s, &cap);
		if(e != cudaSuccess)
		{
			fprintf(stderr, "cpic_poisson_noalloc: set-up on device %d failed: %s\n", dev,
					cudaGetErrorString(e));
			return CPIC_ECUDA;
		}
		g_tables_ready[dev] = cap == cudaStreamCaptureStatusNone;
	}
	*out = g_scratch_addr[dev];
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
	void *base = nullptr;
	cudaStream_t s = (cudaStream_t) stream;
	bool first;                     // the table was launched by this call
	int r = scratch_for_current_device(&base, s, &first);
	if(r) return r;
	double2 *spec = (double2 *) base;
	const double2 *tw = spec + kSpecElems;
	const int nxi = (int) nx, nyi = (int) ny, nh = nxi / 2 + 1;
	const FftPlan px = fft_plan(nxi), py = fft_plan(nyi);
	const FftShape rs = fft_shape<double>(px, 1), cs = fft_shape<double>(py, 1);
	const int sx = kLog2MaxN - px.log2n;

	// one column per block, at most 257 of them
	// (each launch reports its own error, not an earlier one left pending on
	// the thread).  All three are dependent launches: the first waits on the
	// device for whatever the caller has queued.  In a capture, where its
	// predecessors may be any nodes, and behind the table's launch, whose
	// result it reads early, the first one is an ordinary launch.
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
	cudaError_t e = first ? cudaSuccess : cudaStreamIsCapturing(s, &cap);
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
