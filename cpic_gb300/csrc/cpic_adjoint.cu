// cpic_adjoint.cu -- differentiable run of the step and its hand-written
// adjoint: d(final field energy) / d(initial positions and velocities).
//
// Forward step j (j = 0 .. nsteps-1), the reference's order (sim.c:481-581):
//   rho_j = D(p_j)                 CIC deposit, -q/e0 per unit weight
//                                  (interpolate.c:282-346)
//   E_j   = -grad_h P rho_j        periodic FFT Poisson (solver.c:465-509)
//                                  and central differences (field.c:358-416)
//   e_i   = I(p_i; E_j)            CIC gather (interpolate.c:349-404)
//   u    <- M (u + h e) + h e      Boris for B along z, h = q dt'/(2m),
//                                  dt' = -dt/2 at j = 0 (mover.c:15-226)
//   p    <- wrap(p + dt u)         no move at j = 0 (mover.c:204-213)
// Loss: L = 1/2 e0 dx dy sum |E(D(p_N))|^2.
//
// Reverse step j, given the adjoints pb = dL/dp_{j+1} (without the deposit
// term of step j+1) and ub = dL/du_{j+1}:
//   pb   += c grad D(p_{j+1})^T rhob_{j+1}     (deposit adjoint = gather of
//                                                the weight gradients)
//   ut    = ub + move dt pb
//   vb    = M^T ut ;  eb = h (ut + vb) ;  ub = vb
//   pb   += grad I(p_j; E_j)^T eb              (gather's position term)
//   Eb_j  = sum_i w(p_j) eb_i                  (gather adjoint = deposit)
//   rhob_j = P^T (-grad_h)^T Eb_j = P div_h Eb_j
// and finally pb_0 += c grad D(p_0)^T rhob_0.  Only positions p_j and the
// grids E_j of a segment are needed in reverse (the kick is linear in u),
// so a segment of K steps is recomputed from its checkpoint (p, u) storing
// p_j and E_j, then swept backwards.
//
// Sums over particles into grids are 64-bit fixed point (integer atomics,
// order independent, deterministic).  The adjoint deposit's scale comes
// from a bound on |eb| computed on the device from the previous step's
// maxima, so it can never wrap.
//
// Particles are kept sorted by tile of cells: sorted at the start and again
// at segment starts at least kSortSteps steps apart, each order with the
// permutation that leads back to the one before (an "epoch"), along which the
// adjoints travel in the reverse sweep.  A block takes up to a few thousand
// particles of one tile and sums their deposits in shared memory over the tile
// and a margin, adding to the grid once per node: unsorted, 4 to 8 global
// 64-bit atomics per particle (50 to 90 per ns) bounded the FP32 kernels (262,144
// particles, 64 x 64: 20 us forward, 39 us reverse) and, with the FP64 pipe,
// the FP64 ones (1,048,576 particles, 128 x 128: 116 and 189 us).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <utility>
#include <vector>

#include "../../include/cpic_gpu.h"
#include "cpic_common.cuh"
#include "cpic_fft.cuh"

namespace cpic {
namespace adj {

struct AGrid {
	int nx, ny;
	double dx, dy, idx, idy, Lx, Ly;
	bits::Pos idx_p, idy_p;
	// tiles of ts x ts cells (ts a power of two, at most nx and ny) and the
	// deposit region of a block's tile: ts + 2 margin + 1 nodes a side
	int lts, ntx, margin, W;
};

// Boris kick of one iteration: u' = M (u + h e) + h e, M = [[a, s], [-s, a]]
// with t = Bz h, s = 2t / (1 + t^2), a = 1 - s t.
struct Kick {
	double h, t, s, a;
	int move;
	int turns;                   // t != 0
};

// Maxima as double bit patterns.  u, p: of the outputs of the reverse steps,
// by the parity of the step; r: of rhob.
struct Scale {
	unsigned long long u[2], p[2], r;
	int eexp;                    // the adjoint deposit's fixed-point scale 2^eexp
};

// The particles a block takes: [first, end) of the sorted order, all of tile
// `tile` (-1: none).
struct Work { int64_t first, end; int tile, pad; };

constexpr int kThreads = 256;
constexpr int kSortSteps = 8;    // least number of steps between two sorts
constexpr int kMargin = 6;       // cells a particle may drift before its
                                 // deposit goes straight to the grid

// CIC cell and fractions of a position in [0, L]; x == L maps to node 0.
template <typename T>
__device__ __forceinline__ void cell(const AGrid &g, T x, T y, int &ix, int &iy, int &ix1, int &iy1,
		T &fx, T &fy)
{
	T gx = x * (T) g.idx, gy = y * (T) g.idy;
	T flx = floor(gx), fly = floor(gy);
	fx = gx - flx;
	fy = gy - fly;
	// powers of two: the mask wraps x == L to node 0 and keeps every
	// index in range whatever the position
	ix = (int) flx & (g.nx - 1);
	iy = (int) fly & (g.ny - 1);
	ix1 = (ix + 1) & (g.nx - 1);
	iy1 = (iy + 1) & (g.ny - 1);
}

// The FP64 form's cell on the integer pipe (cpic_bits.h); false where it is
// not handled there (cell() then).
__device__ __forceinline__ bool cell_fast(const AGrid &g, double x, double y, int &ix, int &iy,
		bits::Pos &fx, bits::Pos &fy)
{
	bits::Pos px, py;
	bool ok = bits::pos_of(x, px) & bits::pos_of(y, py);
	ok &= bits::pos_frac(px, g.idx_p, ix, fx);
	ok &= bits::pos_frac(py, g.idy_p, iy, fy);
	ok &= bits::pos_normal(fx) & bits::pos_normal(fy);
	ix &= g.nx - 1;
	iy &= g.ny - 1;
	return ok;
}

__device__ __forceinline__ void red_add(unsigned long long *a, long long v)
{
	atomicAdd(a, (unsigned long long) v);
}

// |v| as ordered bits (of the value as a double)
__device__ __forceinline__ unsigned long long abs_bits(double v)
{
	return bits::to_bits(v) & 0x7fffffffffffffffull;
}

// Block-wide maximum of m into *out, one atomic per block.
__device__ __forceinline__ void block_max(unsigned long long m, unsigned long long *out,
		unsigned long long *sh)
{
	for(int o = 16; o > 0; o >>= 1)
	{
		const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
		m = v > m ? v : m;
	}
	if((threadIdx.x & 31) == 0)
		sh[threadIdx.x >> 5] = m;
	__syncthreads();
	if(threadIdx.x == 0)
	{
		for(int w = 1; w < (int) (blockDim.x >> 5); w++)
			m = sh[w] > m ? sh[w] : m;
		if(m) atomicMax(out, m);
	}
	__syncthreads();
}

// ------------------------------------------------------- order by tile

template <typename T>
__device__ __forceinline__ int tile_of(const AGrid &g, T x, T y)
{
	const int ix = (int) floor(x * (T) g.idx) & (g.nx - 1), iy = (int) floor(y * (T) g.idy) & (g.ny - 1);
	return (iy >> g.lts) * g.ntx + (ix >> g.lts);
}

// Blocks take contiguous ranges of the particles and count, and place, in
// shared memory, with one global atomic per block and tile (straight to the
// few hundred global counters, a million particles took 215 us to count
// and 225 us to place).  More tiles than kShTiles: the global counters.
constexpr int kShTiles = 4096;

__device__ __forceinline__ void block_range(int64_t n, int64_t &lo, int64_t &hi)
{
	const int64_t per = (n + gridDim.x - 1) / gridDim.x;
	lo = min(n, (int64_t) blockIdx.x * per);
	hi = min(n, lo + per);
}

// Counts the block's range into cnt (in shared or global memory).
template <typename T>
__device__ __forceinline__ void count_range(const AGrid &g, int64_t lo, int64_t hi, const T *x,
		const T *y, int32_t *cnt)
{
	for(int64_t i0 = lo; i0 < hi; i0 += blockDim.x)
	{
		const int64_t i = i0 + threadIdx.x;
		const bool on = i < hi;
		warp_reserve(cnt, on, on ? tile_of<T>(g, x[i], y[i]) : 0);
	}
}

template <typename T>
__global__ void k_tile_count(AGrid g, int64_t n, const T *x, const T *y, int nt, int32_t *cnt)
{
	__shared__ int32_t sh[kShTiles];
	int64_t lo, hi;
	block_range(n, lo, hi);
	if(nt > kShTiles)
	{
		count_range<T>(g, lo, hi, x, y, cnt);
		return;
	}
	for(int t = threadIdx.x; t < nt; t += blockDim.x) sh[t] = 0;
	__syncthreads();
	count_range<T>(g, lo, hi, x, y, sh);
	__syncthreads();
	for(int t = threadIdx.x; t < nt; t += blockDim.x)
		if(sh[t]) atomicAdd(&cnt[t], sh[t]);
}

// One block: first particle of each tile (into cnt, as cursors; counts and
// cursors are unsigned) and the blocks' work list, `chunk` particles each.
// nwork entries, at least n / chunk + the number of tiles.
__global__ void __launch_bounds__(1024) k_tile_scan(int nt, int chunk, int32_t *cnt, Work *work, int nwork)
{
	__shared__ int64_t s_p[32];
	__shared__ int32_t s_w[32];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int per = (nt + 1023) / 1024, t0 = min(tid * per, nt), t1 = min(t0 + per, nt);
	int64_t np = 0;
	int nw = 0;
	for(int t = t0; t < t1; t++)
	{
		const uint32_t c = (uint32_t) cnt[t];
		np += c;
		nw += (int) (((int64_t) c + chunk - 1) / chunk);
	}
	int64_t ip = np;
	int iw = nw;
	for(int o = 1; o < 32; o <<= 1)
	{
		const int64_t a = __shfl_up_sync(0xffffffffu, ip, o);
		const int b = __shfl_up_sync(0xffffffffu, iw, o);
		if(lane >= o) { ip += a; iw += b; }
	}
	if(lane == 31) { s_p[warp] = ip; s_w[warp] = iw; }
	__syncthreads();
	int64_t bp = ip - np;
	int bw = iw - nw, tw = 0;
	for(int w = 0; w < 32; w++)
	{
		if(w < warp) { bp += s_p[w]; bw += s_w[w]; }
		tw += s_w[w];
	}
	for(int t = t0; t < t1; t++)
	{
		const int64_t c = (uint32_t) cnt[t];
		cnt[t] = (int32_t) (uint32_t) bp;
		for(int64_t f = 0; f < c; f += chunk)
			if(bw < nwork)
				work[bw++] = Work{bp + f, bp + min(c, f + chunk), t, 0};
		bp += c;
	}
	for(int w = tw + tid; w < nwork; w += 1024)
		work[w] = Work{0, 0, -1, 0};
}

// Places every particle at its tile's cursor; src[k]: where particle k of the
// new order was.
template <typename T>
__global__ void k_tile_place(AGrid g, int64_t n, const T *x, const T *y, const T *ux, const T *uy,
		T *ox, T *oy, T *oux, T *ouy, int nt, int32_t *cursor, uint32_t *src)
{
	__shared__ int32_t sh[kShTiles];
	int64_t lo, hi;
	block_range(n, lo, hi);
	int32_t *cur = cursor;
	if(nt <= kShTiles)
	{
		for(int t = threadIdx.x; t < nt; t += blockDim.x) sh[t] = 0;
		__syncthreads();
		count_range<T>(g, lo, hi, x, y, sh);
		__syncthreads();
		for(int t = threadIdx.x; t < nt; t += blockDim.x)
			if(sh[t]) sh[t] = atomicAdd(&cursor[t], sh[t]);
		__syncthreads();
		cur = sh;
	}
	for(int64_t i0 = lo; i0 < hi; i0 += blockDim.x)
	{
		const int64_t i = i0 + threadIdx.x;
		const bool on = i < hi;
		const uint32_t k = (uint32_t) warp_reserve(cur, on, on ? tile_of<T>(g, x[i], y[i]) : 0);
		if(on && k < n)
		{
			ox[k] = x[i]; oy[k] = y[i]; oux[k] = ux[i]; ouy[k] = uy[i];
			src[k] = (uint32_t) i;
		}
	}
}

// out[src[k]] = in[k] for the four adjoints: back to the order before.
template <typename T>
__global__ void k_unsort(int64_t n, const uint32_t *src, const T *a, const T *b, const T *c, const T *d,
		T *oa, T *ob, T *oc, T *od)
{
	for(int64_t k = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; k < n;
			k += (int64_t) gridDim.x * blockDim.x)
	{
		const uint32_t i = src[k];
		oa[i] = a[k]; ob[i] = b[k]; oc[i] = c[k]; od[i] = d[k];
	}
}

// ------------------------------------------- deposit region of a block

// Sums over a block's region in shared memory: `planes` pairs of W x W 32-bit
// planes (low and high words, add64_low).
struct Region {
	uint32_t *sm;
	int x0, y0;                  // the tile's first cell less the margin

	__device__ __forceinline__ void open(const AGrid &g, uint32_t *mem, int tile, int comps)
	{
		sm = mem;
		const int ty = tile / g.ntx, tx = tile - ty * g.ntx;
		x0 = (tx << g.lts) - g.margin;
		y0 = (ty << g.lts) - g.margin;
		for(int i = threadIdx.x; i < 2 * comps * g.W * g.W; i += blockDim.x)
			sm[i] = 0;
	}

	// region node of cell (ix, iy), or -1 outside (or for a cell that the
	// periodic wrap would give a second place)
	__device__ __forceinline__ int node(const AGrid &g, int ix, int iy) const
	{
		const int hx = g.nx >> 1, hy = g.ny >> 1;
		const int lx = ((ix - x0 - g.margin + hx) & (g.nx - 1)) - hx + g.margin;
		const int ly = ((iy - y0 - g.margin + hy) & (g.ny - 1)) - hy + g.margin;
		return (unsigned) lx < (unsigned) (g.W - 1) && (unsigned) ly < (unsigned) (g.W - 1)
			? ly * g.W + lx : -1;
	}

	// the four nodes of a cell: v in the order 00, 10, 01, 11
	__device__ __forceinline__ void add(const AGrid &g, int comp, int node, int ix, int iy,
			const long long v[4], unsigned long long *grid)
	{
		if(node >= 0)
		{
			uint32_t *lo = sm + 2 * comp * g.W * g.W + node, *hi = lo + g.W * g.W;
			const int at[4] = {0, 1, g.W, g.W + 1};
			uint32_t h[4];
			#pragma unroll
			for(int c = 0; c < 4; c++) h[c] = add64_low(lo + at[c], v[c]);
			#pragma unroll
			for(int c = 0; c < 4; c++) atomicAdd(hi + at[c], h[c]);
		}
		else
		{
			const int ix1 = (ix + 1) & (g.nx - 1), iy1 = (iy + 1) & (g.ny - 1);
			red_add(grid + (int64_t) iy * g.nx + ix, v[0]);
			red_add(grid + (int64_t) iy * g.nx + ix1, v[1]);
			red_add(grid + (int64_t) iy1 * g.nx + ix, v[2]);
			red_add(grid + (int64_t) iy1 * g.nx + ix1, v[3]);
		}
	}

	// after a block barrier: the sums of one component onto the grid; returns
	// this thread's share of their total
	__device__ __forceinline__ long long flush(const AGrid &g, int comp, unsigned long long *grid) const
	{
		const uint32_t *lo = sm + 2 * comp * g.W * g.W, *hi = lo + g.W * g.W;
		long long sum = 0;
		for(int i = threadIdx.x; i < g.W * g.W; i += blockDim.x)
		{
			const long long v = (long long) ((uint64_t) hi[i] << 32 | lo[i]);
			if(v != 0)
			{
				const int ly = i / g.W, lx = i - ly * g.W;
				red_add(grid + (int64_t) ((y0 + ly) & (g.ny - 1)) * g.nx + ((x0 + lx) & (g.nx - 1)), v);
				sum += v;
			}
		}
		return sum;
	}
};

// ---------------------------------------------------------------- forward

// The charge deposit's fixed-point factor: the value, and its magnitude and
// sign for the integer path.
struct Charge {
	double q;
	bits::Pos p;
	int neg, fast;
};

// The four fixed-point deposit values rn(w qfix) of a position (order 00, 10,
// 01, 11) on FP64 instructions.  Out of line: the integer path below takes
// nearly every particle.
struct Slow4 { long long v[4]; int ix, iy; };
template <typename T>
static __device__ __noinline__ Slow4 deposit_slow(const AGrid &g, T x, T y, double qfix)
{
	Slow4 o;
	int ix1, iy1;
	T fx, fy;
	cell<T>(g, x, y, o.ix, o.iy, ix1, iy1, fx, fy);
	double w00 = (double) ((1 - fx) * (1 - fy)), w10 = (double) (fx * (1 - fy));
	double w01 = (double) ((1 - fx) * fy), w11 = (double) (fx * fy);
	o.v[0] = __double2ll_rn(w00 * qfix);
	o.v[1] = __double2ll_rn(w10 * qfix);
	o.v[2] = __double2ll_rn(w01 * qfix);
	o.v[3] = __double2ll_rn(w11 * qfix);
	return o;
}

// The same values on the integer pipe: FP64 conversions, products and
// roundings (20 clocks of an SM per warp each) were half of the kernels.
__device__ __forceinline__ void weights_pos(const bits::Pos &fx, const bits::Pos &fy, bits::Pos w[4])
{
	const bits::Pos gx = bits::pos_one_minus(fx), gy = bits::pos_one_minus(fy);
	w[0] = bits::pos_mul(gx, gy);
	w[1] = bits::pos_mul(fx, gy);
	w[2] = bits::pos_mul(gx, fy);
	w[3] = bits::pos_mul(fx, fy);
}

__device__ __forceinline__ bool charge_pos(const bits::Pos w[4], const Charge &c, long long v[4])
{
	bool ok = true;
	#pragma unroll
	for(int k = 0; k < 4; k++)
		ok &= bits::pos_rint(bits::pos_mul(w[k], c.p), c.neg != 0, v[k]);
	return ok;
}

// FP32: the weights are FP32 products (as before), widened exactly.
__device__ __forceinline__ bool charge_f32(const float w[4], const Charge &c, long long v[4])
{
	bool ok = true;
	#pragma unroll
	for(int k = 0; k < 4; k++)
	{
		bits::Pos p;
		const bool normal = bits::pos_of(w[k], p);
		const bool done = normal && bits::pos_rint(bits::pos_mul24(p, c.p), c.neg != 0, v[k]);
		if(w[k] == 0.0f) v[k] = 0;
		ok = ok && (done || w[k] == 0.0f);
	}
	return ok;
}

// Deposit of one position into the block's region.  extra: what went to the
// grid directly (the block's flush sums the rest).
template <typename T>
__device__ __forceinline__ void put_charge(const AGrid &g, Region &r, T x, T y, const Charge &c,
		bool ok, int ix, int iy, long long v[4], unsigned long long *rho, long long &extra)
{
	if(!ok)
	{
		const Slow4 s = deposit_slow<T>(g, x, y, c.q);
		ix = s.ix; iy = s.iy;
		for(int k = 0; k < 4; k++) v[k] = s.v[k];
	}
	const int node = r.node(g, ix, iy);
	if(node < 0) extra += v[0] + v[1] + v[2] + v[3];
	r.add(g, 0, node, ix, iy, v, rho);
}

__device__ __forceinline__ bool charge_of(const AGrid &g, double x, double y, const Charge &c, int &ix,
		int &iy, long long v[4])
{
	bits::Pos fx, fy, w[4];
	const bool ok = cell_fast(g, x, y, ix, iy, fx, fy);
	weights_pos(fx, fy, w);
	return charge_pos(w, c, v) & ok & (c.fast != 0);
}

__device__ __forceinline__ bool charge_of(const AGrid &g, float x, float y, const Charge &c, int &ix,
		int &iy, long long v[4])
{
	int ix1, iy1;
	float fx, fy;
	cell<float>(g, x, y, ix, iy, ix1, iy1, fx, fy);
	const float w[4] = {(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy};
	return c.fast && charge_f32(w, c, v);
}

// The block's sums onto the grid, and their total (FP32 form: the k = 0 mode
// is removed by the exact sum of the charge) onto *rsum.
__device__ __forceinline__ void close_charge(const AGrid &g, const Region &r, unsigned long long *rho,
		unsigned long long *rsum, long long extra)
{
	__syncthreads();
	long long sum = r.flush(g, 0, rho) + extra;
	if(rsum)
	{
		for(int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
		if((threadIdx.x & 31) == 0) red_add(rsum, sum);
	}
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 4)
k_deposit(const __grid_constant__ AGrid g, const Work *work, const T *x, const T *y,
		const __grid_constant__ Charge c, unsigned long long *rho, unsigned long long *rsum)
{
	extern __shared__ uint32_t smem[];
	pdl_wait();
	const Work w = work[blockIdx.x];
	if(w.tile < 0) return;
	Region r;
	r.open(g, smem, w.tile, 1);
	__syncthreads();
	long long extra = 0;
	for(int64_t i = w.first + threadIdx.x; i < w.end; i += blockDim.x)
	{
		const T px = x[i], py = y[i];
		int ix, iy;
		long long v[4];
		const bool ok = charge_of(g, px, py, c, ix, iy, v);
		put_charge<T>(g, r, px, py, c, ok, ix, iy, v, rho, extra);
	}
	close_charge(g, r, rho, rsum, extra);
}

// E = -grad phi by periodic central differences; clears the charge sums for
// the next deposit (the transform has read them).
template <typename T>
__global__ void k_E(AGrid g, const T *phi, T *Ex, T *Ey, long long *rho, long long *rsum)
{
	pdl_wait();
	int64_t ng = (int64_t) g.nx * g.ny;
	T cx = (T) (0.5 * g.idx), cy = (T) (0.5 * g.idy);
	if(blockIdx.x == 0 && threadIdx.x == 0) *rsum = 0;
	const int lx = 31 - __clz(g.nx);
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < ng;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		int iy = (int) (i >> lx), ix = (int) (i & (g.nx - 1));
		int xm = (ix - 1) & (g.nx - 1), xp = (ix + 1) & (g.nx - 1);
		int ym = (iy - 1) & (g.ny - 1), yp = (iy + 1) & (g.ny - 1);
		Ex[i] = (phi[(int64_t) iy * g.nx + xm] - phi[(int64_t) iy * g.nx + xp]) * cx;
		Ey[i] = (phi[(int64_t) ym * g.nx + ix] - phi[(int64_t) yp * g.nx + ix]) * cy;
		rho[i] = 0;
	}
}

// The CIC sum of E at a position.
template <typename T>
__device__ __forceinline__ void gather(const AGrid &g, const T *Ex, const T *Ey, int ix, int iy,
		T w00, T w10, T w01, T w11, T &ex, T &ey)
{
	const int ix1 = (ix + 1) & (g.nx - 1), iy1 = (iy + 1) & (g.ny - 1);
	int64_t n00 = (int64_t) iy * g.nx + ix, n10 = (int64_t) iy * g.nx + ix1;
	int64_t n01 = (int64_t) iy1 * g.nx + ix, n11 = (int64_t) iy1 * g.nx + ix1;
	ex = w00 * Ex[n00] + w10 * Ex[n10] + w01 * Ex[n01] + w11 * Ex[n11];
	ey = w00 * Ey[n00] + w10 * Ey[n10] + w01 * Ey[n01] + w11 * Ey[n11];
}

template <typename T>
__device__ __forceinline__ void gather_cell(const AGrid &g, const T *Ex, const T *Ey, T px, T py, T &ex,
		T &ey)
{
	int ix, iy, ix1, iy1;
	T fx, fy;
	cell<T>(g, px, py, ix, iy, ix1, iy1, fx, fy);
	T w00 = (1 - fx) * (1 - fy), w10 = fx * (1 - fy), w01 = (1 - fx) * fy, w11 = fx * fy;
	gather<T>(g, Ex, Ey, ix, iy, w00, w10, w01, w11, ex, ey);
}

static __device__ __noinline__ double2 gather_slow(const AGrid &g, const double *Ex, const double *Ey,
		double px, double py)
{
	double2 e;
	gather_cell<double>(g, Ex, Ey, px, py, e.x, e.y);
	return e;
}

// Kick, move and wrap of one particle whose field is (ex, ey).
template <typename T>
__device__ __forceinline__ void advance(const AGrid &g, const Kick &k, T dt, T ex, T ey, T &px, T &py,
		T &u, T &v)
{
	T h = (T) k.h, t = (T) k.t, s = (T) k.s;
	T vmx = u + h * ex, vmy = v + h * ey;
	T vpx = vmx + vmy * t, vpy = vmy - vmx * t;
	T vx = vmx + vpy * s + h * ex, vy = vmy - vpx * s + h * ey;
	u = vx;
	v = vy;
	if(k.move)
	{
		px += dt * vx;
		py += dt * vy;
		if(px >= (T) g.Lx) px -= (T) g.Lx;
		else if(px < 0) px += (T) g.Lx;
		if(py >= (T) g.Ly) py -= (T) g.Ly;
		else if(py < 0) py += (T) g.Ly;
	}
}

// The FP64 form of it: no rotation without a field (it adds zeros), the
// wrap's compares on the integer pipe.
__device__ __forceinline__ void advance(const AGrid &g, const Kick &k, double dt, double ex, double ey,
		double &px, double &py, double &u, double &v)
{
	const double h = k.h;
	const double vmx = u + h * ex, vmy = v + h * ey;
	double vx = vmx, vy = vmy;
	if(k.turns)
	{
		const double t = k.t, s = k.s;
		const double vpx = vmx + vmy * t, vpy = vmy - vmx * t;
		vx = vmx + vpy * s;
		vy = vmy - vpx * s;
	}
	vx += h * ex;
	vy += h * ey;
	u = vx;
	v = vy;
	if(k.move)
	{
		px += dt * vx;
		py += dt * vy;
		if(bits::ge_pos(px, g.Lx)) px -= g.Lx;
		else if(bits::lt_zero(px)) px += g.Lx;
		if(bits::ge_pos(py, g.Ly)) py -= g.Ly;
		else if(bits::lt_zero(py)) py += g.Ly;
	}
}

// Gather, kick, move, wrap; deposit of the new position.  hx/hy (may be
// null) receive the positions before the move.
__device__ __forceinline__ void push_one(const AGrid &g, Region &r, const Kick &k, double dt,
		const double *Ex, const double *Ey, const Charge &c, double &px, double &py, double &u, double &v,
		unsigned long long *rho, long long &extra)
{
	// pass 0: the old position's weights, gather and kick; pass 1: the new
	// one's, the deposit (a loop, not two copies of the weights' code)
	#pragma unroll 1
	for(int pass = 0; ; pass++)
	{
		int ix, iy;
		bits::Pos fx, fy, w[4];
		bool ok = cell_fast(g, px, py, ix, iy, fx, fy) & (c.fast != 0);
		weights_pos(fx, fy, w);
		if(pass)
		{
			long long q[4];
			ok &= charge_pos(w, c, q);
			put_charge<double>(g, r, px, py, c, ok, ix, iy, q, rho, extra);
			return;
		}
		ok &= bits::pos_normal(w[0]) & bits::pos_normal(w[1]) & bits::pos_normal(w[2])
			& bits::pos_normal(w[3]);
		double ex, ey;
		if(ok)
			gather<double>(g, Ex, Ey, ix, iy, bits::pos_val(w[0]), bits::pos_val(w[1]),
					bits::pos_val(w[2]), bits::pos_val(w[3]), ex, ey);
		else
		{
			const double2 e = gather_slow(g, Ex, Ey, px, py);
			ex = e.x; ey = e.y;
		}
		advance(g, k, dt, ex, ey, px, py, u, v);
	}
}

__device__ __forceinline__ void push_one(const AGrid &g, Region &r, const Kick &k, float dt,
		const float *Ex, const float *Ey, const Charge &c, float &px, float &py, float &u, float &v,
		unsigned long long *rho, long long &extra)
{
	float ex, ey;
	gather_cell<float>(g, Ex, Ey, px, py, ex, ey);
	advance<float>(g, k, dt, ex, ey, px, py, u, v);
	int ix, iy;
	long long q[4];
	const bool ok = charge_of(g, px, py, c, ix, iy, q);
	put_charge<float>(g, r, px, py, c, ok, ix, iy, q, rho, extra);
}

template <typename T>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 5 : 4)
k_push(const __grid_constant__ AGrid g, const Work *work, T *x, T *y, T *ux, T *uy, const T *Ex,
		const T *Ey, const __grid_constant__ Kick k, T dt, const __grid_constant__ Charge c,
		unsigned long long *rho, unsigned long long *rsum, T *hx, T *hy)
{
	extern __shared__ uint32_t smem[];
	pdl_wait();
	const Work w = work[blockIdx.x];
	if(w.tile < 0) return;
	Region r;
	r.open(g, smem, w.tile, 1);
	__syncthreads();
	long long extra = 0;
	for(int64_t i = w.first + threadIdx.x; i < w.end; i += blockDim.x)
	{
		T px = x[i], py = y[i], u = ux[i], v = uy[i];
		if(hx) { hx[i] = px; hy[i] = py; }
		push_one(g, r, k, dt, Ex, Ey, c, px, py, u, v, rho, extra);
		x[i] = px;
		y[i] = py;
		ux[i] = u;
		uy[i] = v;
	}
	close_charge(g, r, rho, rsum, extra);
}

// Per-block partial sums of |E|^2 (FP64), then one block adds them in a
// fixed order: deterministic.
template <typename T>
__global__ void k_energy_part(int64_t ng, const T *Ex, const T *Ey, double *part)
{
	__shared__ double sh[32];
	double acc = 0.0;
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < ng;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		double a = (double) Ex[i], b = (double) Ey[i];
		acc += a * a + b * b;
	}
	for(int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	if((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
	__syncthreads();
	if(threadIdx.x == 0)
	{
		double s = 0.0;
		for(int w = 0; w < (int) (blockDim.x >> 5); w++) s += sh[w];
		part[blockIdx.x] = s;
	}
}

__global__ void k_sum_parts(int nb, const double *part, double scale, double *out)
{
	if(threadIdx.x == 0 && blockIdx.x == 0)
	{
		double s = 0.0;
		for(int b = 0; b < nb; b++) s += part[b];
		*out = s * scale;
	}
}

// ---------------------------------------------------------------- reverse

// Eb = e0 dx dy E (dL/dE of the loss).
template <typename T>
__global__ void k_loss_grad(int64_t ng, const T *Ex, const T *Ey, double f, T *Ebx, T *Eby)
{
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < ng;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		Ebx[i] = (T) (f * (double) Ex[i]);
		Eby[i] = (T) (f * (double) Ey[i]);
	}
}

// phib = (-grad_h)^T Eb: phib_m = (Ebx[m+1] - Ebx[m-1]) / (2dx) + same in y.
// fix: Eb as fixed-point sums (two components, scale 2^eexp) instead of real.
// Clears the maximum of rhob that the solve's last kernel takes.
template <typename T>
__global__ void k_div(AGrid g, const T *Ebx, const T *Eby, const long long *fix, Scale *sc, T *phib)
{
	pdl_wait();
	int64_t ng = (int64_t) g.nx * g.ny;
	T cx = (T) (0.5 * g.idx), cy = (T) (0.5 * g.idy);
	if(blockIdx.x == 0 && threadIdx.x == 0) sc->r = 0;
	const double inv = bits::from_bits((uint64_t) (uint32_t) (1023 - sc->eexp) << 52);
	const int lx = 31 - __clz(g.nx);
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < ng;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		int iy = (int) (i >> lx), ix = (int) (i & (g.nx - 1));
		int xm = (ix - 1) & (g.nx - 1), xp = (ix + 1) & (g.nx - 1);
		int ym = (iy - 1) & (g.ny - 1), yp = (iy + 1) & (g.ny - 1);
		const int64_t e = (int64_t) iy * g.nx + xp, w = (int64_t) iy * g.nx + xm;
		const int64_t s = (int64_t) yp * g.nx + ix, n = (int64_t) ym * g.nx + ix;
		T be, bw, bs, bn;
		if(fix)
		{
			be = (T) ((double) fix[e] * inv);
			bw = (T) ((double) fix[w] * inv);
			bs = (T) ((double) fix[ng + s] * inv);
			bn = (T) ((double) fix[ng + n] * inv);
		}
		else { be = Ebx[e]; bw = Ebx[w]; bs = Eby[s]; bn = Eby[n]; }
		phib[i] = (be - bw) * cx + (bs - bn) * cy;
	}
}

// max |rhob| into sc->r; clears the fixed-point Eb sums (k_div has read them)
// and the step maxima that the reverse step after next writes.
template <typename T>
__global__ void k_absmax(int64_t ng, const T *v, Scale *sc, long long *fix, int par)
{
	__shared__ unsigned long long sh[kThreads / 32];
	pdl_wait();
	if(blockIdx.x == 0 && threadIdx.x == 0) { sc->u[par] = 0; sc->p[par] = 0; }
	unsigned long long m = 0;
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < ng;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		const unsigned long long b = abs_bits((double) v[i]);
		m = b > m ? b : m;
		fix[i] = 0;
		fix[ng + i] = 0;
	}
	block_max(m, &sc->r, sh);
}

// Exponent of the next adjoint deposit's scale from a bound on |eb|:
//   |ut|_inf <= umax + move dt (pmax + |c| 2 max(idx, idy) rmax)
//   |eb|_inf <= |h| (1 + |a| + |s|) |ut|_inf
// and a node sums at most n such contributions (weights sum to 1), which stay
// below 2^61.
__device__ __forceinline__ int scale_exp(const Scale *sc, int par, const Kick &k, double dt, double c,
		double gmax, double n)
{
	const double umax = __longlong_as_double((long long) sc->u[par]);
	const double pmax = __longlong_as_double((long long) sc->p[par]);
	const double rmax = __longlong_as_double((long long) sc->r);
	const double ut = umax + (k.move ? dt * (pmax + fabs(c) * 2.0 * gmax * rmax) : 0.0);
	const double eb = fabs(k.h) * (1.0 + fabs(k.a) + fabs(k.s)) * ut;
	const double bound = n * eb;
	const uint64_t b = bits::to_bits(bound);
	const int e = (int) (b >> 52) - 1023;           // floor(log2 bound)
	if(b == 0 || (b >> 63) || e > 1023)
		return 0;                                   // zero, infinite or NaN: unscaled
	// floor(62 - log2 bound) - 1 (kept a normal double's exponent)
	return min(960, ((b & 0xfffffffffffffull) == 0 ? 62 - e : 61 - e) - 1);
}

// grad of sum_n w_n(p) F_n with respect to p.
template <typename T>
__device__ __forceinline__ void wgrad(const AGrid &g, T fx, T fy, T f00, T f10, T f01, T f11,
		T &gx, T &gy)
{
	gx = (T) g.idx * ((1 - fy) * (f10 - f00) + fy * (f11 - f01));
	gy = (T) g.idy * ((1 - fx) * (f01 - f00) + fx * (f11 - f10));
}

// FP64: both from the four differences (the mixed one shared), 8
// instructions instead of 12.
__device__ __forceinline__ void wgrad(const AGrid &g, double fx, double fy, double f00, double f10,
		double f01, double f11, double &gx, double &gy)
{
	const double ax = f10 - f00, ay = f01 - f00;
	const double m = (f11 - f01) - ax;
	gx = g.idx * (ax + fy * m);
	gy = g.idy * (ay + fx * m);
}

// Fractions of a position, and its cell.
__device__ __forceinline__ void frac_of(const AGrid &g, double x, double y, int &ix, int &iy, int &ix1,
		int &iy1, double &fx, double &fy)
{
	bits::Pos px, py;
	if(cell_fast(g, x, y, ix, iy, px, py))
	{
		ix1 = (ix + 1) & (g.nx - 1);
		iy1 = (iy + 1) & (g.ny - 1);
		fx = bits::pos_val(px);
		fy = bits::pos_val(py);
	}
	else
		cell<double>(g, x, y, ix, iy, ix1, iy1, fx, fy);
}
__device__ __forceinline__ void frac_of(const AGrid &g, float x, float y, int &ix, int &iy, int &ix1,
		int &iy1, float &fx, float &fy)
{
	cell<float>(g, x, y, ix, iy, ix1, iy1, fx, fy);
}

// The adjoint deposit's four values rn(w eb 2^eexp), order 00, 10, 01, 11, on
// FP64 instructions.
template <typename T>
static __device__ __noinline__ Slow4 eb_slow(T fx, T fy, T eb, int eexp)
{
	Slow4 o;
	o.ix = o.iy = 0;
	const double e = (double) eb * bits::from_bits((uint64_t) (uint32_t) (1023 + eexp) << 52);
	double w00 = (double) ((1 - fx) * (1 - fy)), w10 = (double) (fx * (1 - fy));
	double w01 = (double) ((1 - fx) * fy), w11 = (double) (fx * fy);
	o.v[0] = __double2ll_rn(w00 * e);
	o.v[1] = __double2ll_rn(w10 * e);
	o.v[2] = __double2ll_rn(w01 * e);
	o.v[3] = __double2ll_rn(w11 * e);
	return o;
}

// The same on the integer pipe (w eb is exact in 48 bits for the FP32 form).
__device__ __forceinline__ bool eb_values(const bits::Pos w[4], double eb, int eexp, long long v[4])
{
	bits::Pos e;
	const uint64_t b = bits::to_bits(eb);
	bool ok = bits::pos_of(bits::from_bits(b & 0x7fffffffffffffffull), e);
	e.e += eexp;
	#pragma unroll
	for(int k = 0; k < 4; k++)
		ok &= bits::pos_rint(bits::pos_mul(w[k], e), (b >> 63) != 0, v[k]);
	return ok;
}
__device__ __forceinline__ bool eb_values(const bits::Pos w[4], float eb, int eexp, long long v[4])
{
	bits::Pos e;
	bool ok = bits::pos_of(fabsf(eb), e);
	e.e += eexp;
	#pragma unroll
	for(int k = 0; k < 4; k++)
		ok &= bits::pos_rint(bits::pos_mul24x24(w[k], e), eb < 0.0f, v[k]);
	return ok;
}
__device__ __forceinline__ bool eb_weights(double fx, double fy, bits::Pos w[4])
{
	bits::Pos px, py;
	bool ok = bits::pos_of(fx, px) & bits::pos_of(fy, py);
	ok &= (px.e < 0) & (py.e < 0);
	weights_pos(px, py, w);
	return ok;
}
__device__ __forceinline__ bool eb_weights(float fx, float fy, bits::Pos w[4])
{
	const float f[4] = {(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy};
	bool ok = true;
	#pragma unroll
	for(int k = 0; k < 4; k++) ok &= bits::pos_of(f[k], w[k]);
	return ok;
}

// ub <- M^T ut, eb = h (ut + ub)
template <typename T>
__device__ __forceinline__ void kick_back(const Kick &k, T utx, T uty, T &vbx, T &vby, T &ebx, T &eby)
{
	T a = (T) k.a, s = (T) k.s, h = (T) k.h;
	vbx = a * utx - s * uty;
	vby = s * utx + a * uty;
	ebx = h * (utx + vbx);
	eby = h * (uty + vby);
}

// One reverse step j, fused with the deposit term of step j+1 (nxt = p_{j+1},
// rhob = rhob_{j+1}).  par: parity of this step's maxima; the scale comes
// from the other one's.
template <typename T>
__global__ void __launch_bounds__(kThreads, 4)
k_rev(const __grid_constant__ AGrid g, const Work *work, const T *nx_, const T *ny_, const T *rhob,
		double c, const T *px_, const T *py_, const T *Ex, const T *Ey, const __grid_constant__ Kick k,
		T dt, T *pbx, T *pby, T *ubx, T *uby, Scale *sc, int par, double gmax, double n,
		unsigned long long *Ebx, unsigned long long *Eby)
{
	extern __shared__ uint32_t smem[];
	__shared__ unsigned long long sh[kThreads / 32];
	__shared__ int s_eexp;
	pdl_wait();
	const Work w = work[blockIdx.x];
	// (block 0 leaves the scale for k_div even without work of its own)
	if(w.tile < 0 && blockIdx.x != 0) return;
	if(threadIdx.x == 0)
	{
		s_eexp = scale_exp(sc, par ^ 1, k, (double) dt, c, gmax, n);
		if(blockIdx.x == 0) sc->eexp = s_eexp;
	}
	if(w.tile < 0) return;
	Region r;
	r.open(g, smem, w.tile, 2);
	__syncthreads();
	const int eexp = s_eexp;
	unsigned long long umax = 0, pmax = 0;
	for(int64_t i = w.first + threadIdx.x; i < w.end; i += blockDim.x)
	{
		T bx = pbx[i], by = pby[i];
		int ix, iy, ix1, iy1;
		T fx, fy, gx, gy;
		frac_of(g, nx_[i], ny_[i], ix, iy, ix1, iy1, fx, fy);
		wgrad(g, fx, fy, rhob[(int64_t) iy * g.nx + ix], rhob[(int64_t) iy * g.nx + ix1],
				rhob[(int64_t) iy1 * g.nx + ix], rhob[(int64_t) iy1 * g.nx + ix1], gx, gy);
		bx += (T) c * gx;
		by += (T) c * gy;
		T utx = ubx[i], uty = uby[i];
		if(k.move) { utx += dt * bx; uty += dt * by; }
		T vbx, vby, ebx, eby;
		kick_back(k, utx, uty, vbx, vby, ebx, eby);
		frac_of(g, px_[i], py_[i], ix, iy, ix1, iy1, fx, fy);
		int64_t n00 = (int64_t) iy * g.nx + ix, n10 = (int64_t) iy * g.nx + ix1;
		int64_t n01 = (int64_t) iy1 * g.nx + ix, n11 = (int64_t) iy1 * g.nx + ix1;
		T d00 = Ex[n00] * ebx + Ey[n00] * eby, d10 = Ex[n10] * ebx + Ey[n10] * eby;
		T d01 = Ex[n01] * ebx + Ey[n01] * eby, d11 = Ex[n11] * ebx + Ey[n11] * eby;
		wgrad(g, fx, fy, d00, d10, d01, d11, gx, gy);
		bx += gx;
		by += gy;
		pbx[i] = bx;
		pby[i] = by;
		ubx[i] = vbx;
		uby[i] = vby;
		const unsigned long long b0 = abs_bits((double) vbx), b1 = abs_bits((double) vby);
		const unsigned long long b2 = abs_bits((double) bx), b3 = abs_bits((double) by);
		umax = max(umax, max(b0, b1));
		pmax = max(pmax, max(b2, b3));
		bits::Pos wp[4];
		const bool ok = eb_weights(fx, fy, wp);
		const int node = r.node(g, ix, iy);
		#pragma unroll
		for(int comp = 0; comp < 2; comp++)
		{
			const T eb = comp ? eby : ebx;
			long long v[4];
			if(!(ok && eb_values(wp, eb, eexp, v)))
			{
				const Slow4 s = eb_slow<T>(fx, fy, eb, eexp);
				for(int q = 0; q < 4; q++) v[q] = s.v[q];
			}
			r.add(g, comp, node, ix, iy, v, comp ? Eby : Ebx);
		}
	}
	block_max(umax, &sc->u[par], sh);
	block_max(pmax, &sc->p[par], sh);
	r.flush(g, 0, Ebx);
	r.flush(g, 1, Eby);
}

// Last term: pb_0 += c grad D(p_0)^T rhob_0; results to FP64, in the caller's
// order (src of the first epoch).
template <typename T>
__global__ void k_finish(AGrid g, int64_t n, const uint32_t *src, const T *px_, const T *py_,
		const T *rhob, double c, const T *pbx, const T *pby, const T *ubx, const T *uby, double *out)
{
	for(int64_t k = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; k < n;
			k += (int64_t) gridDim.x * blockDim.x)
	{
		int ix, iy, ix1, iy1;
		T fx, fy, gx, gy;
		frac_of(g, px_[k], py_[k], ix, iy, ix1, iy1, fx, fy);
		wgrad(g, fx, fy, rhob[(int64_t) iy * g.nx + ix], rhob[(int64_t) iy * g.nx + ix1],
				rhob[(int64_t) iy1 * g.nx + ix], rhob[(int64_t) iy1 * g.nx + ix1], gx, gy);
		const int64_t i = src[k];
		out[i] = (double) pbx[k] + c * (double) gx;
		out[n + i] = (double) pby[k] + c * (double) gy;
		out[2 * n + i] = (double) ubx[k];
		out[3 * n + i] = (double) uby[k];
	}
}

// Whether the staged state (x, y, ux, uy, n doubles each) is one that the run
// accepts: positions in [0, L), finite velocities.  *bad is set otherwise.
__global__ void k_check(int64_t n, const double *in, double Lx, double Ly, int32_t *bad)
{
	bool b = false;
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		const double x = in[i], y = in[n + i];
		b = b || !(x >= 0.0 && x < Lx && y >= 0.0 && y < Ly)
			|| !bits::is_finite(in[2 * n + i]) || !bits::is_finite(in[3 * n + i]);
	}
	if(b) *bad = 1;
}

template <typename T>
__global__ void k_from_f64(int64_t n, const double *in, T *x, T *y, T *ux, T *uy)
{
	for(int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n;
			i += (int64_t) gridDim.x * blockDim.x)
	{
		x[i] = (T) in[i];
		y[i] = (T) in[n + i];
		ux[i] = (T) in[2 * n + i];
		uy[i] = (T) in[3 * n + i];
	}
}

} // namespace adj
} // namespace cpic

using namespace cpic;
using namespace cpic::adj;

struct cpic_adj {
	cpic_adj_params_t p;
	AGrid g;
	Grid fg;                  // for the FFT launchers (nx, ny)
	int64_t n, ng;
	bool f64;
	size_t ts;                // sizeof(T)
	double qfix, qinv;        // forward charge fixed point
	cudaStream_t st;
	cudaEvent_t ev[4];
	// particles (T): x, y, ux, uy; adjoints pbx, pby, ubx, uby
	void *x, *y, *ux, *uy, *pbx, *pby, *ubx, *uby;
	void *ckpt;               // nckpt x 4 x n (T)
	void *hist;               // K x 2 x n (T): positions p_j of a segment
	void *histE;              // K x 2 x ng (T): fields E_j of a segment
	void *Ex, *Ey;            // current field (T)
	void *phi, *rhob, *Ebx, *Eby, *spec;
	long long *rho, *Ebfix;   // ng; 2 x ng
	long long *rsum;
	Scale *sc;
	// particle orders: nep of them, each with the permutation from the order
	// before (src) and the blocks' work list
	int nep, sort_every;      // segments per order
	int nt, chunk, nwork;
	bool idx_ok;              // 1/dx, 1/dy are normal doubles
	uint32_t *src;
	int32_t *tcnt;
	Work *work;
	int32_t *bad;
	double *part, *loss_d, *stage;
	void *twx, *twy;
	void *green;              // Green's function, column order (T)
	int nckpt;
	bool have_forward;
	double loss;
	float ms_fwd, ms_bwd;
};

namespace {

int blocks_for(int64_t n)
{
	int64_t b = (n + 255) / 256;
	if(b > 152 * 16) b = 152 * 16;
	return (int) (b < 1 ? 1 : b);
}

Kick kick_of(const cpic_adj *a, int64_t j)
{
	Kick k;
	double dtp = j == 0 ? -0.5 * a->p.dt : a->p.dt;   // mover.c:204-213
	k.h = 0.5 * dtp * a->p.q / a->p.m;
	k.t = a->p.Bz * k.h;
	k.s = 2.0 * k.t / (1.0 + k.t * k.t);
	k.a = 1.0 - k.s * k.t;
	k.move = j == 0 ? 0 : 1;
	k.turns = k.t != 0.0;
	return k;
}

template <typename T>
T *P(void *v, int64_t off = 0) { return reinterpret_cast<T *>(v) + off; }

Charge charge_consts(const cpic_adj *a)
{
	Charge c;
	c.q = a->qfix;
	c.neg = a->qfix < 0.0;
	c.fast = bits::pos_of(fabs(a->qfix), c.p) && a->idx_ok;
	return c;
}

int epoch_of(const cpic_adj *a, int64_t seg) { return (int) (seg / a->sort_every); }
const Work *work_of(const cpic_adj *a, int64_t seg) { return a->work + (int64_t) epoch_of(a, seg) * a->nwork; }
size_t region_bytes(const cpic_adj *a, int comps)
{
	return 2 * (size_t) comps * a->g.W * a->g.W * sizeof(uint32_t);
}

unsigned long long *U(long long *p) { return reinterpret_cast<unsigned long long *>(p); }

// The FP32 form's exact sum of the charge (its mean is removed before the
// transform); null for the FP64 form.
long long *mean_sum(const cpic_adj *a) { return a->f64 ? nullptr : a->rsum; }

// rho (fixed point) -> E (T) into Ex/Ey; clears rho.
template <typename T>
void solve_E(cpic_adj *a, T *Ex, T *Ey)
{
	typedef typename Cx<T>::t C;
	poisson_launch<T>(a->fg, a->rho, a->qinv, mean_sum(a), P<C>(a->spec), P<C>(a->twx), P<C>(a->twy),
			P<T>(a->phi), a->st, P<T>(a->green));
	launch_pdl(k_E<T>, blocks_for(a->ng), 256, 0, a->st, a->g, P<T>(a->phi), Ex, Ey, a->rho, a->rsum);
}

// The charge of the current positions, from nothing.
template <typename T>
void deposit_all(cpic_adj *a, int64_t seg)
{
	cudaMemsetAsync(a->rho, 0, a->ng * sizeof(long long), a->st);
	cudaMemsetAsync(a->rsum, 0, sizeof(long long), a->st);
	launch_pdl(k_deposit<T>, a->nwork, kThreads, region_bytes(a, 1), a->st, a->g, work_of(a, seg),
			P<T>(a->x), P<T>(a->y), charge_consts(a), U(a->rho), U(mean_sum(a)));
}

// Sorts the state by tile; the order becomes that of epoch ep.
template <typename T>
void sort_state(cpic_adj *a, int ep)
{
	const int64_t n = a->n;
	cudaMemsetAsync(a->tcnt, 0, a->nt * sizeof(int32_t), a->st);
	const int nb = (int) std::max<int64_t>(1, std::min<int64_t>(152 * 4, n / 2048));
	k_tile_count<T><<<nb, 256, 0, a->st>>>(a->g, n, P<T>(a->x), P<T>(a->y), a->nt, a->tcnt);
	k_tile_scan<<<1, 1024, 0, a->st>>>(a->nt, a->chunk, a->tcnt, a->work + (int64_t) ep * a->nwork,
			a->nwork);
	// (the adjoints' buffers are free in the forward sweep)
	k_tile_place<T><<<nb, 256, 0, a->st>>>(a->g, n, P<T>(a->x), P<T>(a->y), P<T>(a->ux),
			P<T>(a->uy), P<T>(a->pbx), P<T>(a->pby), P<T>(a->ubx), P<T>(a->uby), a->nt, a->tcnt,
			a->src + (int64_t) ep * n);
	std::swap(a->x, a->pbx);
	std::swap(a->y, a->pby);
	std::swap(a->ux, a->ubx);
	std::swap(a->uy, a->uby);
}

// Steps [j0, j1) from the current state.  first: the forward sweep, which
// sorts and keeps checkpoints; else a segment's recompute, which keeps p_j
// and E_j.
template <typename T>
void run_steps(cpic_adj *a, int64_t j0, int64_t j1, bool first)
{
	const int64_t n = a->n, ng = a->ng;
	const int K = (int) a->p.checkpoint_every;
	const Charge c = charge_consts(a);
	for(int64_t j = j0; j < j1; j++)
	{
		if(first && j % K == 0)
		{
			if(j > 0 && (j / K) % a->sort_every == 0)
				sort_state<T>(a, epoch_of(a, j / K));
			T *ck = P<T>(a->ckpt, (j / K) * 4 * n);
			cudaMemcpyAsync(ck, a->x, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
			cudaMemcpyAsync(ck + n, a->y, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
			cudaMemcpyAsync(ck + 2 * n, a->ux, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
			cudaMemcpyAsync(ck + 3 * n, a->uy, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
		}
		const int64_t s = j - j0;
		T *Ex = first ? P<T>(a->Ex) : P<T>(a->histE, s * 2 * ng);
		T *Ey = first ? P<T>(a->Ey) : Ex + ng;
		solve_E<T>(a, Ex, Ey);
		T *hx = first ? nullptr : P<T>(a->hist, s * 2 * n);
		T *hy = first ? nullptr : hx + n;
		launch_pdl(k_push<T>, a->nwork, kThreads, region_bytes(a, 1), a->st, a->g, work_of(a, j / K),
				P<T>(a->x), P<T>(a->y), P<T>(a->ux), P<T>(a->uy), Ex, Ey, kick_of(a, j), (T) a->p.dt, c,
				U(a->rho), U(mean_sum(a)), hx, hy);
	}
}

// Eb (T, in a->Ebx/Eby, or the fixed-point sums) -> rhob and its maximum.
// par: parity of the next reverse step.
template <typename T>
void grid_adjoint(cpic_adj *a, bool fixed, int par)
{
	typedef typename Cx<T>::t C;
	launch_pdl(k_div<T>, blocks_for(a->ng), 256, 0, a->st, a->g, P<T>(a->Ebx), P<T>(a->Eby),
			fixed ? a->Ebfix : nullptr, a->sc, P<T>(a->phi));
	poisson_launch_real<T>(a->g.nx, a->g.ny, P<T>(a->phi), P<C>(a->spec), P<C>(a->twx), P<C>(a->twy),
			P<T>(a->green), P<T>(a->rhob), a->st);
	launch_pdl(k_absmax<T>, blocks_for(a->ng), kThreads, 0, a->st, a->ng, P<T>(a->rhob), a->sc, a->Ebfix,
			par);
}

template <typename T>
int forward_impl(cpic_adj *a)
{
	int64_t n = a->n, ng = a->ng;
	cudaEventRecord(a->ev[0], a->st);
	k_from_f64<T><<<blocks_for(n), 256, 0, a->st>>>(n, a->stage, P<T>(a->x), P<T>(a->y), P<T>(a->ux),
			P<T>(a->uy));
	sort_state<T>(a, 0);
	deposit_all<T>(a, 0);
	run_steps<T>(a, 0, a->p.nsteps, true);
	solve_E<T>(a, P<T>(a->Ex), P<T>(a->Ey));
	int nb = 152;
	k_energy_part<T><<<nb, 256, 0, a->st>>>(ng, P<T>(a->Ex), P<T>(a->Ey), a->part);
	k_sum_parts<<<1, 32, 0, a->st>>>(nb, a->part, 0.5 * a->p.e0 * a->g.dx * a->g.dy, a->loss_d);
	cudaEventRecord(a->ev[1], a->st);
	cudaMemcpyAsync(&a->loss, a->loss_d, sizeof(double), cudaMemcpyDeviceToHost, a->st);
	if(cudaStreamSynchronize(a->st) != cudaSuccess) return CPIC_ECUDA;
	cudaEventElapsedTime(&a->ms_fwd, a->ev[0], a->ev[1]);
	return CPIC_OK;
}

template <typename T>
int backward_impl(cpic_adj *a)
{
	int64_t n = a->n, ng = a->ng, N = a->p.nsteps;
	int K = (int) a->p.checkpoint_every;
	double c = -a->p.q / a->p.e0;                 // interpolate.c:307
	double gmax = a->g.idx > a->g.idy ? a->g.idx : a->g.idy;
	cudaEventRecord(a->ev[2], a->st);
	// dL/dE of the final field (a->Ex/Ey still hold it), then rhob_N
	k_loss_grad<T><<<blocks_for(ng), 256, 0, a->st>>>(ng, P<T>(a->Ex), P<T>(a->Ey),
			a->p.e0 * a->g.dx * a->g.dy, P<T>(a->Ebx), P<T>(a->Eby));
	cudaMemsetAsync(a->sc, 0, sizeof(Scale), a->st);
	int par = 0;
	grid_adjoint<T>(a, false, par);
	cudaMemsetAsync(a->pbx, 0, n * sizeof(T), a->st);
	cudaMemsetAsync(a->pby, 0, n * sizeof(T), a->st);
	cudaMemsetAsync(a->ubx, 0, n * sizeof(T), a->st);
	cudaMemsetAsync(a->uby, 0, n * sizeof(T), a->st);
	int64_t nseg = (N + K - 1) / K;
	for(int64_t sgi = nseg - 1; sgi >= 0; sgi--)
	{
		int64_t j0 = sgi * K, j1 = j0 + K < N ? j0 + K : N;
		if(sgi + 1 < nseg && epoch_of(a, sgi) != epoch_of(a, sgi + 1))
		{
			// the adjoints to this segment's order (the state's buffers are
			// about to be overwritten)
			k_unsort<T><<<blocks_for(n), 256, 0, a->st>>>(n, a->src + (int64_t) epoch_of(a, sgi + 1) * n,
					P<T>(a->pbx), P<T>(a->pby), P<T>(a->ubx), P<T>(a->uby), P<T>(a->x), P<T>(a->y),
					P<T>(a->ux), P<T>(a->uy));
			std::swap(a->x, a->pbx);
			std::swap(a->y, a->pby);
			std::swap(a->ux, a->ubx);
			std::swap(a->uy, a->uby);
		}
		// restore the checkpoint and recompute the segment
		T *ck = P<T>(a->ckpt, sgi * 4 * n);
		cudaMemcpyAsync(a->x, ck, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
		cudaMemcpyAsync(a->y, ck + n, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
		cudaMemcpyAsync(a->ux, ck + 2 * n, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
		cudaMemcpyAsync(a->uy, ck + 3 * n, n * sizeof(T), cudaMemcpyDeviceToDevice, a->st);
		deposit_all<T>(a, sgi);
		run_steps<T>(a, j0, j1, false);
		// after the recompute a->x/y hold p_{j1}
		for(int64_t j = j1 - 1; j >= j0; j--)
		{
			int64_t s = j - j0;
			const T *nxp, *nyp;
			if(j + 1 == j1) { nxp = P<T>(a->x); nyp = P<T>(a->y); }
			else { nxp = P<T>(a->hist, (s + 1) * 2 * n); nyp = nxp + n; }
			const T *hp = P<T>(a->hist, s * 2 * n);
			const T *hE = P<T>(a->histE, s * 2 * ng);
			launch_pdl(k_rev<T>, a->nwork, kThreads, region_bytes(a, 2), a->st, a->g, work_of(a, sgi), nxp, nyp,
					P<T>(a->rhob), c, hp, hp + n, hE, hE + ng, kick_of(a, j), (T) a->p.dt, P<T>(a->pbx),
					P<T>(a->pby), P<T>(a->ubx), P<T>(a->uby), a->sc, par, gmax, (double) n, U(a->Ebfix),
					U(a->Ebfix + ng));
			par ^= 1;
			grid_adjoint<T>(a, true, par);
		}
	}
	// pb_0 += c grad D(p_0)^T rhob_0 (p_0 = the first checkpoint)
	T *p0 = P<T>(a->ckpt);
	k_finish<T><<<blocks_for(n), 256, 0, a->st>>>(a->g, n, a->src, p0, p0 + n, P<T>(a->rhob), c,
			P<T>(a->pbx), P<T>(a->pby), P<T>(a->ubx), P<T>(a->uby), a->stage);
	cudaEventRecord(a->ev[3], a->st);
	if(cudaStreamSynchronize(a->st) != cudaSuccess) return CPIC_ECUDA;
	cudaEventElapsedTime(&a->ms_bwd, a->ev[2], a->ev[3]);
	return CPIC_OK;
}

bool pow2i(int64_t v) { return v >= 4 && (v & (v - 1)) == 0; }

} // namespace

CPIC_API int cpic_adj_create(const cpic_adj_params_t *p, int64_t n, cpic_adj_t **out)
{
	if(!p || !out || n <= 0) return CPIC_EINVAL;
	*out = nullptr;
	if(!pow2i(p->nx) || !pow2i(p->ny) || p->nx > 16384 || p->ny > 16384) return CPIC_EINVAL;
	if(!(p->Lx > 0) || !(p->Ly > 0) || !(p->dt > 0) || !(p->e0 > 0) || p->m == 0.0 || p->q == 0.0)
		return CPIC_EINVAL;
	if(p->nsteps < 1 || p->checkpoint_every < 1) return CPIC_EINVAL;
	if(p->precision != CPIC_FP64 && p->precision != CPIC_MIXED) return CPIC_EINVAL;
	int ndev = 0;
	if(cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return CPIC_ENODEV;

	cpic_adj *a = new cpic_adj();
	a->p = *p;
	if(a->p.checkpoint_every > a->p.nsteps) a->p.checkpoint_every = a->p.nsteps;
	a->n = n;
	a->g.nx = (int) p->nx; a->g.ny = (int) p->ny;
	a->g.Lx = p->Lx; a->g.Ly = p->Ly;
	a->g.dx = p->Lx / p->nx; a->g.dy = p->Ly / p->ny;
	a->g.idx = 1.0 / a->g.dx; a->g.idy = 1.0 / a->g.dy;
	memset(&a->fg, 0, sizeof(a->fg));
	a->fg.nx = a->g.nx; a->fg.ny = a->g.ny;
	a->ng = p->nx * p->ny;
	a->f64 = p->precision == CPIC_FP64;
	a->ts = a->f64 ? sizeof(double) : sizeof(float);
	// |rho| sums at most n |q/e0| (weights sum to 1): no wrap below 2^62
	double bound = (double) n * fabs(p->q / p->e0);
	int k = (int) floor(62.0 - log2(bound)) - 1;
	a->qfix = -p->q / p->e0 * ldexp(1.0, k);
	a->qinv = ldexp(1.0, -k);
	int K = (int) a->p.checkpoint_every;
	a->nckpt = (int) ((p->nsteps + K - 1) / K);
	a->idx_ok = bits::pos_of(a->g.idx, a->g.idx_p) & bits::pos_of(a->g.idy, a->g.idy_p);
	// Particles per block: enough blocks for the SMs to finish together (four
	// or five are resident on each), else as many as amortise the region's
	// flush.  Forward and reverse of 20 steps, ms, with 256, 512, 1024 and 2048
	// per block: FP64 (whose particles take longest) 140,000 on 128 x 128
	// 2.95, 3.22, 3.52, 3.95; 300,000 3.50, 3.74, 4.54, 4.91; 1,048,576 6.52,
	// 6.44, 6.58, 7.52; 3,145,728 on 256 x 256 16.3, 15.6, 15.5, 16.3; 5,242,880
	// 26.0, 24.7, 24.1, 24.6; 10,485,760 on 512 x 512 53.4, 50.6, 49.2, 49.5.
	// FP32 70,000 on 64 x 64 1.38, 1.44, 1.54, 1.91; 150,000 1.56, 1.56, 1.68,
	// 1.90; 600,000 on 128 x 128 2.64, 2.48, 2.70, 3.19; 1,572,864 4.57, 4.07,
	// 3.95, 4.13; 3,145,728 on 256 x 256 8.38, 7.25, 6.83, 6.89; 5,242,880 13.5,
	// 11.6, 10.7, 10.4.  (The FP64 limits at 150,000 and 8 million lie a few per
	// cent from where the curves cross.)
	if(a->f64)
		a->chunk = n >= 8 << 20 ? 2048 : n >= 4 << 20 ? 1024 : n >= 150000 ? 512 : 256;
	else
		a->chunk = n >= 4 << 20 ? 2048 : n >= 1 << 20 ? 1024 : n >= 75000 ? 512 : 256;
	// tiles of 8 cells, more on sparse and on large grids
	int tside = 8;
	while(tside > p->nx || tside > p->ny) tside >>= 1;
	auto tiles = [&]() { return ((int64_t) p->nx / tside) * (p->ny / tside); };
	while(tside < 32 && 2 * tside <= p->nx && 2 * tside <= p->ny
			&& (tiles() > 4096 || n / tiles() < a->chunk))
		tside <<= 1;
	a->nt = (int) tiles();
	a->nwork = (int) (n / a->chunk + a->nt);
	a->g.lts = 0;
	while((1 << a->g.lts) < tside) a->g.lts++;
	a->g.ntx = (int) p->nx / tside;
	a->g.margin = kMargin;
	a->g.W = tside + 2 * kMargin + 1;
	a->sort_every = (kSortSteps + K - 1) / K;
	a->nep = (a->nckpt + a->sort_every - 1) / a->sort_every;
	int64_t ng = a->ng, nh = p->nx / 2 + 1;
	double *cosx = nullptr, *cosy = nullptr;
	size_t ts = a->ts, cs = 2 * ts;
	int r = CPIC_OK;
	if(cudaStreamCreateWithFlags(&a->st, cudaStreamNonBlocking) != cudaSuccess)
	{
		delete a;
		return CPIC_ECUDA;
	}
	for(int i = 0; i < 4; i++) cudaEventCreate(&a->ev[i]);
#define AL(ptr, bytes) do { if(cudaMalloc((void **) &(ptr), (bytes)) != cudaSuccess) { r = CPIC_ENOMEM; goto fail; } } while(0)
	AL(a->x, n * ts); AL(a->y, n * ts); AL(a->ux, n * ts); AL(a->uy, n * ts);
	AL(a->pbx, n * ts); AL(a->pby, n * ts); AL(a->ubx, n * ts); AL(a->uby, n * ts);
	AL(a->ckpt, (size_t) a->nckpt * 4 * n * ts);
	AL(a->hist, (size_t) K * 2 * n * ts);
	AL(a->histE, (size_t) K * 2 * ng * ts);
	AL(a->Ex, ng * ts); AL(a->Ey, ng * ts);
	AL(a->phi, ng * ts); AL(a->rhob, ng * ts); AL(a->Ebx, ng * ts); AL(a->Eby, ng * ts);
	AL(a->spec, (size_t) p->ny * nh * cs);
	AL(a->rho, ng * sizeof(long long));
	AL(a->Ebfix, 2 * ng * sizeof(long long));
	AL(a->rsum, sizeof(long long));
	AL(a->sc, sizeof(Scale));
	AL(a->src, (size_t) a->nep * n * sizeof(uint32_t));
	AL(a->work, (size_t) a->nep * a->nwork * sizeof(Work));
	AL(a->tcnt, a->nt * sizeof(int32_t));
	AL(a->bad, sizeof(int32_t));
	AL(a->part, 152 * sizeof(double));
	AL(a->loss_d, sizeof(double));
	AL(a->stage, 4 * n * sizeof(double));
	AL(a->twx, p->nx / 2 * cs); AL(a->twy, p->ny / 2 * cs);
	AL(a->green, (size_t) nh * p->ny * ts);
	AL(cosx, p->nx * sizeof(double)); AL(cosy, p->ny * sizeof(double));
#undef AL
	{
		// Green's function cosines (solver.c:257-278) and twiddles, as the
		// step's own solver builds them
		std::vector<double> cx(p->nx), cy(p->ny);
		for(int64_t i = 0; i < p->nx; i++) cx[i] = cos(2.0 * M_PI / p->nx * i);
		for(int64_t i = 0; i < p->ny; i++) cy[i] = cos(2.0 * M_PI / p->ny * i);
		cudaMemcpy(cosx, cx.data(), p->nx * sizeof(double), cudaMemcpyHostToDevice);
		cudaMemcpy(cosy, cy.data(), p->ny * sizeof(double), cudaMemcpyHostToDevice);
		if(a->f64) k_green<double><<<blocks_for(nh * p->ny), 256>>>(a->g.nx, a->g.ny, cosx, cosy,
				P<double>(a->green), green_scale<double>(a->g.nx, a->g.ny));
		else k_green<float><<<blocks_for(nh * p->ny), 256>>>(a->g.nx, a->g.ny, cosx, cosy,
				P<float>(a->green), green_scale<float>(a->g.nx, a->g.ny));
		for(int dim = 0; dim < 2; dim++)
		{
			int64_t m = dim == 0 ? p->nx : p->ny;
			std::vector<double2> tw(m / 2);
			std::vector<float2> tf(m / 2);
			for(int64_t i = 0; i < m / 2; i++)
			{
				double ang = -2.0 * M_PI * i / m;
				tw[i] = make_double2(cos(ang), sin(ang));
				tf[i] = make_float2((float) cos(ang), (float) sin(ang));
			}
			void *dst = dim == 0 ? a->twx : a->twy;
			if(a->f64) cudaMemcpy(dst, tw.data(), m / 2 * sizeof(double2), cudaMemcpyHostToDevice);
			else cudaMemcpy(dst, tf.data(), m / 2 * sizeof(float2), cudaMemcpyHostToDevice);
		}
	}
	{
		static PerDeviceOnce once;
		cudaError_t e = once.run([] {
			return set_max_dyn_smem({(const void *) k_rows_fwd<double>, (const void *) k_cols<double>,
					(const void *) k_rows_inv<double>, (const void *) k_rows_fwd_real<double>,
					(const void *) k_rows_fwd<float>, (const void *) k_cols<float>,
					(const void *) k_rows_inv<float>, (const void *) k_rows_fwd_real<float>},
					kFftMaxSmem);
		});
		if(e != cudaSuccess)
		{
			fprintf(stderr, "cpic_adj_create: kernel set-up failed: %s\n", cudaGetErrorString(e));
			r = CPIC_ECUDA;
			goto fail;
		}
	}
	if(cudaDeviceSynchronize() != cudaSuccess) { r = CPIC_ECUDA; goto fail; }
	cudaFree(cosx);
	cudaFree(cosy);
	*out = a;
	return CPIC_OK;
fail:
	cudaFree(cosx);
	cudaFree(cosy);
	cpic_adj_destroy(a);
	return r;
}

CPIC_API void cpic_adj_destroy(cpic_adj_t *a)
{
	if(!a) return;
	void *bufs[] = {a->x, a->y, a->ux, a->uy, a->pbx, a->pby, a->ubx, a->uby, a->ckpt, a->hist,
		a->histE, a->Ex, a->Ey, a->phi, a->rhob, a->Ebx, a->Eby, a->spec, a->rho, a->Ebfix,
		a->rsum, a->sc, a->src, a->work, a->tcnt, a->bad, a->part, a->loss_d, a->stage, a->twx, a->twy, a->green};
	for(void *b : bufs) if(b) cudaFree(b);
	for(int i = 0; i < 4; i++) if(a->ev[i]) cudaEventDestroy(a->ev[i]);
	if(a->st) cudaStreamDestroy(a->st);
	delete a;
}

CPIC_API int cpic_adj_forward(cpic_adj_t *a, const double *x, const double *y, const double *ux,
		const double *uy, double *loss)
{
	if(!a || !x || !y || !ux || !uy) return CPIC_EINVAL;
	int64_t n = a->n;
	const double *src[4] = {x, y, ux, uy};
	int32_t bad = 0;
	// (a state that is refused leaves the last run's as it is)
	if(cudaMemsetAsync(a->bad, 0, sizeof(int32_t), a->st) != cudaSuccess) return CPIC_ECUDA;
	for(int c = 0; c < 4; c++)
		if(cudaMemcpyAsync(a->stage + c * n, src[c], n * sizeof(double), cudaMemcpyHostToDevice, a->st)
				!= cudaSuccess)
			return CPIC_ECUDA;
	k_check<<<blocks_for(n), 256, 0, a->st>>>(n, a->stage, a->p.Lx, a->p.Ly, a->bad);
	if(cudaMemcpyAsync(&bad, a->bad, sizeof(int32_t), cudaMemcpyDeviceToHost, a->st) != cudaSuccess
			|| cudaStreamSynchronize(a->st) != cudaSuccess)
		return CPIC_ECUDA;
	if(bad) return CPIC_EINVAL;
	int r = a->f64 ? forward_impl<double>(a) : forward_impl<float>(a);
	if(r) return r;
	if(cudaGetLastError() != cudaSuccess) return CPIC_ECUDA;
	a->have_forward = true;
	if(loss) *loss = a->loss;
	return CPIC_OK;
}

CPIC_API int cpic_adj_backward(cpic_adj_t *a, double *gx, double *gy, double *gux, double *guy)
{
	if(!a) return CPIC_EINVAL;
	if(!a->have_forward) return CPIC_ESTATE;
	int r = a->f64 ? backward_impl<double>(a) : backward_impl<float>(a);
	if(r) return r;
	if(cudaGetLastError() != cudaSuccess) return CPIC_ECUDA;
	// the forward state was overwritten by the recompute: a new forward is
	// needed before the next backward
	a->have_forward = false;
	double *outs[4] = {gx, gy, gux, guy};
	int64_t n = a->n;
	for(int c = 0; c < 4; c++)
		if(outs[c] && cudaMemcpy(outs[c], a->stage + c * n, n * sizeof(double),
					cudaMemcpyDeviceToHost) != cudaSuccess)
			return CPIC_ECUDA;
	return CPIC_OK;
}

CPIC_API int cpic_adj_times(const cpic_adj_t *a, double *ms_forward, double *ms_backward)
{
	if(!a) return CPIC_EINVAL;
	if(ms_forward) *ms_forward = a->ms_fwd;
	if(ms_backward) *ms_backward = a->ms_bwd;
	return CPIC_OK;
}
