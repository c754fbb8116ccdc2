// cpic_layout.h -- the tile layout's host rules and the index arithmetic that
// depends on them.  Plain C++ (host and device), so a CPU test checks the
// rules' results over the whole range of grids against the ranges that the
// kernels' indices need.
#pragma once
#include <algorithm>
#include <cstdint>

#include "cpic_bits.h"

namespace cpic {

// Block shape of the fused particle kernel (build-time knobs).
#ifndef CPIC_PUSH_THREADS
#define CPIC_PUSH_THREADS 256
#endif
#ifndef CPIC_PPT
#define CPIC_PPT 2
#endif
constexpr int kPushThreads = CPIC_PUSH_THREADS;
// Particles per thread per chunk: the default, and the compiled instances of
// the fused kernel a context may choose from (the autotuner times them).
constexpr int kPPT = CPIC_PPT;
constexpr int kPPTChoices[] = {1, 2, 4};
constexpr int kWeightBits = 18;
// Particles per chunk with P particles per thread.
CPIC_HD constexpr int chunk_of(int P) { return kPushThreads * P; }
// 32-bit (unsigned) shared weight sums: a node gains at most 2^kWeightBits
// per particle.  A check every check_chunks(P) chunks folds the sums into the
// grid when it sees a node at 2^kCheckBits or above.  It reads the sums before
// its barrier, when other warps may still owe deposits of the chunks before:
// a chunk is issued once every warp has released the one that was in its
// buffer, which a warp does before the last push, so a warp can be two chunks
// and one push behind another.  A node that the check passes is therefore
// below 2^kCheckBits plus those deposits, and the interval leaves room for
// them: every sum stays below 2^32.  A check costs a block barrier and a pass
// over the sums (two-stream 2048 x 2048 benchmark: every 8 chunks, with a limit
// of 2^30, took 1.4 % longer over the whole kernel than every 31).
constexpr int kCheckBits = 27;
CPIC_HD constexpr int owed_deposits(int P) { return 2 * chunk_of(P) + kPushThreads; }
CPIC_HD constexpr int check_chunks(int P)
{
	return (int) (((((1ll << 32) - (1ll << kCheckBits)) >> kWeightBits) - owed_deposits(P)) / chunk_of(P));
}
static_assert(check_chunks(4) >= 1, "chunk too large for 32-bit weight sums");

// Periodic wrap for any extent, i in [-n, 2n).
CPIC_HD int wrapn(int i, int n)
{
	if(i < 0) i += n;
	else if(i >= n) i -= n;
	return i;
}

namespace layout {

// Along one side of n nodes: the node held at place l (0 .. T) of the field
// tile whose first node is t0 (a multiple of the tile size T, below n).  T < 2n
// keeps t0 + l below 2n: with one tile t0 is 0, with more T is below n.
CPIC_HD int field_node(int t0, int l, int n)
{
	return wrapn(t0 + l, n);
}

inline int64_t tiles_of(int64_t nx, int64_t ny, int T)
{
	return ((nx + T - 1) / T) * ((ny + T - 1) / T);
}

// The library's tile size for n evenly spread particles of one species: the largest of 32,
// 16, 8 and 4 cells whose tiles keep the SMs busy to the end.  One block takes
// a tile, an SM holds 5 or 6 of them, and a block alone on an SM works off
// its particles at a fraction of the SM's rate, so: over two waves of tiles
// (2048), whatever they hold; about a wave (912) if none takes long (8192
// particles, FP64 2048: its particles take four times as long); a tile per
// SM if each is short; or next to nothing per tile, where launch latency is
// all there is.  Smaller tiles than that only add edges.  Measured (particle
// kernel, us per step, mixed unless said): 128 x 128 with 128 per cell,
// 16-cell tiles 113, 8-cell 40, 4-cell 31; 256 x 256 with 32, 16-cell 40,
// 8-cell 31, 4-cell 38; 512 x 512 with 4, 16-cell 25, 8-cell 31, with 100,
// 16-cell 241, 8-cell 222; 1024 x 1024 with 25, 32-cell 252, 16-cell 233;
// 2048 x 2048 with 6, 64-cell 402, 32-cell 254, 16-cell 324; FP64 64 x 64
// with 64, 8-cell 111, 4-cell 46; FP64 512 x 512 with 16, 16-cell 723,
// 8-cell 690, 4-cell 824.
//
// A tile below twice the shorter side at most (field_node): its first power of
// two that covers that side, beyond which a tile only holds places of no cell.
inline int auto_tile(int64_t nx, int64_t ny, bool f64, int64_t n)
{
	int T = 32;
	while(T >= 2 * nx || T >= 2 * ny) T >>= 1;
	for(; T > 4; T >>= 1)
	{
		const int64_t tiles = tiles_of(nx, ny, T);
		const int64_t per = n / tiles;
		if(tiles >= 2048 || (tiles >= 912 && per <= (f64 ? 2048 : 8192))
				|| (tiles >= 152 && per <= (f64 ? 512 : 1024)) || per <= 128)
			return T;
	}
	return 4;
}

// How evenly a species fills the tiles: for tiles of 4, 8, 16 and 32 cells
// (index log2 T - 2) the number of equal tiles with the same load as a particle
// sees on average, (sum c)^2 / (sum c^2 - sum c) for tiles of c particles (the
// subtraction takes out chance: evenly scattered particles give the number of
// tiles).
struct Spread { double tiles[4]; };
constexpr int kSpreadBin = 4;                  // cells per side of a counted bin

inline Spread spread(int64_t nx, int64_t ny, double count, const double squares[4])
{
	Spread e;
	for(int k = 0; k < 4; k++)
	{
		e.tiles[k] = (double) tiles_of(nx, ny, kSpreadBin << k);
		if(squares[k] > count)
			e.tiles[k] = std::min(e.tiles[k], count * count / (squares[k] - count));
	}
	return e;
}

// Time of the particle kernel on n unevenly spread particles, us: a share for
// every tile, most of them empty, over the blocks that the GPU holds, and the
// heavy tiles' particles, which one block works off.  Fitted to a sweep of 140
// loads (boxes, a bell, half of the particles in a tenth of the grid, a sine;
// 64^2 to 2048^2 cells, 0.26 to 8 million particles, 4 tile sizes each).
inline double uneven_cost(int64_t nx, int64_t ny, bool f64, int64_t n, int T, double tiles)
{
	const double all = (double) tiles_of(nx, ny, T) / 912 * (1.0 + T * T / 800.0);
	const double load = (double) n / std::max(tiles, 1.0);
	return f64 ? 10.0 + 4.6 * all + 61e-6 * n + 32e-3 * load : 9.0 + 3.1 * all + 6.8e-6 * n + 5.8e-3 * load;
}

// The tile size for n particles spread as e says: that of an even load, unless
// fewer than three quarters of those tiles carry it and a smaller tile costs at
// most 0.85 as much by uneven_cost.  Particle kernel, us, with the even load's
// tile, with the tile chosen here and with the best of the four: mixed 512 x 512,
// 4 million in a fifth of each side 299, 83, 83; a bell of a tenth of the side
// 189, 83, 83; 1024 x 1024, 2 million in a fifth 145, 56, 56; 2048 x 2048, 8
// million, a bell 122 (kept), 122; FP64 256 x 256, 2 million in a fifth 1148,
// 348, 348; 1024 x 1024, 8 million, half in a tenth 585 (kept), 585.  Over the
// sweep the worst choice is 1.15 times the best (27 us instead of 24).
inline int uneven_tile(int64_t nx, int64_t ny, bool f64, int64_t n, const Spread &e)
{
	int T = auto_tile(nx, ny, f64, n), k = 0;
	while(kSpreadBin << k < T) k++;
	if(e.tiles[k] >= 0.75 * (double) tiles_of(nx, ny, T))
		return T;
	double least = 0.85 * uneven_cost(nx, ny, f64, n, T, e.tiles[k]);
	while(--k >= 0)
	{
		const double cost = uneven_cost(nx, ny, f64, n, kSpreadBin << k, e.tiles[k]);
		if(cost < least)
		{
			least = cost;
			T = kSpreadBin << k;
		}
	}
	return T;
}

// Room for arrivals in percent of a tile's particles, for a species that moves
// `move` cells per step on average (|dx| + |dy|): at most move / T of the
// particles leave their tile of T cells in a step, and as many come in where
// the density is even; a tenth more than that.  At least a quarter, or a
// quarter of the slack that overflows have raised.  Without room for them most
// movers go through the spill list, which holds an eighth of a species (64 x
// 64, 64 per cell, two beams of 2.5 cells per step in 4-cell tiles: the list
// is full in the second step, and tiles overflow before the next check).
inline int arrivals_pct(double move, int T, int slack_pct)
{
	const double leave = move < T ? move / T : 1.0;
	const int pct = (int) (110.0 * leave) + 1;
	return std::max(std::max(25, slack_pct / 4), pct);
}

} // namespace layout
} // namespace cpic
