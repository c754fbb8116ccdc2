// layout_check.cpp -- the tile sizes that cpic_gb300/csrc/cpic_layout.h chooses
// against the index ranges of the kernels that use them (CPU test driven by
// tests/test_layout.py).  Prints the number of failures; 0 is a pass.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "../cpic_gb300/csrc/cpic_layout.h"

using namespace cpic;

static long bad = 0;

// Every node that the field tiles of one side hold lies on it, and is the
// periodic image of its place.
static void check_side(int n, int T, int nx, int ny, long long count)
{
	for(int t0 = 0; t0 < n; t0 += T)
		for(int l = 0; l <= T; l++)
		{
			const int at = layout::field_node(t0, l, n);
			if(at >= 0 && at < n && at == (t0 + l) % n) continue;
			if(bad++ < 10)
				std::printf("%d x %d, %lld particles: tile %d at %d, place %d is node %d of %d\n", nx, ny,
						count, T, t0, l, at, n);
			return;
		}
}

static void check_grid(int nx, int ny)
{
	for(int f64 = 0; f64 < 2; f64++)
		for(long long per : {0, 1, 2, 4, 8, 16, 64, 300, 5000})
		{
			const long long count = per * nx * ny + (per == 0 ? 3 : 0);
			const int T = layout::auto_tile(nx, ny, f64 != 0, count);
			if(T != 4 && T != 8 && T != 16 && T != 32)
			{
				bad++;
				std::printf("tile %d\n", T);
				continue;
			}
			check_side(nx, T, nx, ny, count);
			check_side(ny, T, nx, ny, count);
		}
}

// Room for the movers of a plasma at any speed, never less than a quarter or
// a quarter of the slack.
static void check_arrivals()
{
	for(int T = 1; T <= 64; T *= 2)
		for(int slack : {0, 25, 50, 100, 200, 1000})
			for(double move : {0.0, 1e-300, 0.01, 0.3, 1.0, 2.5, 3.999, 4.0, 12.0, 63.9, 64.1, 32768.0})
			{
				const int pct = layout::arrivals_pct(move, T, slack);
				const double leave = std::min(1.0, move / T);
				if(pct >= 25 && pct >= slack / 4 && pct >= 109.99 * leave && pct <= std::max(111, slack / 4))
					continue;
				bad++;
				std::printf("room for arrivals: %d %% at %g cells per step, T %d, slack %d\n", pct, move, T, slack);
			}
}

// Uneven loads: the tile of an even load or a smaller one, whatever the spread;
// that of an even load where the load is even.
static void check_uneven(int nx, int ny)
{
	for(int f64 = 0; f64 < 2; f64++)
		for(long long per : {0, 1, 4, 16, 300})
			for(double share : {1e-6, 0.01, 0.1, 0.3, 0.7, 0.9, 1.0})
			{
				const long long n = per * nx * ny;
				layout::Spread e;
				for(int k = 0; k < 4; k++)
					e.tiles[k] = std::max(1.0, share * layout::tiles_of(nx, ny, 4 << k));
				const int even = layout::auto_tile(nx, ny, f64 != 0, n), T = layout::uneven_tile(nx, ny, f64 != 0, n, e);
				if((T == 4 || T == 8 || T == 16 || T == 32) && T <= even && (share < 0.75 || T == even)) continue;
				bad++;
				std::printf("%d x %d, %lld particles, share %g: tile %d, even %d\n", nx, ny, n, share, T, even);
			}
	// a count and its squares: even tiles, one tile, no particles
	const double all = (double) layout::tiles_of(nx, ny, 4), c = 1000.0;
	const double even[4] = {all * c * c, 0, 0, 0}, one[4] = {all * c * all * c, 0, 0, 0}, none[4] = {0, 0, 0, 0};
	const double a = layout::spread(nx, ny, all * c, even).tiles[0], b = layout::spread(nx, ny, all * c, one).tiles[0];
	if(a > 0.99 * all && a <= all && b >= 1.0 && b < 1.1 && layout::spread(nx, ny, 0, none).tiles[0] == all) return;
	bad++;
	std::printf("%d x %d: spread %g and %g of %g\n", nx, ny, a, b, all);
}

// Measured loads (particle kernel, us, tiles of 4, 8, 16 and 32 cells; the even
// tiles of the same load): the choice is within a fifth of the best.
static void check_measured()
{
	struct Load { int f64, n; double count, us[4], tiles[4]; };
	const Load loads[] = {
		{0, 256, 500e3, {24.9, 63.9, 156.1, 541.8}, {171, 45, 12, 4}},          // a fifth of each side
		{0, 256, 500e3, {22.3, 41.9, 85.2, 227.9}, {515, 130, 33, 9}},          // a bell
		{0, 256, 2e6, {68.6, 164.7, 594.1, 2032.6}, {171, 45, 12, 4}},
		{0, 512, 1e6, {55.7, 28.1, 70.0, 164.9}, {2061, 516, 130, 33}},
		{0, 512, 1e6, {49.0, 23.6, 27.2, 57.4}, {4160, 1045, 272, 69}},         // half of each side
		{0, 512, 4e6, {83.2, 121.8, 298.4, 1106.1}, {672, 171, 45, 12}},
		{0, 512, 4e6, {98.3, 55.9, 61.1, 156.8}, {9843, 2473, 633, 169}},       // a sine
		{0, 1024, 2e6, {157.5, 55.8, 65.1, 145.1}, {2650, 672, 171, 45}},
		{0, 1024, 8e6, {335.8, 143.0, 87.6, 148.8}, {20324, 5093, 1298, 328}},  // half of them in a tenth
		{0, 2048, 8e6, {897.4, 287.7, 135.8, 121.9}, {32946, 8237, 2060, 516}},
		{0, 512, 4e6, {92.2, 55.4, 50.6, 65.3}, {16383, 4096, 1024, 256}},      // even
		{1, 256, 2e6, {348.3, 1149.7, 4337.6, 16791.2}, {171, 45, 12, 4}},
		{1, 512, 1e6, {157.7, 124.5, 382.5, 1294.3}, {2061, 516, 130, 33}},
		{1, 512, 4e6, {420.6, 307.5, 574.2, 2328.2}, {5086, 1297, 327, 89}},
		{1, 1024, 8e6, {1070.2, 708.8, 585.3, 1066.3}, {20324, 5093, 1298, 328}},
		{1, 2048, 8e6, {1348.3, 755.0, 780.0, 1370.5}, {10552, 2651, 672, 171}},
	};
	for(const Load &l : loads)
	{
		layout::Spread e;
		for(int k = 0; k < 4; k++) e.tiles[k] = l.tiles[k];
		const int T = layout::uneven_tile(l.n, l.n, l.f64 != 0, (long long) l.count, e);
		const double us = l.us[T == 4 ? 0 : T == 8 ? 1 : T == 16 ? 2 : 3], least = *std::min_element(l.us, l.us + 4);
		if(us <= 1.2 * least) continue;
		bad++;
		std::printf("%d x %d, %g particles: tile %d, %g us of %g\n", l.n, l.n, l.count, T, us, least);
	}
}

int main()
{
	check_arrivals();
	check_measured();
	for(int n : {4, 5, 16, 33, 64, 100, 250, 512, 1000, 4096})
		for(int m : {4, 7, 64, 150, 512, 2048}) check_uneven(n, m);
	std::vector<int> sides;
	for(int n = 4; n <= 70; n++) sides.push_back(n);
	for(int n = 128; n <= 16384; n *= 2)
		for(int d : {-1, 0, 1})
			if(n + d <= 16384) sides.push_back(n + d);
	for(int nx : sides)
		for(int ny : sides)
			if(std::min(nx, ny) <= 70) check_grid(nx, ny);
	for(int n : sides) check_grid(n, n);
	std::printf("%ld failures\n", bad);
	return bad ? 1 : 0;
}
