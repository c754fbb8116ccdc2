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

int main()
{
	check_arrivals();
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
