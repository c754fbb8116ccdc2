// bits_arith_check.cpp -- checks the arithmetic of cpic_gb300/csrc/cpic_bits.h
// (division by a constant) against the FP64 operations (CPU test driven by
// tests/test_bits_arith.py).  Prints the number of mismatches; 0 is a pass.
#include <cfenv>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "../cpic_gb300/csrc/cpic_bits.h"

using namespace cpic::bits;

static long bad = 0, checked = 0;

static bool same(double a, double b)
{
	return std::memcmp(&a, &b, 8) == 0 || (std::isnan(a) && std::isnan(b));
}

static void check_div(double a, double d)
{
	checked++;
	const double got = div_by(a, d, 1.0 / d), want = a / d;
	if(!same(got, want))
	{
		if(bad < 10)
			std::printf("div %.17g / %.17g: %.17g, want %.17g\n", a, d, got, want);
		bad++;
	}
}

int main()
{
	std::fesetround(FE_TONEAREST);
	std::mt19937_64 rng(4321);
	std::uniform_real_distribution<double> u(1.0, 2.0);
	auto any = [&](int lo, int hi) {
		const double s = (rng() & 1) ? 1.0 : -1.0;
		return s * std::ldexp(u(rng), lo + (int) (rng() % (uint64_t) (hi - lo)));
	};
	// node counts and cell sizes of real grids, and random divisors
	for(int nx = 4; nx <= 400; nx++)
		for(int ny : {4, 15, 40, 150, 400, 1920})
			for(int k = 0; k < 40; k++)
			{
				check_div(any(-200, 200), (double) nx * ny);
				check_div(any(-60, 60), 2 * (6.283185307179586 / nx));
			}
	for(int k = 0; k < 4000000; k++)
		check_div(any(-300, 300), std::fabs(any(-40, 40)));
	for(double d : {3.0, 0.1, 1e-3, 6.0e4})
		for(double a : {0.0, (double) INFINITY, (double) -INFINITY, (double) NAN, 1.0, d, -d, 3 * d})
			check_div(a, d);
	std::printf("%ld mismatches of %ld\n", bad, checked);
	return bad != 0;
}
