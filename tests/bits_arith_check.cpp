// bits_arith_check.cpp -- checks the arithmetic of cpic_gb300/csrc/cpic_bits.h
// (division by a constant, products, 1 - x, the offset in a cell and the
// fixed-point split on integers) against the FP64 operations (CPU test driven by
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

static void check_mul(double a, double b)
{
	Pos p, q;
	if(!pos_of(a, p) || !pos_of(b, q))
		return;
	const Pos r = pos_mul(p, q);
	if(!pos_normal(r))
		return;
	checked++;
	if(!same(pos_val(r), a * b))
	{
		if(bad < 10)
			std::printf("mul %.17g %.17g: %.17g, want %.17g\n", a, b, pos_val(r), a * b);
		bad++;
	}
}

static void check_one_minus(double a)
{
	Pos p;
	if(!pos_of(a, p) || p.e >= 0)
		return;
	checked++;
	const Pos r = pos_one_minus(p);
	if(!same(pos_val(r), 1.0 - a) || !(r.h >> 31) || (r.l & 0x7ff))
	{
		if(bad < 10)
			std::printf("1 - %.17g: %.17g, want %.17g\n", a, pos_val(r), 1.0 - a);
		bad++;
	}
}

static long rel_taken = 0, rel_all = 0;

static void check_rel(double x, double dx, double idx)
{
	Pos p, d, i, rel;
	int i0 = -1;
	rel_all++;
	if(!pos_of(x, p) || !pos_of(dx, d) || !pos_of(idx, i) || !pos_rel(p, d, i, i0, rel))
		return;
	rel_taken++;
	checked++;
	const double start = std::floor(x * idx);
	const double grid = x - start * dx;
	const double want = grid * idx;
	if(i0 != (int) start || !same(pos_val(rel), want))
	{
		if(bad < 10)
			std::printf("rel %.17g dx %.17g: %d %.17g, want %d %.17g\n", x, dx, i0, pos_val(rel),
					(int) start, want);
		bad++;
	}
}

static void check_split(double v, int lo_exp)
{
	Pos p;
	long long hi, lo;
	for(int neg = 0; neg < 2; neg++)
	{
		if(!pos_of(v, p) || !pos_split(p, neg != 0, lo_exp, hi, lo))
			continue;
		checked++;
		const double sv = neg ? -v : v;
		const long long rhi = std::llrint(sv);
		const long long rlo = std::llrint((sv - (double) rhi) * std::ldexp(1.0, lo_exp));
		if(hi != rhi || lo != rlo)
		{
			if(bad < 10)
				std::printf("split %.17g exp %d: %lld %lld, want %lld %lld\n", sv, lo_exp, hi, lo, rhi, rlo);
			bad++;
		}
	}
}

static void check_frac(double x, double idx)
{
	Pos p, i, f;
	int i0 = -1;
	if(!pos_of(x, p) || !pos_of(idx, i) || !pos_frac(p, i, i0, f))
		return;
	checked++;
	// floor of the exact product: of the rounded one, less one where that
	// rounded up to an integer
	double fl = std::floor(x * idx);
	if(std::fma(x, idx, -fl) < 0.0)
		fl -= 1.0;
	const double want = std::fma(x, idx, -fl);
	if(i0 != (int) fl || !same(pos_val(f), want))
	{
		if(bad < 10)
			std::printf("frac %.17g * %.17g: %d %.17g, want %d %.17g\n", x, idx, i0, pos_val(f), (int) fl, want);
		bad++;
	}
}

static void check_rint(double v)
{
	Pos p;
	long long got;
	for(int neg = 0; neg < 2; neg++)
	{
		if(!pos_of(v, p) || !pos_rint(p, neg != 0, got))
			continue;
		checked++;
		const long long want = std::llrint(neg ? -v : v);
		if(got != want)
		{
			if(bad < 10)
				std::printf("rint %.17g: %lld, want %lld\n", v, got, want);
			bad++;
		}
	}
}

static void check_mul24(float a, double b, float c)
{
	Pos p, q, r;
	if(!pos_of(a, p) || !pos_of(c, r) || !pos_of(b, q))
		return;
	checked++;
	const double want = (double) a * b, want2 = (double) a * (double) c;
	if(!same(pos_val(pos_mul24(p, q)), want) || !same(pos_val(pos_mul24x24(p, r)), want2))
	{
		if(bad < 10)
			std::printf("mul24 %.9g %.17g %.9g\n", a, b, c);
		bad++;
	}
}

// doubles whose products and differences come near ties: few significant
// bits, runs of ones, a bit at the end
static double sparse(std::mt19937_64 &rng)
{
	uint64_t m = 1ull << 52;
	for(int k = (int) (rng() % 4); k >= 0; k--)
		m |= 1ull << (rng() % 52);
	if(rng() & 1)
		m = (1ull << 53) - (m & ((1ull << 52) - 1)) - 1;
	return (double) m;
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
	for(int k = 0; k < 6000000; k++)
	{
		check_mul(std::fabs(any(-200, 200)), std::fabs(any(-200, 200)));
		check_mul(std::ldexp(sparse(rng), -52), std::ldexp(sparse(rng), -60));
		const double a = u(rng) - 1.0;
		check_one_minus(a);
		check_one_minus(std::ldexp(a, -(int) (rng() % 70)));
		check_one_minus(std::ldexp(sparse(rng), -53 - (int) (rng() % 70)));
	}
	for(double a : {0.5, 0.25, std::nextafter(0.5, 0.0), std::nextafter(0.5, 1.0), std::nextafter(1.0, 0.0),
			std::ldexp(1.0, -53), std::ldexp(1.0, -54), std::ldexp(1.0, -64), std::ldexp(1.0, -65),
			std::ldexp(3.0, -54), std::ldexp(3.0, -55), std::ldexp(1.0, -300)})
		check_one_minus(a);
	// positions in boxes of real grids: random, next to cell edges, at the
	// ends
	for(int nx : {4, 15, 25, 48, 64, 150, 250, 512, 1000, 1920, 2048, 16384})
		for(double L : {6.283185307179586, 1.0, 12.566370614359172, 3.7})
		{
			const double dx = L / nx, idx = 1.0 / dx;
			for(int k = 0; k < 40000; k++)
			{
				check_rel((u(rng) - 1.0) * L, dx, idx);
				double e = (double) (rng() % (uint64_t) (nx + 1)) * dx;
				check_rel(e, dx, idx);
				for(int n = 0; n < 3; n++)
					check_rel(e = std::nextafter(e, (k & 1) ? 1e300 : 0.0), dx, idx);
				check_rel(std::ldexp(u(rng), -(int) (rng() % 60)), dx, idx);
			}
			check_rel(L, dx, idx);
		}
	for(int nx : {4, 16, 64, 128, 256, 4096})
		for(double L : {6.283185307179586, 1.0, 3.7})
			for(int k = 0; k < 100000; k++)
			{
				const double idx = 1.0 / (L / nx);
				check_frac((u(rng) - 1.0) * L, idx);
				check_frac(std::nextafter((double) (rng() % (uint64_t) nx) * (L / nx), (k & 1) ? 1e9 : 0.0), idx);
				check_frac(std::ldexp(u(rng), -(int) (rng() % 80)), idx);
			}
	for(int k = 0; k < 3000000; k++)
	{
		check_rint(std::ldexp(u(rng), (int) (rng() % 66) - 4));
		check_mul24((float) std::ldexp(u(rng), -(int) (rng() % 30)), any(-40, 40) * ((k & 1) ? 1.0 : -1.0),
				(float) std::ldexp(u(rng), -(int) (rng() % 60)));
	}
	for(long long k = 0; k < 5000; k++)
		for(double d : {0.0, 0.5, 0.25, 0.75})
		{
			check_rint((double) k + d);
			check_rint(std::nextafter((double) k + d, 1e300));
			check_rint(std::nextafter((double) k + d, 0.0));
		}
	const int exps[] = {1, 7, 20, 30, 37, 39, 45, 52, 60, 61, 62};
	for(long long k = 1; k <= 4096; k++)
		for(int sc = -12; sc <= 45; sc++)
			for(int e : exps)
			{
				const double b = std::ldexp((double) k, sc);
				check_split(b, e);
				check_split(b + 0.5, e);
				check_split(std::nextafter(b + 0.5, 1e300), e);
				check_split(std::nextafter(b + 0.5, 0.0), e);
			}
	for(int k = 0; k < 4000000; k++)
		check_split(std::ldexp(u(rng), (int) (rng() % 62)), exps[k % 11]);
	// the fast path takes nearly every position (not those in a box's first
	// cell next to 0, nor offsets that round to 0 or 1)
	if(rel_taken < rel_all / 2)
	{
		std::printf("only %ld of %ld offsets taken\n", rel_taken, rel_all);
		bad++;
	}
	for(double d : {3.0, 0.1, 1e-3, 6.0e4})
		for(double a : {0.0, (double) INFINITY, (double) -INFINITY, (double) NAN, 1.0, d, -d, 3 * d})
			check_div(a, d);
	std::printf("%ld mismatches of %ld\n", bad, checked);
	return bad != 0;
}
