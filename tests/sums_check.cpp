// sums_check.cpp -- the bound of the mixed form's 32-bit weight sums
// (cpic_gb300/csrc/cpic_layout.h) against every interleaving of the fused
// kernel's warps (CPU test driven by tests/test_sums_bound.py).  Prints the
// number of failures; 0 is a pass.
//
// A warp takes, per chunk c: [the check of the sums]; the producer only: wait
// until every warp has released chunk c - 1, issue chunk c + 1; wait until
// chunk c is issued; P times: read a record (before the last one's push:
// release chunk c), push, deposit.  The check reads the sums before its
// barrier, so what it may miss are the deposits that other warps still owe
// when one of them arrives at it.
#include <algorithm>
#include <cstdio>
#include <set>
#include <tuple>
#include <vector>

#include "../cpic_gb300/csrc/cpic_layout.h"

using namespace cpic;

constexpr int kChunks = 7;

// A warp's place: chunk * (P + 3) + step; steps: 0 at the top (the check), 1
// the producer has issued, 2 the chunk has landed, 3 + k: deposit k done (the
// last one's wraps to the next chunk's top).  Released: the last record read.
struct Warps {
	int P;
	// places per chunk: top, issued, landed, deposits 1 .. P - 1, released
	int per() const { return 3 + P; }
	int chunk(int w) const { return w / per(); }
	int step(int w) const { return w % per(); }
	// deposits done (per thread)
	int done(int w) const { return chunk(w) * P + std::clamp(step(w) - 2, 0, P - 1); }
	bool released(int w, int c) const { return chunk(w) > c || (chunk(w) == c && step(w) == per() - 1); }
	// step per() - 1: chunk released, the last deposit still owed
};

// Most deposits per thread that a warp may owe of the chunks before the one at
// whose top another warp is.
static int most_owed(int P)
{
	const Warps m{P};
	typedef std::tuple<int, int, int> State;   // producer, another, a third warp
	std::set<State> seen{{0, 0, 0}};
	std::vector<State> todo{{0, 0, 0}};
	int most = 0;
	while(!todo.empty())
	{
		const State s = todo.back();
		todo.pop_back();
		const int at[3] = {std::get<0>(s), std::get<1>(s), std::get<2>(s)};
		// chunks issued: 0 at the start, c + 1 once the producer is past its
		// issue in chunk c
		const int issued = m.chunk(at[0]) + (m.step(at[0]) >= 1 ? 1 : 0);
		for(int w = 0; w < 3; w++)
		{
			const int c = m.chunk(at[w]), st = m.step(at[w]);
			if(st == 0)
				for(int o = 0; o < 3; o++)
					most = std::max(most, c * P - m.done(at[o]));
			if(c >= kChunks) continue;
			bool go = true;
			if(st == 0 && w == 0 && c >= 1)
				for(int o = 0; o < 3; o++) go = go && m.released(at[o], c - 1);
			if(st == 1) go = c <= issued;
			if(!go) continue;
			int n[3] = {at[0], at[1], at[2]};
			n[w]++;
			const State t(n[0], n[1], n[2]);
			if(seen.insert(t).second) todo.push_back(t);
		}
	}
	return most;
}

int main()
{
	long bad = 0;
	for(int P : {1, 2, 4})
	{
		const long long owed = (long long) most_owed(P) * kPushThreads;
		const long long interval = (long long) check_chunks(P) * chunk_of(P);
		// a check passes a node below 2^kCheckBits; owed deposits and those of
		// the chunks up to the next check follow, each of 2^kWeightBits at most
		const long long sum = (1ll << kCheckBits) - 1 + ((owed + interval) << kWeightBits);
		std::printf("P %d: %lld deposits owed, %d chunks between checks, sum up to 2^32 %+lld\n", P, owed,
				check_chunks(P), sum - (1ll << 32));
		if(sum >= 1ll << 32 || check_chunks(P) < 1) bad++;
	}
	std::printf("%ld failures\n", bad);
	return bad ? 1 : 0;
}
