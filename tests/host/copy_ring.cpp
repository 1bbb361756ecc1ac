// The sequences of copies and waits of the kernels that keep a ring of bulk copies (copy_ring.h), on made-up barriers.  One copy is so
// late that the wait for it runs out, or another thread's wait runs out at some step; then no barrier may be armed while its copy is in
// flight, and no copy may be in flight when the sequence has ended.  Status 0: all sequences sound.
#include "copy_ring.h"

#include <cstdio>

using namespace glb;

// Stages' barriers with the parity rule of mbarrier.try_wait, and the copies in flight on them.
template <unsigned N>
struct Barriers
{
	unsigned done[N] = {};       // phases completed
	bool flying[N] = {}, late[N] = {};
	bool abort = false;          // somebody's wait has run out
	int copies = 0, late_copy, other_at, waits = 0, twice = 0, early = 0;
	Barriers(int late_copy_, int other_at_) : late_copy(late_copy_), other_at(other_at_) {}
	void arm(unsigned s)
	{
		if (flying[s]) ++twice;
		flying[s] = true;
		late[s] = copies++ == late_copy;
	}
	void land(unsigned s)
	{
		flying[s] = false;
		++done[s];
	}
	// (copies land in front of the wait for them, no sooner)
	bool wait(unsigned s, unsigned parity)
	{
		if (waits++ == other_at) abort = true;
		if (flying[s] && !late[s] && !abort) land(s);
		if ((done[s] & 1u) != parity) return true;
		abort = true;  // the limit has passed, or another thread's has
		return false;
	}
	void drain(unsigned lo, unsigned hi)
	{
		for (unsigned k = lo; k < hi; ++k)
		{
			if (flying[k % N]) land(k % N);
			if ((done[k % N] & 1u) == ((k / N) & 1u)) ++early;  // a wait for a copy that nobody asked for
		}
	}
	int faults() const
	{
		int left = 0;
		for (unsigned s = 0; s < N; ++s) left += flying[s];
		return twice + early + left;
	}
};

// A table's tiles (transform_tiles_kernel; the thread that asks).
static int table(int tiles, int late, int other)
{
	Barriers<2> b(late, other);
	CopyRing<2> r;
	auto copy = [&](int, unsigned stage) { b.arm(stage); };
	r.begin(tiles);
	r.start(2, copy);
	for (int k = 0; k < tiles; ++k)
	{
		r.await(k, 2, [&](unsigned s, unsigned p) { return b.wait(s, p); }, [&](unsigned lo, unsigned hi) { b.drain(lo, hi); });
		r.refill(k, 2, copy);
	}
	return b.faults();
}

// The gradient phase of the whole-window kernel, a warp's ring: runs of `steps` copies, up to three or (a narrow layer's) two in flight;
// the warp goes through all its steps whatever the waits said.
static int gradient(int steps, int late, int other)
{
	Barriers<3> b(late, other);
	CopyRing<3> r;
	auto copy = [&](int, unsigned stage) { b.arm(stage); };
	for (int run = 0; run < 3; ++run)
	{
		const int depth = run == 1 ? 2 : 3;
		r.begin(steps);
		r.start(depth, copy);
		for (int s = 0; s < steps; ++s)
		{
			r.await(s, depth, [&](unsigned st, unsigned p) { return b.wait(st, p); }, [&](unsigned lo, unsigned hi) { b.drain(lo, hi); });
			r.refill(s, depth, copy);
		}
		r.end(steps);
	}
	return b.faults();
}

// The same kernel's weight tiles: one thread asks, as far ahead as the ring allows; another reads, stops waiting once its wait has run out and
// gives no stage back from then on.
static int weights(int count, int late, int other)
{
	const int tiles = 3 * count;
	Barriers<3> b(late, other);
	CopyRing<3> r;
	unsigned read[3] = {};  // phases of the stages' "read" barriers
	int consumed = 0;
	bool dead = false;
	auto drain = [&](unsigned lo, unsigned hi) { b.drain(lo, hi); };
	auto reader = [&]() {
		const unsigned st = consumed % 3;
		if (!dead && !b.wait(st, (consumed / 3) & 1)) dead = true;
		read[st] += !dead;
		++consumed;
	};
	for (int k = 0; k < tiles; ++k)
	{
		if (r.may_ask(
		        [&](unsigned st, unsigned p) {
			        while ((read[st] & 1u) == p)
			        {
				        if (b.abort) return false;
				        reader();
			        }
			        return true;
		        },
		        drain))
		{
			b.arm(r.base % 3);
			r.end(1);
		}
	}
	while (consumed < tiles) reader();
	r.finish(b.abort, drain);
	return b.faults();
}

template <class F>
static int sweep(const char* name, int most, F run)
{
	int bad = 0, n = 0;
	for (int count = 0; count <= most; ++count)
		for (int late = -1; late < 3 * count; ++late)
			for (int other = -1; other < 3 * count; ++other, ++n) bad += run(count, late, other) != 0;
	if (bad) printf("%s: %d of %d sequences arm a barrier twice or leave a copy in flight\n", name, bad, n);
	return bad;
}

int main()
{
	int bad = 0;
	bad += sweep("table", 9, table);
	bad += sweep("gradient", 9, gradient);
	bad += sweep("weight tiles", 9, weights);
	return bad != 0;
}
