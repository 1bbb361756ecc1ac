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
	// Copies land in front of the wait for them, those of the other stages whenever they like: `lazy` lets them fly until their own wait.
	bool wait(unsigned s, unsigned parity)
	{
		if (waits++ == other_at) abort = true;
		if (flying[s] && !late[s] && !abort) land(s);
		if ((done[s] & 1u) != parity) return true;
		abort = true;  // the limit has passed, or another thread's has
		return false;
	}
	void drain(unsigned s, unsigned parity)
	{
		if (flying[s]) land(s);
		if ((done[s] & 1u) == parity) ++early;  // not the phase of the stage's last copy
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
	r.start(tiles, 2, copy);
	for (int k = 0; k < tiles; ++k)
	{
		r.await(k, tiles, 2, [&](unsigned s, unsigned p) { return b.wait(s, p); });
		r.refill(k, tiles, 2, copy);
	}
	r.drain([&](unsigned s, unsigned p) { b.drain(s, p); });
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
	return bad != 0;
}
