// The bookkeeping of a ring of asynchronous bulk copies, each of which completes on an mbarrier.
//
// Copy k of a ring of N lies in stage k % N and completes phase k / N of that stage's barrier.  Two rules keep such a ring sound: a
// barrier is armed for a copy only when the copy that it was armed for before has landed, and no CTA ends while a copy that it asked for is in
// flight.  (A barrier armed twice, or shared memory that belongs to another CTA when the copy lands, faults the GPU.)  In the
// ordinary course both follow from the waits: copy k + N is asked for behind the wait for copy k, and the last copies are waited for.
// Waits are bounded, though, and one that ran out says nothing about its copy.  So a thread whose wait ran out asks for nothing any more, and
// waits -- bounded again -- for those of its copies whose landing nobody has seen.
//
// No device code, so that the kernels' sequences can be run against made-up barriers on the CPU (tests/host/copy_ring.cpp).
#pragma once

#ifdef __CUDACC__
#define GL_RING __device__ __forceinline__
#else
#define GL_RING inline
#endif

namespace glb {

template <unsigned N>
struct CopyRing
{
	unsigned base = 0;     // number of the current run's copy 0 (a run: the copies of one weight tile, of one table)
	int most = 0;          // copies of the run that may be asked for: all of them, none once a wait ran out
	bool stopped = false;  // a wait ran out

	// A run of `count` copies, its first `depth` (at most N) of them.  copy(s, stage): arms the stage's barrier and asks for copy s.
	GL_RING void begin(int count) { most = stopped ? 0 : count; }
	template <class Copy>
	GL_RING void start(int depth, Copy copy)
	{
		for (int s = 0; s < depth && s < most; ++s) copy(s, (base + (unsigned)s) % N);
	}
	// The wait for copy s, before it is read.  wait(stage, parity): bounded, false when it ran out or another thread's has.
	// drain(lo, hi): bounded waits for the copies lo .. hi - 1 that do not look at other threads' state.
	template <class Wait, class Drain>
	GL_RING void await(int s, int depth, Wait wait, Drain drain)
	{
		const unsigned k = base + (unsigned)s;
		if (!stopped && !wait(k % N, (k / N) & 1u))
		{
			stopped = true;
			drain(k, base + (unsigned)(s + depth < most ? s + depth : most));
			most = 0;
		}
	}
	// Behind the reading of copy s: the copy that takes its place.
	template <class Copy>
	GL_RING void refill(int s, int depth, Copy copy)
	{
		if (s + depth < most) copy(s + depth, (base + (unsigned)(s + depth)) % N);
	}
	GL_RING void end(int count) { base += (unsigned)count; }

	// For a thread that asks and does not read, a run being one copy: whether that copy's stage is free.  read(stage, parity): the bounded wait
	// for the stage's readers, who give a stage back only when they have seen its copy land.
	template <class Read, class Drain>
	GL_RING bool may_ask(Read read, Drain drain)
	{
		if (!stopped && base >= N && !read(base % N, (base / N - 1) & 1u)) finish(true, drain);
		return !stopped;
	}
	// The same thread when its readers have read all copies, or given up.
	template <class Drain>
	GL_RING void finish(bool given_up, Drain drain)
	{
		if (stopped || !given_up) return;
		stopped = true;
		drain(base > N ? base - N : 0u, base);
	}
};

}  // namespace glb
