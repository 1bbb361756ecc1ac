// The bookkeeping of a ring of asynchronous bulk copies, each of which completes on an mbarrier.
//
// Copy k of a ring of N lies in stage k % N and completes phase k / N of that stage's barrier.  Two rules keep such a ring sound: a
// barrier is armed for a copy only when the copy that it was armed for before has landed, and no CTA ends while a copy that it asked for is in
// flight.  (A barrier armed twice, or shared memory that belongs to another CTA when the copy lands, faults the GPU.)  In the
// ordinary course both follow from the waits: copy k + N is asked for behind the wait for copy k, and the last copies are waited for.
// Waits are bounded, though, and one that ran out says nothing about its copy.  So a thread whose wait ran out asks for nothing any more,
// and before the CTA ends whoever asks waits -- bounded again -- for those of its copies whose landing nobody has seen.
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
	unsigned base = 0;        // number of the current run's copy 0 (a run: the copies of one weight tile, of one table)
	bool stopped = false;     // a wait ran out: nothing more is asked for, and nothing waited for except by drain
	unsigned lo = 0, hi = 0;  // then: the copies asked for whose landing nobody has seen

	// Copy s of the run.  copy(s, stage): arms the stage's barrier and asks for the copy.
	template <class Copy>
	GL_RING void ask(int s, Copy copy)
	{
		if (!stopped) copy(s, (base + (unsigned)s) % N);
	}
	// The first copies of a run of `count`, `depth` (at most N) of them.
	template <class Copy>
	GL_RING void start(int count, int depth, Copy copy)
	{
		for (int s = 0; s < depth && s < count; ++s) ask(s, copy);
	}
	// The wait for copy s, before it is read.  wait(stage, parity): bounded, false when it ran out or another thread's has.
	template <class Wait>
	GL_RING void await(int s, int count, int depth, Wait wait)
	{
		const unsigned k = base + (unsigned)s;
		if (!stopped && !wait(k % N, (k / N) & 1u)) stop(k, base + (unsigned)(s + depth < count ? s + depth : count));
	}
	// Behind the reading of copy s: the copy that takes its place.
	template <class Copy>
	GL_RING void refill(int s, int count, int depth, Copy copy)
	{
		if (s + depth < count) ask(s + depth, copy);
	}
	GL_RING void end(int count) { base += (unsigned)count; }

	// For a thread that asks and does not read, a run being one copy: whether that copy's stage is free.  read(stage, parity): the bounded wait
	// for the stage's readers.  Readers whose own wait ran out give their stage back with the copy still in flight, so
	// that given_up() -- somebody's wait has run out -- is looked at behind the wait.
	template <class Read, class GivenUp>
	GL_RING bool may_ask(Read read, GivenUp given_up)
	{
		if (!stopped && base >= N && (!read(base % N, (base / N - 1) & 1u) || given_up())) stop(base - N, base);
		return !stopped;
	}
	// The same thread at the end, when its readers have read or given up.
	GL_RING void finish(bool given_up)
	{
		if (!stopped && given_up) stop(base > N ? base - N : 0, base);
	}

	// The end of the CTA.  landed(stage, parity): a bounded wait that does not look at other threads' state.
	template <class Landed>
	GL_RING void drain(Landed landed) const
	{
		if (stopped)
#ifdef __CUDACC__
#pragma unroll 1
#endif
			for (unsigned k = lo; k < hi; ++k) landed(k % N, (k / N) & 1u);
	}
	GL_RING void stop(unsigned lo_, unsigned hi_)
	{
		stopped = true;
		lo = lo_;
		hi = hi_;
	}
};

}  // namespace glb
