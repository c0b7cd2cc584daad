// streams.h -- the two-halves schedule: a wave's solves as two chains of steps
// on two streams.
#pragma once

#include <cuda_runtime.h>

namespace gbfwi {

// The schedule's second stream, per (device, host thread, caller's stream), with
// its fork / join events.  Kept for the process (a graph capture records work on
// it) and freed by gb_fwi2d_release_caches.
struct SideStream {
    cudaStream_t s = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaStream_t caller = nullptr;
};

// A thread has at most this many on a device; callers' streams beyond share them.
constexpr int kMaxSideStreams = 8;

// The side stream of this thread's work on `caller`, on the current device: its
// own, so that calls on different streams do not queue behind one another.
// Created on first use unless `create` is false (a stream being captured), which
// takes any that the thread has: a capture records on it and queues nothing.
const SideStream *side_stream(cudaStream_t caller, bool create);

// A wave's two halves (or, without a side stream, the whole wave): the solves
// [0, nlo) on st and [nlo, nres) on the side stream, between fork() and join().
struct Halves {
    const SideStream *side;
    cudaStream_t st;
    int nlo, nres;
    Halves(const SideStream *side, cudaStream_t st, int nres)
        : side(side), st(st), nlo(side ? nres / 2 : nres), nres(nres)
    {
    }
    void fork() const
    {
        if (!side) return;
        cudaEventRecord(side->fork, st);
        cudaStreamWaitEvent(side->s, side->fork, 0);
    }
    void join() const
    {
        if (!side) return;
        cudaEventRecord(side->join, side->s);
        cudaStreamWaitEvent(st, side->join, 0);
    }
    // f(first solve, solves, stream) for each half.
    template <typename F>
    void each(F f) const
    {
        f(0, nlo, st);
        if (side) f(nlo, nres - nlo, side->s);
    }
};

}  // namespace gbfwi
