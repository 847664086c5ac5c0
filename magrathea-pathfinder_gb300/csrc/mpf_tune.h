// The slices of a tuning batch: each candidate launch shape traces one of them
// and is judged by its photon-steps per second, so the slices have to be alike.
// On a refined octree the rays run in the order of their directions, where four
// contiguous quarters are four regions of the sky with their own refinement and
// step counts.  The order is dealt out instead: chunk c of kTuneChunk rays goes
// to slice c % kTuneSlices, so that each slice samples the whole sky and a
// warp's 32 rays are still neighbours.
#pragma once
#include "mpf_keys.cuh"

namespace mpf {

constexpr int kTuneSlices = 4;
constexpr long long kTuneChunk = 256;

// rays of a slice (the last one also takes what is left)
MPF_HD long long tune_slice(long long n) { return n / (kTuneSlices * kTuneChunk) * kTuneChunk; }

// the place in the order that place i of the dealt order holds
MPF_HD long long tune_dealt(long long i, long long n)
{
    const long long slice = tune_slice(n);
    if (i >= kTuneSlices * slice) return i;
    const long long k = i / slice, r = i % slice;
    return (kTuneSlices * (r / kTuneChunk) + k) * kTuneChunk + r % kTuneChunk;
}

}  // namespace mpf
