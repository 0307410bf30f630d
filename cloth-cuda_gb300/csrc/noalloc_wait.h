// The wait at the allocation-free frame's grid barrier.  A word counts the
// arrivals of all barriers of the frame; a block that has waited too long sets
// kNaGaveUp in the same word, by a compare-and-swap against the count that it
// found short.  Every block therefore draws the same conclusion about a barrier:
// either its last arrival came first and all blocks pass, or the mark came
// first and none does.  With the mark in a word of its own a block could pass
// the last barrier and write its vertices while another one left without.
// The mark also ends the other blocks' waits at their next look.
#pragma once

#ifdef __CUDACC__
#define PDG_HD __host__ __device__ __forceinline__
#else
#define PDG_HD inline
#endif

namespace pdg {

constexpr unsigned kNaGaveUp = 0x80000000u;   // above any count: 8,196 barriers of a few hundred blocks

// Arrives at a barrier and waits until the count is `want`; false when the
// frame was given up.  Word: arrive() adds one and releases, look() reads and
// acquires, start() begins the time of the wait, late() says that it is over,
// replace(v, to) is the compare-and-swap.
template <class Word>
PDG_HD bool na_wait_on(Word& w, unsigned want)
{
    w.arrive();
    unsigned v = w.look();
    if (v < want) {
        w.start();
        do {
            v = w.look();
            if (v < want && w.late()) w.replace(v, v | kNaGaveUp);   // (seen at the next look; no effect if one arrived)
        } while (v < want);
    }
    return (v & kNaGaveUp) == 0;
}

}  // namespace pdg
