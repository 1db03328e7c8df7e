// The words by which a block's top-k hands the routed experts of a layer to the block's producers: one for each slot, {layer + 1, expert} in 16 bits each,
// in shared memory.  Plain C++ for both sides.
//
// Single words, written by one lane without a fence and read by threads of other warps: each carries its own mark, and a thread that has seen the word
// of one slot knows nothing of the others (relaxed accesses to different words have no order, whichever was stored first).  So whoever takes an
// expert from a word has seen the layer's mark in that very word.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LEMOQ_BOTH __host__ __device__ __forceinline__
#else
#define LEMOQ_BOTH inline
#endif

namespace lemoq {
namespace tile {

// The slots whose experts' rows a tile holds.
struct RouteSlots {
    int first, count;
};
// Gate/up: the tiles of a slot are 2^shift in a row.
LEMOQ_BOTH RouteSlots slots_of_gate_up(int tile, int shift) { return RouteSlots{tile >> shift, 1}; }
// Down: tile pp of a block of output rows holds slot pp, or, `paired`, slots 2 pp and 2 pp + 1 (the last one alone when top_k is odd).
LEMOQ_BOTH RouteSlots slots_of_down(int pp, bool paired, int top_k) {
    return paired ? RouteSlots{2 * pp, 2 * pp + 1 < top_k ? 2 : 1} : RouteSlots{pp, 1};
}

LEMOQ_BOTH uint32_t route_mark(int layer) { return static_cast<uint32_t>(layer + 1) << 16; }
LEMOQ_BOTH uint32_t route_expert(uint32_t word) { return word & 0xffffu; }
LEMOQ_BOTH bool route_known(const volatile uint32_t* route, int layer, RouteSlots s) {
    const uint32_t mark = route_mark(layer);
    return (route[s.first] & 0xffff0000u) == mark && (s.count == 1 || (route[s.first + 1] & 0xffff0000u) == mark);
}

}  // namespace tile
}  // namespace lemoq
