// The ring of shared-memory stages of the pipelined binary-coded GEMV: which slot and which barrier phases a stage has.  Plain C++,
// so that the schedule can be checked on the host (tests/test_stage_ring.py).
//
// Stage i lives in slot i % S and is taken by consumer group i % G.  A slot has a `free` barrier (all warps of the group arrived);
// the `full` barriers (the stage's copies landed) go round by themselves: stage i uses number i % F.  A wait on a barrier names a
// parity: it tells a phase from its neighbours and from nothing else, so it may only be made while the barrier stands at most
// one phase from the awaited one.
//  * The producer waits for stage i - S on `free` before it issues stage i, in the order of the stages: one phase at most.
//  * A warp that comes to stage i has taken stage i - G, so the stages up to i - G were issued and those up to i - G - S were
//    freed.  With F >= G + S that includes stage i - F, the phase before the awaited one, whatever the order in which copies
//    land; and the phase after it cannot end before this warp has arrived on `free`.
//  * Where S is a multiple of G, F = S will do: the phase before is stage i - S, which this very warp has read.
// One `full` barrier per slot is not enough for other S.  With 2 slots and 3 groups, group 2 starts at stage 2 and finds slot 0's
// barrier in phase 0, which its parity cannot tell from phase 1 completed: it reads a slot that is being written.  With 4 slots it
// takes a first copy that lands after a later one's group is done.
// Measured (us, fp16, 28672 x 4096 at 2, 3 and 4 bits: 8, 5 and 3 slots; one barrier per slot 12.1, 15.2 and 20.4): this 11.8, 14.8 and
// 20.5.  The consumers, who are short of registers, find places by multiplication, the producer by division: with divisions on
// both sides 12.4, 15.4 and 21.6, with multiplications 12.0, 14.9 and 21.4.  Two barriers per slot for every S and as many groups as
// slots 12.3, 14.8 and 21.9; consumers that wait for `free` as well 4 % more over the launches of an 8B block.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define DD_RING_FN __host__ __device__ __forceinline__
#else
#define DD_RING_FN inline
#endif

namespace dd {

// number of `full` barriers: a multiple of the slots
DD_RING_FN uint32_t ring_full_barriers(uint32_t slots, uint32_t groups) {
    return slots % groups == 0u ? slots : (groups + slots + slots - 1u) / slots * slots;
}
// stands for a division by n (1 <= n <= 16) of stages below 2^12 (a tile has at most 2^11: the accumulators hold 2^18 outputs, 128
// of them to a stage)
DD_RING_FN uint32_t ring_inverse(uint32_t n) { return (1u << 20) / n + 1u; }
DD_RING_FN uint32_t ring_turn(uint32_t stage, uint32_t inverse) { return (stage * inverse) >> 20; }
// place on a ring of n: the slot with n = slots, the `full` barrier with n = full barriers
DD_RING_FN uint32_t ring_place(uint32_t stage, uint32_t n, uint32_t inverse) { return stage - ring_turn(stage, inverse) * n; }
// parity of the phase that belongs to a stage on a barrier that is used once per turn of its ring
DD_RING_FN uint32_t ring_parity(uint32_t stage, uint32_t inverse) { return ring_turn(stage, inverse) & 1u; }

}  // namespace dd
