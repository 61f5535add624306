// The order in which a block of the decode attention (attn.cu) uses its ring of stages: which slot a stage goes to, which parity its
// quad waits for, which stage takes whose place. Apart from the kernel so that the order can be played through without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define QB_RING __host__ __device__ __forceinline__
#else
#define QB_RING inline
#endif

namespace qb {

// QUADS quads take a split's stages in turn (stage j: quad j % QUADS); NSTG slots; a split's first stage goes to slot OFF.
template <int QUADS, int NSTG, int OFF>
struct DecRing {
    int j0 = 0;         // the stages of the block's splits before this one
    uint32_t pars = 0;  // bit i: the parity that this split's first stage in slot i waits for

    QB_RING static int slot(int j) { return (j + OFF) % NSTG; }
    QB_RING uint32_t parity(int j) const { return ((j / NSTG) ^ (pars >> slot(j))) & 1; }
    // A slot's stages go to different quads, and a parity says nothing to a waiter that is two phases behind: one whose slot still waits for
    // its last stage's copies would be let through. So a slot keeps the number of the stage asked for last, counted through the block's
    // splits (a number of the split before says nothing of this one), and a quad looks for its own before it waits. Not for a split's first
    // stages, which are asked for before its quads begin.
    QB_RING int number(int j) const { return j0 + j; }
    QB_RING static bool looks(int j) { return j >= NSTG; }
    // the stage that is asked for when all of the quad is done with its stage before j (two quads: in the middle of j), and when all
    // of it is done with j itself (more quads: with two the next stage would be late then); -1: none
    QB_RING static int in_the_middle(int j, int nstg) { return QUADS == 2 && j >= 2 && j - 2 + NSTG < nstg ? j - 2 + NSTG : -1; }
    QB_RING static int at_the_end(int j, int nstg) { return QUADS > 2 && j + NSTG < nstg ? j + NSTG : -1; }
    // the next split begins: every slot has seen as many phases as it had stages
    QB_RING void next_split(int nstg) {
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int sl = 0; sl < NSTG; sl++) {
            const int j = (sl + NSTG - OFF) % NSTG;  // the first stage in this slot
            if (j < nstg) pars ^= (((nstg - 1 - j) / NSTG + 1) & 1) << sl;
        }
        j0 += nstg;
    }
};

}  // namespace qb
