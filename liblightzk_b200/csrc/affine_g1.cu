// affine_g1.cu -- the batched affine rounds of G1 (affine.cuh).
#include "affine.cuh"

namespace lzk {

int affine_round(const AffineRound<Fq>& a, unsigned blocks, cudaStream_t st)
{
    const uint32_t count = blocks * kAffThreads;
    (a.r == 1 ? k_affine_prefix_g1<true> : k_affine_prefix_g1<false>)<<<blocks, kAffThreads, 0, st>>>(a); note_launch();
    k_affine_invert<<<grid_for(count / kInvGroup, kAffThreads), kAffThreads, 0, st>>>(a.acc, count); note_launch();
    (a.r == 1 ? k_affine_sum_g1<true> : k_affine_sum_g1<false>)<<<blocks, kAffThreads, 0, st>>>(a); note_launch();
    return launch_status();
}

uint32_t debug_word_affine_g1(bool clear) { return debug_word_here(clear); }

}  // namespace lzk
