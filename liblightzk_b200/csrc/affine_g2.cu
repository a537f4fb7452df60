// affine_g2.cu -- the batched affine rounds of G2 (affine.cuh).
#include "affine.cuh"

namespace lzk {

int affine_round(const AffineRound<Fq2>& a, unsigned blocks, cudaStream_t st)
{
    const uint32_t count = blocks * kAffThreads;
    (a.r == 1 ? k_affine_prefix_g2<true> : k_affine_prefix_g2<false>)<<<blocks, kAffThreads, 0, st>>>(a); note_launch();
    k_affine_invert<<<grid_for(count / kInvGroup, kAffThreads), kAffThreads, 0, st>>>(a.acc, count); note_launch();
    (a.r == 1 ? k_affine_sum_g2<true> : k_affine_sum_g2<false>)<<<blocks, kAffThreads, 0, st>>>(a); note_launch();
    return launch_status();
}

uint32_t debug_word_affine_g2(bool clear) { return debug_word_here(clear); }

}  // namespace lzk
