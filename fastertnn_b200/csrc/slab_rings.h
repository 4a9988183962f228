// Depths of the two rings of the slab-fed GEMM (gemm_slab.cu): slab buffers and weight stages share a block's shared memory.
// Host code without CUDA headers.
#pragma once

#include <algorithm>

constexpr int SL_MAXSLAB = 8;    // slab buffers at most
constexpr int SL_MAXSTG = 12;    // weight ring depth at most

// Who fetches the slabs: tensor copies; loader warps with one MMA issuer; loader warps of the form that has two MMA issuers where
// the weights stay.
enum SlabFeed { SLAB_COPIES, SLAB_LOADERS, SLAB_LOADERS_TWO };

struct SlabRings {
    int nslab, nstg;
    bool resident;  // the kernel tile's weight stages all fit the ring: fetched once per block
};

// Depths that fit `avail` bytes; false when not even two slabs and three weight stages do.
//   two issuers   as many slabs as leave the weights resident, an even number (the issuers take them in turn), up to eight.
//                 GEMM alone, image out, 2 / 4 / 8 slabs: 32 x 128x112x112 -> 64 (23 KB each) 22.4 / 21.6 / 18.8 us,
//                 8 x 64x224x224 -> 64 (19 KB) 15.6 / 15.1 / 14.2, 256 x 64x56x56 -> 64 (8 KB) 27.4 / 26.3 / 26.2
//   one issuer    loaders: two slabs, the rest for the weights.  More slabs gained nothing there and displaced weights that could stay:
//                 2 / 4 / 8 slabs 32 x 64x80x80 -> 128 5x5 29.5 / 29.9 / 33.7 us, 64 x 128x112x112 -> 128 50.0 / 50.2 / 65.7, 256 x
//                 128x28x28 -> 128 (weights resident with all three) 16.9 / 17.2 / 17.6.
//   copies        four, three or two by their size
inline bool slab_rings(int slab_bytes, int b_stage, int avail, int nchunks, bool one_kernel_tile, SlabFeed feed, SlabRings* r) {
    const bool may_stay = one_kernel_tile && nchunks <= SL_MAXSTG;
    if (feed == SLAB_LOADERS_TWO && may_stay)
        for (int ns = SL_MAXSLAB; ns >= 2; ns -= 2)
            if (avail - ns * slab_bytes >= std::max(nchunks, 3) * b_stage) {
                *r = {ns, nchunks, true};
                return true;
            }
    int ns = feed != SLAB_COPIES ? 2 : slab_bytes <= 16384 ? 4 : slab_bytes <= 32768 ? 3 : 2;
    for (; ns >= 2; ns--) {
        const int rest = avail - ns * slab_bytes;
        if (rest < 3 * b_stage) continue;
        const int nb = std::min(SL_MAXSTG, rest / b_stage);
        const bool stay = may_stay && nchunks <= nb;
        *r = {ns, stay ? nchunks : nb, stay};
        return true;
    }
    return false;
}
