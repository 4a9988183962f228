// Bitwise GEMM + PReLU on the tensor cores for stride-1 layers, fed from a BORDERED 4-bit image: one
// slab of pixels per tile serves every filter tap (reference: mm_tnn / mm_tbn / mm_btn / mm_bnn,
// src/tnns/mm_p2_final_*_avx2.c, on the rows t2r_p2_opt / b2r would have scattered,
// src/tnns/ternarize2row_avx2.c:285-313).
//
// The layer input is stored as e2m1 operands with its padding around every image:
// [n][Hp = H + 2*PH][Wp = W + 2*PW][C/2 bytes], border pixels = the padding value (ternary 0, binary
// +1).  Output rows are laid over that same padded lattice: virtual row q = (n*Hp + y)*Wp + x is the
// window whose top-left corner is padded pixel (y, x); it is a real output pixel (oh, ow) = (y, x)
// when y < OH and x < OW, and is computed but never stored otherwise ((Hp*Wp)/(OH*OW) - 1 more
// MMAs: 13 % at 32x32, 7 % at 56x56).  Filter tap (kh, kw) of 128 consecutive virtual rows then
// reads the 128 consecutive pixels q0 + kh*Wp + kw ..., so ALL taps of a tile are row-shifted views of
// ONE slab of 128 + (KH-1)*Wp + (KW-1) pixels: one tiled tensor copy per tile and 128-byte channel
// group instead of one im2col copy per tap -- 25 KB instead of 144 KB per 512-channel tile at 32x32,
// and one request instead of twelve per 64-channel tile.  The tensor core reads a shifted view by
// starting its shared-memory descriptor at the slab's row kh*Wp + kw: the swizzle pattern is a
// function of the absolute shared-memory address, which the copy engine and the MMA share.
//
// A pixel's bytes per slab row follow the channel count as in the im2col form: 128 bytes (256
// channels; more channels = several slabs per tile, one after the other), 64 or 32 (128 / 64
// channels; 64- / 32-byte swizzle), and a weight stage is the same pre-expanded 128-byte-row image
// (four plane words), so K steps that only exist because rows are padded to four words are skipped.
// Weights that fit the ring entirely are fetched once per block and stay (64-kernel layers).
//
// Roles per block: producer warp (slabs and weight stages), MMA warp, eight or twelve epilogue warps; image outputs of 32- and
// 64-byte pixels: two more warps that fetch the slabs, sixteen epilogue warps on tiles of 64 kernels; with QF
// four quantiser warps and a publisher as in the im2col form (gemm_tc.cu).  Block pairs
// (tcgen05.mma.cta_group::2) share a 256-row tile, each block with its own slab and half of the
// weight stage.  Every wait is bounded.
#include <algorithm>
#include <type_traits>

#include "gemm_tc_common.cuh"
#include "slab_rings.h"

namespace {

constexpr int SL_TAPMAX = 4096;  // filter taps at most
constexpr int SL_BAR_BYTES = 512;

struct SlabArgs {
    const unsigned char* Aimg;  // the bordered image
    const unsigned char* Bimg;  // expanded weights [n_tile][stage][BN rows][128 B]
    float* y;
    int Mv;                     // virtual rows: N * Hp * Wp
    int KN, nchunks;            // kernels, weight stages per kernel tile
    int b_rows, b_shift;        // kernels per tile of the weight image (a power of two) and its logarithm: BN, or a multiple of it (few tiles)
    int y_vec;                  // floats of a pixel-major output row that may be stored at once: 4, 2 or 1
    int OH, OW, Wp, HpWp;       // output size, padded input lattice
    int KW, T;                  // filter width, taps KH*KW
    int G;                      // 128-byte channel groups per pixel (one slab each); 1 for 64 / 128 channels
    int slab_bytes, slab_rows, copy_rows, ncopies;  // slab buffer size, rows; rows per tensor copy and copies per slab
    int nslab, nstg;            // ring depths: slabs, weight stages
    int b_resident;             // the kernel tile's weight stages all fit the ring: fetched once per block
    int layout, zero_passes, acc_bias;
    float alpha;
    unsigned int* status;
    // optional quantised output for a following layer (instead of y)
    uint32_t* pimg;
    const float* thr_next;
    int next_format;            // 0 binary bit planes, 1 ternary bit planes, 2 plain 4-bit image, 3 bordered 4-bit image
    int next_binary;            // formats 2 / 3: the next layer's activations are binary
    int cp_next;
    int o_Wp, o_Hp, o_PH, o_PW; // format 3: the next image's padded lattice (== this layer's) and its border
    // fused quantisation
    const float* qthr;
    uint4* qimg;
    unsigned int* q_sync;
    int qN, qC, q_nbands, q_H, q_W, q_PH, q_PW, q_binary, q_self_clean, Cp;
    FastDiv div_hpwp, div_wp, div_ntn;
};

// 16 bytes, global -> shared memory by this thread's own copy; the last `16 - bytes` of them zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// IMG: quantised output for a following layer, in kernels of its own: either epilogue's registers and code cost the other (the
// one-launch forms, which the library never picks by itself, keep both).  On single blocks with 32- or 64-byte pixels it comes with
// slab loaders and, on tiles of 64 kernels, two MMA issuers and a set of epilogue warps per accumulator.
template <int BN, int CG, int TAPS, bool QF, bool IMG>
struct SlabCfg {
    static constexpr int RB = 128 / TAPS;             // bytes of a pixel in a slab row
    static constexpr int B_STAGE = (BN / CG) * KCH;   // bytes of a weight stage in one block
    static constexpr bool OVL = BN == 256;            // overlapping accumulator sets (scales leave 480 columns)
    static constexpr int ACC_OFF = OVL ? BN - 32 : BN;
    static constexpr int NBUF = OVL ? 2 : (BN == 64 ? 4 : 3);  // accumulator sets in tensor memory
    // Epilogue warps: EPW per lane quadrant share a tile's columns, and NSETS such groups take the tiles in turn.  On tiles of
    // 64 / 128 kernels a tile's drain is a chain of latencies (barrier, row addresses, tensor-memory load, 32 columns of
    // arithmetic) several times as long as its MMAs, so three tiles are drained at once.  Eight warps on one tile / two sets /
    // three sets, inside the 11-layer stack: 64 -> 64 @56 48.3 / 39.8 / 33.0 us, 128 -> 128 @28 25.9 / 22.1 / 19.4.  A fourth set gains
    // nothing by itself; two issuers need one per accumulator (below).
    static constexpr bool LOADER = IMG && CG == 1 && TAPS > 1 && !QF;
    static constexpr bool TWO = LOADER && BN == 64;   // two MMA issuers (see the kernel)
    static constexpr int EPW = OVL ? 2 : 1, NSETS = OVL ? 1 : TWO ? 4 : (QF ? 2 : 3);
    // (a set's next tile waits for its barrier's phase by parity: the phase before must be complete by then)
    static_assert(NSETS <= NBUF, "a set may not be a whole turn of the accumulators ahead");
    static constexpr int NEPI = 4 * EPW * NSETS;      // epilogue warps
    // issuers may finish their tiles out of turn: every accumulator then belongs to one issuer and one set
    static_assert(!TWO || (NBUF % 2 == 0 && NSETS == NBUF), "waits by parity: everyone meets a barrier in successive phases");
    // Slab loaders.  A tiled tensor copy moves one box row in about 2.6 clocks whatever its length, so slabs of 32-byte pixels came
    // at 640 clocks a tile of 64 kernels (246 rows at 56x56), whose MMAs take 432.  The slab is contiguous in the image: two warps
    // fetch it in 16-byte pieces and place them in the swizzle pattern.  Image out, one GEMM, before loaders, second issuer and the
    // epilogue of quantise32_e2m1 / after: 256 x 64x56x56 -> 64 34.3 / 26.1 us, 256 x 128x28x28 -> 128 21.1 / 16.8, 8 x 64x112x112 ->
    // 64 7.4 / 7.0 (the drain alone takes some 900 clocks a tile of 64 kernels, the MMAs alone 475).
    static constexpr int NLOAD = LOADER ? 2 : 0, WARP_LOAD0 = 2;
    static constexpr int WARP_EPI0 = 2 + NLOAD, WARP_Q0 = WARP_EPI0 + NEPI;
    static constexpr int NTHREADS = 32 * (WARP_EPI0 + NEPI + (QF ? 5 : 0));
    static constexpr int Q_STAGE = Q_PIX * 64 * 4;
    static constexpr int SMEM_MAX = 232448;
};

// GRP = weight stages per slot of their ring (one pair of barriers per slot).  3: a filter row of a 3x3 layer of 128-byte pixels on
// tiles of 64 or 128 kernels whose weights stream.  There the producer's wait, announcement and copy take some 300 clocks a
// slot and the MMA warp's wait and commit another 80, the four MMAs of a stage of 64 kernels 192.  GEMM alone, one stage a slot and a
// division per stage / one stage / three: 8 x 512x14x14 -> 512 9.0 / 6.4 / 6.3 us, 8 x 1024x14x14 -> 1024 16.1 / 11.4 / 10.8, 8 x
// 256x28x28 -> 256 7.3 / 6.0 / 5.9.
template <int BN, int CG, int TAPS, bool QF, bool SINGLE, int GRP, bool IMG>
__global__ void __launch_bounds__(SlabCfg<BN, CG, TAPS, QF, IMG>::NTHREADS, 1)
gemm_slab_kernel(SlabArgs p, const __grid_constant__ TensorMaps<maps_of(CG, QF)> maps) {
    const CUtensorMap &tmap_a = maps.m[0], &tmap_b = maps.m[CG == 2 ? 1 : 0], &tmap_q = maps.m[QF ? 2 : 0];
    using Cfg = SlabCfg<BN, CG, TAPS, QF, IMG>;
    static_assert(GRP == 1 || (GRP == 3 && TAPS == 1 && CG == 1 && !QF), "slots of three stages: streamed 3x3 weights of 128-byte pixels");
    constexpr int RB = Cfg::RB, B_STAGE = Cfg::B_STAGE, WARP_EPI0 = Cfg::WARP_EPI0, EPW = Cfg::EPW, ACC_OFF = Cfg::ACC_OFF;
    constexpr bool OVL = Cfg::OVL;
    constexpr int NBUF = Cfg::NBUF, NSETS = Cfg::NSETS;
    static_assert((2 * SL_MAXSLAB + 2 * SL_MAXSTG + 2 * NBUF) * 8 + 8 <= SL_BAR_BYTES, "barriers");
    constexpr int TILE_M = CG * BM;
    // e2m1 A and B (1<<7, 1<<10), ue8m0 scales (1<<23), K-major, N>>3 at bit 17, M>>4 at bit 24
    constexpr uint32_t IDESC = (1u << 23) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((CG * BM) >> 4) << 24);
    constexpr uint32_t SF_COL = 480;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = smem;
    unsigned char* sB = smem + p.nslab * p.slab_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + p.nstg * B_STAGE);
    const uint32_t bar_sfull = smem_u32(bars), bar_sempty = smem_u32(bars + SL_MAXSLAB), bar_bfull = smem_u32(bars + 2 * SL_MAXSLAB),
                   bar_bempty = smem_u32(bars + 2 * SL_MAXSLAB + SL_MAXSTG), bar_tfull = smem_u32(bars + 2 * SL_MAXSLAB + 2 * SL_MAXSTG),
                   bar_tempty = smem_u32(bars + 2 * SL_MAXSLAB + 2 * SL_MAXSTG + NBUF);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SL_MAXSLAB + 2 * SL_MAXSTG + 2 * NBUF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* q_ring = reinterpret_cast<unsigned char*>(bars) + SL_BAR_BYTES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntn = (p.KN + BN - 1) / BN;
    const int ntm = (p.Mv + TILE_M - 1) / TILE_M;
    const int ntiles = ntm * ntn;
    const uint32_t rank = (CG == 2) ? cluster_ctarank() : 0u;
    const int unit = blockIdx.x / CG, nunits = gridDim.x / CG;
    const int SPG = (TAPS == 1) ? p.T : p.nchunks;  // weight stages per slab

    if (tid == 0) {
        for (int s = 0; s < SL_MAXSLAB; s++) {
            mbar_init(bar_sfull + 8 * s, 1);
            mbar_init(bar_sempty + 8 * s, 1);
        }
        for (int s = 0; s < SL_MAXSTG; s++) {
            mbar_init(bar_bfull + 8 * s, 1);
            mbar_init(bar_bempty + 8 * s, 1);
        }
        for (int b = 0; b < NBUF; b++) {
            mbar_init(bar_tfull + 8 * b, 1);
            mbar_init(bar_tempty + 8 * b, CG * 4 * EPW);
        }
        if (QF) {
            uint64_t* qbars = reinterpret_cast<uint64_t*>(q_ring + Q_STG * Cfg::Q_STAGE);
            for (int s = 0; s < Q_STG; s++) {
                mbar_init(smem_u32(qbars + s), 1);
                mbar_init(smem_u32(qbars + Q_STG + s), 4);
            }
            volatile QuantCtl* ctl = reinterpret_cast<volatile QuantCtl*>(qbars + 2 * Q_STG);
            ctl->done[0] = ctl->done[1] = ctl->done[2] = ctl->done[3] = 0;
            ctl->published = 0;
            ctl->total = 0xFFFFFFFFu;
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == WARP_MMA) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        // dependents may be placed once this block holds its tensor memory, and the producer of a single block goes ahead of the rest
        // of the set-up (gemm_tc.cu has the reasons for both)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    constexpr bool LONE = CG == 1;
    const bool ahead = LONE && warp == WARP_TMA;
    // Two warps issue the MMAs of every other tile each where a tile has few of them and the weights stay: the producer's warp has
    // nothing left to do, and a tile's two waits (110-140 clocks each even when complete) pass beside the other's MMAs.  Both take an
    // even number of slabs (slab_rings.h; one issuer on an odd one) and accumulators in turn, so each meets the same ones in successive phases.
    const bool two = Cfg::TWO && p.b_resident && p.T == 9 && p.KW == 3 && (p.nslab & 1) == 0;
    uint32_t tmem_base = 0;
    if (ahead) {
        named_arrive(1, blockDim.x);
    } else {
        tc_fence_before();
        if (CG == 2) cluster_sync_all(); else named_sync(1, blockDim.x);
        tc_fence_after();
        tmem_base = *tmem_slot;
    }
    // unit block scales (ue8m0 0x7F) in columns 480..511, as in the im2col form
    if (warp >= WARP_EPI0 && warp < WARP_EPI0 + 4) {
        const uint32_t one = 0x7F7F7F7Fu;
#pragma unroll 1
        for (uint32_t c = 0; c < 32; c += 8) {
            const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + SF_COL + c;
            asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(one) : "memory");
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    if (!ahead) {
        tc_fence_before();
        if (CG == 2) cluster_sync_all(); else named_sync(2, two ? blockDim.x : blockDim.x - 32);
        tc_fence_after();
    }

    // weight stage c of kernel tile n_tile -> ring slot; a tile is rows [n_tile*BN % b_rows, +BN) of an image tile of b_rows kernels
    const uint32_t bfull_lead = (CG == 2) ? mapa_shared(bar_bfull, 0) : bar_bfull;
    // (no division and little arithmetic per stage: with one of each the producer took 500 clocks a stage)
    const size_t b_step = (size_t)p.b_rows * KCH;
    auto weights_of = [&](int n_tile) -> const unsigned char* {
        const uint32_t k0 = (uint32_t)(n_tile * BN), big = k0 >> p.b_shift;
        return p.Bimg + (size_t)big * p.nchunks * b_step + (size_t)(k0 & (uint32_t)(p.b_rows - 1)) * KCH;
    };
    const size_t j_step = (TAPS == 1) ? (size_t)p.G * b_step : b_step;  // from a stage of a slab to the next
    // the GRP stages from w (stage c of the tile) on -> the slot whose first ring stage is `at`
    auto request_weights = [&](const unsigned char* w, int n_tile, int c, uint32_t at, uint32_t slot) {
        if (CG == 2) {
            if (rank == 0) mbar_arrive_expect_tx(bar_bfull + 8 * slot, CG * B_STAGE);
            tma_tile2d_g2s_pair(smem_u32(sB + at * B_STAGE), &tmap_b, 0, (n_tile * p.nchunks + c) * BN + (int)rank * (BN / CG), bfull_lead + 8 * slot);
        } else {
            mbar_arrive_expect_tx(bar_bfull + 8 * slot, (uint32_t)(GRP * B_STAGE));
#pragma unroll
            for (int g = 0; g < GRP; g++) bulk_g2s(smem_u32(sB + (at + g) * B_STAGE), w + g * j_step, B_STAGE, bar_bfull + 8 * slot);
        }
    };
    // the first stages of the block's first tile, before the wait for the launch in front (32 KB of constant weights, see gemm_tc.cu, in
    // whole slots of the first slab's stages: one of 48 KB where a slot is three stages of 128 kernels)
    constexpr int EARLY = 32768 / (GRP * B_STAGE) > 0 ? 32768 / (GRP * B_STAGE) * GRP : GRP;
    const int early = min(min(EARLY, p.nstg), SPG);
    if (warp == WARP_TMA && lane == 0 && unit < ntiles) {
        if (!Cfg::LOADER) prefetch_tensor_map(&tmap_a);
        const int n_tile = unit - (int)p.div_ntn.div((uint32_t)unit) * ntn;
        const unsigned char* src = weights_of(n_tile);
        for (int j = 0; j < early; j += GRP) {
            const int c = (TAPS == 1) ? j * p.G : j;
            const uint32_t at = p.b_resident ? (uint32_t)c : (uint32_t)j;
            request_weights(src + (size_t)j * j_step, n_tile, c, at, at / GRP);
        }
    }

    if (two && warp == WARP_TMA) {
        __syncwarp();
        named_sync(2, blockDim.x);
        tc_fence_after();
        tmem_base = *tmem_slot;
    }

    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == WARP_TMA) {
        if (lane == 0) {
            uint32_t sl = 0, slph = 1, s = 0, ph = 1;
            const uint32_t nslots = (uint32_t)p.nstg / GRP;
            bool first_tile = true;
            const uint32_t sfull_lead = (CG == 2) ? mapa_shared(bar_sfull, 0) : bar_sfull;
            const uint32_t copy_bytes = (uint32_t)(p.ncopies * p.copy_rows * RB);
            // (with loaders and weights that stay only the first tile's weights are left to request)
            for (int t = unit; t < ntiles && !(Cfg::LOADER && p.b_resident && !first_tile); t += nunits, first_tile = false) {
                const int m_tile = (int)p.div_ntn.div((uint32_t)t), n_tile = t - m_tile * ntn;
                const unsigned char* src = weights_of(n_tile);
                const int q0 = m_tile * TILE_M + (int)rank * BM;  // first virtual row = first pixel of the block's slab
                if (QF && q0 < p.Mv) {
                    // the slab reads the images its pixels belong to: wait until the quantiser warps (of any
                    // block) have finished them, border item included
                    const int q_last = min(q0 + p.ncopies * p.copy_rows, p.Mv) - 1;
                    const int n_first = (int)p.div_hpwp.div((uint32_t)q0), n_last = (int)p.div_hpwp.div((uint32_t)q_last);
                    const unsigned int per_image = (unsigned int)(p.q_nbands * p.Cp + 1) * 4u;
                    for (int n = n_first; n <= n_last; n++)
                        if (!counter_wait(p.q_sync + Q_FLAG0 + n, per_image, abort_flag, p.status, 6)) goto done;
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                }
                for (int cg = 0; cg < p.G; cg++) {
                    if (!Cfg::LOADER && !mbar_wait(bar_sempty + 8 * sl, slph, abort_flag, p.status, 0x11)) goto done;
                    const uint32_t dst = smem_u32(sA + sl * p.slab_bytes);
                    if (Cfg::LOADER) {
                    } else if (CG == 2) {
                        if (rank == 0) mbar_arrive_expect_tx(bar_sfull + 8 * sl, CG * copy_bytes);
                        for (int i = 0; i < p.ncopies; i++)
                            tma_tile2d_g2s_pair(dst + i * p.copy_rows * RB, &tmap_a, cg * KCH, q0 + i * p.copy_rows, sfull_lead + 8 * sl);
                    } else {
                        mbar_arrive_expect_tx(bar_sfull + 8 * sl, copy_bytes);
                        for (int i = 0; i < p.ncopies; i++)
                            tma_tile2d_g2s(dst + i * p.copy_rows * RB, &tmap_a, cg * KCH, q0 + i * p.copy_rows, bar_sfull + 8 * sl);
                    }
                    if (++sl == (uint32_t)p.nslab) { sl = 0; slph ^= 1; }
                    if (p.b_resident) {
                        if (first_tile)
                            for (int j = cg == 0 ? early : 0; j < SPG; j++) {
                                const int c = (TAPS == 1) ? j * p.G + cg : j;
                                request_weights(src + (size_t)c * b_step, n_tile, c, (uint32_t)c, (uint32_t)c);
                            }
                        continue;
                    }
                    const unsigned char* w = src + ((TAPS == 1) ? (size_t)cg * b_step : 0);
                    int j = 0;
                    if (first_tile && cg == 0) {
                        j = early;
                        s = (uint32_t)early / GRP;
                        if (s == nslots) { s = 0; ph ^= 1; }
                        w += (size_t)early * j_step;
                    }
                    for (; j < SPG; j += GRP) {
                        if (!mbar_wait(bar_bempty + 8 * s, ph, abort_flag, p.status, 1)) goto done;
                        const uint32_t s1 = s + 1 == nslots ? 0u : s + 1;
                        request_weights(w, n_tile, (TAPS == 1) ? j * p.G + cg : j, s * GRP, s);
                        w += GRP * j_step;
                        s = s1;
                        if (s1 == 0) ph ^= 1;
                    }
                }
            }
        }
        // On to issuing: lane 0 left no wait behind that could have sent it to `done` (loaders, weights that stay).  In every other form
        // its failed wait goes to `done` directly, and a barrier here would leave it one warp barrier behind the other lanes.
        if (two) __syncwarp();
    }
    if (warp == WARP_MMA || (two && warp == WARP_TMA)) {
        if (rank == 0) {  // pair: the first block issues for both
            // This warp's instruction stream paces the tensor pipe: it runs warp-uniform (see elect_one), nothing that
            // touches shared memory stands between two MMAs of a slab (a table look-up per tap, queued behind the MMAs just
            // issued, cost 60 clocks per MMA: tap offsets are registers or running counters), and a slab's MMAs sit in as few
            // elected regions as the weight waits allow (one by one, every reconvergence waited for the MMA before it).
            const bool elected = elect_one();
            const uint32_t step = two ? 2u : 1u;  // issuers that take the tiles in turn
            uint32_t lt = warp == WARP_MMA ? 0u : 1u, sl = lt, slph = 0, s = 0, ph = 0;
            bool first_tile = true;
            const uint64_t da0 = make_desc_taps(smem_u32(sA), TAPS), db0 = make_desc(smem_u32(sB));
            const uint32_t slab16 = (uint32_t)(p.slab_bytes >> 4);
            const uint32_t row16 = (uint32_t)(p.Wp * (RB / 16));  // one image row further down the slab, in descriptor units
            const uint32_t a_lo0 = (uint32_t)da0, a_hi = (uint32_t)(da0 >> 32), b_lo0 = (uint32_t)db0, b_hi = (uint32_t)(db0 >> 32);
            const uint32_t sfa = tmem_base + SF_COL, sfb = tmem_base + SF_COL + 16;
            auto mma = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t acc) {
                if (CG == 2) tc_mma_f4_pair_lh(d_tmem, a_lo, a_hi, b_lo, b_hi, IDESC, sfa, sfb, acc);
                else tc_mma_f4_lh(d_tmem, a_lo, a_hi, b_lo, b_hi, IDESC, sfa, sfb, acc);
            };
            auto commit = [&](uint32_t bar) {
                if (CG == 2) tc_commit_pair(bar); else tc_commit(bar);
            };
            const bool fast3x3 = GRP == 3 || (p.T == 9 && p.KW == 3);
            if (fast3x3) {
                // 3x3 filters: the MMAs of a slab (or, where weights stream, of a stage) are straight-line code, every operand one
                // of four uniform values (the slab's first three image rows, the weights) plus a constant.
                const uint32_t nslots = (uint32_t)p.nstg / GRP;
                constexpr int KPT = 4 / TAPS;               // K steps (32 bytes) per tap: 1, 2 or 4
                constexpr int NK = 9 * KPT, NST = (NK + 3) / 4;  // K steps and weight stages of a slab
                for (int t = unit + (int)lt * nunits; t < ntiles; t += (int)step * nunits, lt += step, first_tile = false) {
                    const int buf = (int)(lt % NBUF);
                    if (!mbar_wait(OVL ? bar_tempty : bar_tempty + 8 * buf, (OVL ? (lt & 1) : ((lt / NBUF) & 1)) ^ 1, abort_flag, p.status, 2)) goto done;
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * ACC_OFF;
                    for (int cg = 0; cg < p.G; cg++) {
                        if (!mbar_wait(bar_sfull + 8 * sl, slph, abort_flag, p.status, 0x13)) goto done;
                        const uint32_t slab_lo = a_lo0 + sl * slab16, slab_lo1 = slab_lo + row16, slab_lo2 = slab_lo1 + row16;
                        // K step q of the slab: 32 bytes x (q % KPT) into the pixels of tap q / KPT
                        auto a_of = [&](int q) {
                            const int tap = q / KPT;
                            return (tap < 3 ? slab_lo : tap < 6 ? slab_lo1 : slab_lo2) + (uint32_t)((tap % 3) * (RB / 16) + 2 * (q % KPT));
                        };
                        if (GRP == 3) {
                            // a slot = the three taps of one filter row
                            uint32_t row_lo = slab_lo;
#pragma unroll 1
                            for (int kh = 0; kh < 3; kh++, row_lo += row16) {
                                if (!mbar_wait(bar_bfull + 8 * s, ph, abort_flag, p.status, 3)) goto done;
                                tc_fence_after();
                                const uint32_t s1 = s + 1 == nslots ? 0u : s + 1;
                                const uint32_t b_lo = b_lo0 + s * (uint32_t)(GRP * (B_STAGE >> 4));
                                if (elected) {
#pragma unroll
                                    for (int q = 0; q < 12; q++)
                                        mma(d_tmem, row_lo + (uint32_t)((q / 4) * (RB / 16) + 2 * (q % 4)), b_lo + (uint32_t)((q / 4) * (B_STAGE >> 4) + 2 * (q % 4)), (uint32_t)(cg | kh | q));
                                    commit(bar_bempty + 8 * s);
                                    if (kh == 2) commit(bar_sempty + 8 * sl);
                                }
                                s = s1;
                                if (s1 == 0) ph ^= 1;
                            }
                        } else if (BN == 256 && p.b_resident && first_tile) {
                            // stage by stage as the weights land (waiting for all of them first: 40 x 128x14x14 -> 256 BNN, one
                            // tile per SM, 11.3 us per layer call against 10.3; on narrower tiles most of them were requested before the
                            // wait for the launch in front); rolled up, it runs once per block and group
#pragma unroll 1
                            for (int j = 0; j < NST; j++) {
                                const uint32_t slot = (TAPS == 1) ? (uint32_t)(j * p.G + cg) : (uint32_t)j;
                                if (!mbar_wait(bar_bfull + 8 * slot, 0u, abort_flag, p.status, 3)) goto done;
                                tc_fence_after();
                                if (elected) {
                                    const uint32_t b_lo = b_lo0 + slot * (uint32_t)(B_STAGE >> 4);
#pragma unroll
                                    for (int k = 0; k < 4; k++) {
                                        const int q = 4 * j + k, tap = q / KPT;
                                        if (q < NK)
                                            mma(d_tmem, slab_lo + (uint32_t)(tap / 3) * row16 + (uint32_t)(tap % 3) * (RB / 16) + 2u * (uint32_t)(q % KPT), b_lo + 2u * k, (uint32_t)(cg | q));
                                    }
                                    if (j == NST - 1) commit(bar_sempty + 8 * sl);
                                }
                            }
                        } else if (p.b_resident) {
                            if (BN != 256 && first_tile)
                                for (int j = 0; j < NST; j++)
                                    if (!mbar_wait(bar_bfull + 8 * ((TAPS == 1) ? j * p.G + cg : j), 0u, abort_flag, p.status, 3)) goto done;
                            tc_fence_after();
                            if (elected) {
#pragma unroll
                                for (int q = 0; q < NK; q++)  // stage q / 4 is slot q / 4: nine taps of one channel group fill the ring (G = 1)
                                    mma(d_tmem, a_of(q), b_lo0 + (uint32_t)((q >> 2) * (B_STAGE >> 4) + 2 * (q & 3)), (uint32_t)q);
                                commit(bar_sempty + 8 * sl);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < NST; j++) {
                                if (!mbar_wait(bar_bfull + 8 * s, ph, abort_flag, p.status, 3)) goto done;
                                tc_fence_after();
                                const uint32_t s1 = s + 1 == nslots ? 0u : s + 1;
                                const uint32_t b_lo = b_lo0 + s * (uint32_t)(B_STAGE >> 4);
                                if (elected) {
#pragma unroll
                                    for (int q = 4 * j; q < 4 * j + 4 && q < NK; q++)
                                        mma(d_tmem, a_of(q), b_lo + 2u * (q & 3), (uint32_t)(cg | q));
                                    commit(bar_bempty + 8 * s);
                                    if (j == NST - 1) commit(bar_sempty + 8 * sl);
                                }
                                s = s1;
                                if (s1 == 0) ph ^= 1;
                            }
                        }
                        if ((sl += step) >= (uint32_t)p.nslab) { sl -= (uint32_t)p.nslab; slph ^= 1; }
                    }
                    if (elected) commit(bar_tfull + 8 * buf);
                }
            } else
            for (int t = unit; t < ntiles; t += nunits, lt++, first_tile = false) {
                const int buf = (int)(lt % NBUF);
                if (!mbar_wait(OVL ? bar_tempty : bar_tempty + 8 * buf, (OVL ? (lt & 1) : ((lt / NBUF) & 1)) ^ 1, abort_flag, p.status, 2))
                    goto done;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * ACC_OFF;
                uint32_t acc = 0;
                for (int cg = 0; cg < p.G; cg++) {
                    if (!mbar_wait(bar_sfull + 8 * sl, slph, abort_flag, p.status, 0x13)) goto done;
                    tc_fence_after();
                    const uint32_t slab_lo = a_lo0 + sl * slab16;
                    // tap (kh, kw) starts kh*Wp + kw rows into the slab: kept as running counters -- a table in
                    // shared memory would put a load, queued behind the MMAs just issued, in front of every MMA
                    uint32_t kwc = 0, rowoff = 0, tapoff = 0;
                    int tap = 0;
                    for (int j = 0; j < SPG; j++) {
                        const int c = (TAPS == 1) ? j * p.G + cg : j;
                        const uint32_t slot = p.b_resident ? (uint32_t)c : s;
                        if (!p.b_resident || first_tile) {
                            if (!mbar_wait(bar_bfull + 8 * slot, p.b_resident ? 0u : ph, abort_flag, p.status, 3)) goto done;
                            tc_fence_after();
                        }
                        const uint32_t b_lo = b_lo0 + slot * (uint32_t)(B_STAGE >> 4);
                        // offsets of the stage's four K steps (64 elements = 32 bytes of one tap's pixel row each)
                        uint32_t ak[4];
                        int steps = 0;
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const uint32_t koff = (TAPS == 1) ? 2u * k : (TAPS == 2 ? 2u * (k & 1) : 0u);
                            ak[k] = slab_lo + tapoff + koff;
                            if (TAPS == 1 || tap < p.T) steps = k + 1;
                            // the next K step belongs to the next tap: after every step (32-byte pixels), every second
                            // (64-byte pixels) or the stage's last (128-byte pixels)
                            if (TAPS == 4 || (TAPS == 2 && (k & 1)) || (TAPS == 1 && k == 3)) {
                                tap++;
                                if (++kwc == (uint32_t)p.KW) { kwc = 0; rowoff += row16; tapoff = rowoff; }
                                else tapoff += RB / 16;
                            }
                        }
                        if (elected) {
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (k < steps) mma(d_tmem, ak[k], b_lo + 2u * k, acc | (uint32_t)k);
                            if (!p.b_resident) commit(bar_bempty + 8 * s);
                        }
                        acc = 1;
                        if (!p.b_resident && ++s == (uint32_t)p.nstg) { s = 0; ph ^= 1; }
                    }
                    if (elected) commit(bar_sempty + 8 * sl);
                    if (++sl == (uint32_t)p.nslab) { sl = 0; slph ^= 1; }
                }
                if (elected) commit(bar_tfull + 8 * buf);
            }
        }
    } else if (warp == WARP_TMA) {
        // (done above)
    } else if (Cfg::LOADER && warp < WARP_EPI0) {
        // ---------------- slab loaders: every NLOAD-th tile of the block's sequence ----------------
        constexpr int NLOAD = Cfg::LOADER ? Cfg::NLOAD : 1;
        const int me = warp - Cfg::WARP_LOAD0;
        // piece i of a slab goes to byte 16*i with the swizzle pattern applied: address bits 4.. are XORed with bits 7.. (one bit for
        // 32-byte rows, two for 64-byte rows), and since a warp's 32 pieces are 512 bytes only the lane decides those
        const uint32_t lane_dst = (uint32_t)(lane * 16) ^ ((uint32_t)((lane >> 3) & (RB / 16 - 1)) << 4);
        const int pieces = p.slab_rows * (RB / 16);
        const long long total = (long long)p.Mv * (RB / 16);  // pieces of the image; past its end a slab is filled with zeros
        // Slabs requested and not yet announced, oldest first.  A fill may have to wait for the slab nslab fills before it to be
        // multiplied, so those this warp holds back must be younger than that.
        const int hold = min(2, (p.nslab - 1) / NLOAD);
        int held = 0;
        uint32_t sl = (uint32_t)me, slph = 1, oldest = (uint32_t)me;
        auto announce = [&]() {
            fence_proxy_async();  // these lanes' pieces -> visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sfull + 8 * oldest);
            oldest += NLOAD;
            if (oldest >= (uint32_t)p.nslab) oldest -= (uint32_t)p.nslab;
            held--;
        };
        for (int t = unit + me * nunits; t < ntiles; t += NLOAD * nunits) {
            const long long piece0 = (long long)p.div_ntn.div((uint32_t)t) * (TILE_M * (RB / 16));
            if (!mbar_wait(bar_sempty + 8 * sl, slph, abort_flag, p.status, 0x11)) goto done;
            const uint32_t dst = smem_u32(sA + sl * p.slab_bytes) + lane_dst;
            const unsigned char* src = p.Aimg + (size_t)piece0 * 16 + lane * 16;
            if (piece0 + pieces <= total) {
                int i = lane;
#pragma unroll 1
                for (; i + 7 * 32 < pieces; i += 8 * 32, src += 8 * 512) {
#pragma unroll
                    for (int u = 0; u < 8; u++) cp_async16(dst + (uint32_t)(i - lane + u * 32) * 16, src + u * 512, 16);
                }
                for (; i < pieces; i += 32, src += 512) cp_async16(dst + (uint32_t)(i - lane) * 16, src, 16);
            } else {
                for (int i = lane; i < pieces; i += 32, src += 512) {
                    const bool there = piece0 + i < total;
                    cp_async16(dst + (uint32_t)(i - lane) * 16, there ? src : p.Aimg, there ? 16 : 0);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (++held > hold) {
                if (hold == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
                else if (hold == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                announce();
            }
            sl += NLOAD;
            if (sl >= (uint32_t)p.nslab) { sl -= (uint32_t)p.nslab; slph ^= 1; }
        }
        if (held == 2) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            announce();
        }
        if (held == 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            announce();
        }
    } else if (QF && warp >= Cfg::WARP_Q0) {
        uint64_t* qbars = reinterpret_cast<uint64_t*>(q_ring + Q_STG * Cfg::Q_STAGE);
        if (warp < Cfg::WARP_Q0 + 4) {
            QuantArgs qa;
            qa.qthr = p.qthr; qa.qimg = p.qimg; qa.q_sync = p.q_sync; qa.qN = p.qN; qa.qC = p.qC; qa.q_nbands = p.q_nbands; qa.Cp = qa.pitch = p.Cp;
            qa.HW = p.q_H * p.q_W; qa.status = p.status;
            qa.W = p.q_W; qa.Wp = p.Wp; qa.HpWp = p.HpWp; qa.off0 = p.q_PH * p.Wp + p.q_PW; qa.border = 1; qa.binary = p.q_binary; qa.nhwc = 0;
            quantise_items(qa, &tmap_q, q_ring, qbars, abort_flag, tid - Cfg::WARP_Q0 * 32);
        } else if (lane == 0) {
            publish_items(p.q_sync, p.status, qbars, abort_flag);
        }
    } else if (warp >= WARP_EPI0 && warp < WARP_EPI0 + Cfg::NEPI) {
        // ---------------- epilogue ----------------
        const int q = warp & 3;                        // tensor-memory lane quadrant this warp may access
        const int ecol = ((warp - WARP_EPI0) >> 2) % EPW;         // which share of the columns
        const int group = NSETS == 1 ? 0 : ((warp - WARP_EPI0) >> 2) / EPW;
        // which tiles: every NSETS-th of the block's sequence; where no block has more than one (the launcher starts
        // two groups only), the groups share its columns
        const bool one_tile = NSETS > 1 && ntiles <= nunits;
        const int set = one_tile ? 0 : group, slice0 = one_tile ? group : 0, slice_step = one_tile ? ONE_TILE_GROUPS : 1;
        constexpr int ECOLS = BN / EPW;
        constexpr int NSL = ECOLS / 32;
        const bool alpha_in_unit = p.alpha > 0.f && p.alpha <= 1.f;
        const float bias_f = (float)p.acc_bias;
        const int OHW = p.OH * p.OW;
        uint32_t lt = (uint32_t)set;
        const uint32_t bar_release = (CG == 2 && rank != 0) ? mapa_shared(bar_tempty, 0) : 0u;
        // quantised output with 0 < alpha <= 1: PReLU and the next layer's rule collapse into thresholds on the accumulator
        const bool next_tern = !p.next_binary && p.next_format != 0;
        const bool img_out = IMG || (QF && p.pimg != nullptr);
        const bool by_thr = img_out && alpha_in_unit && (BN == 256 || p.next_format >= 2);
        tnns_thr::Pair qt = {0.f, 0.f};
        E2m1Rule qe = {0.f, 0.f};
        float qt_t = 0.f;
        bool qt_set = false;
        // pixel-major fp32 output: the accumulator is fetched in the 16x256b shape (four lanes = 32 contiguous bytes of a row)
        // -- float pairs (y_vec), or, in kernels of their own, single floats (SINGLE)
        const bool rows16 = !img_out && p.layout == TNNS_NHWC && (SINGLE || p.y_vec > 1);
        for (int t = unit + set * nunits; t < ntiles; t += NSETS * nunits, lt += NSETS) {
            const int buf = (int)(lt % NBUF);
            const int m_tile = (int)p.div_ntn.div((uint32_t)t), n0 = (t - m_tile * ntn) * BN;
            // where this thread's row sits in the lattice, and its image's threshold: worked out while the tile's MMAs run
            const int row = m_tile * TILE_M + (int)rank * BM + q * 32 + lane;  // virtual row
            const bool row_ok = row < p.Mv;
            const int n_img = row_ok ? (int)p.div_hpwp.div((uint32_t)row) : 0;
            const int rem = row - n_img * p.HpWp;
            const int yy = (int)p.div_wp.div((uint32_t)max(rem, 0)), xx = rem - yy * p.Wp;
            const bool valid = row_ok && yy < p.OH && xx < p.OW;   // a real output pixel (oh, ow) = (yy, xx)
            const int opix = yy * p.OW + xx;
            // (worked out here, while the tile's MMAs run: in the loop below it cost the fp32 layers up to a tenth)
            float* ybase = IMG ? nullptr : (p.layout == TNNS_NHWC) ? p.y + ((size_t)n_img * OHW + opix) * p.KN : p.y + (size_t)n_img * p.KN * OHW + opix;
            // 4-bit image out: where the row's pixel goes, nullptr if it has none.  In a bordered image a row that is no output pixel
            // (yy >= OH or xx >= OW) stands for one border pixel -- the next layer's padded lattice is this layer's: shifted by the
            // border and wrapped, the rows that are output pixels cover the interior and these rows exactly the frame.  They
            // write the padding value, so every launch rewrites the whole image and nothing has to be cleared beforehand.
            uint4* e_out = nullptr;
            if (img_out && p.next_format >= 2 && (valid || (row_ok && p.next_format == 3))) {
                uint32_t px = (uint32_t)(n_img * OHW + opix);
                if (p.next_format == 3) {
                    int y2 = yy + p.o_PH, x2 = xx + p.o_PW;
                    if (y2 >= p.o_Hp) y2 -= p.o_Hp;
                    if (x2 >= p.o_Wp) x2 -= p.o_Wp;
                    px = (uint32_t)(n_img * p.HpWp + y2 * p.o_Wp + x2);  // o_Hp * o_Wp = HpWp (checked by the launcher)
                }
                e_out = reinterpret_cast<uint4*>(p.pimg) + (size_t)px * (uint32_t)(p.cp_next * 2);
            }
            const float tq = (img_out && valid) ? __ldg(p.thr_next + n_img) + 0.0f : 0.f;
            if (by_thr && valid && !(qt_set && tq == qt_t)) {
                // the next layer's rule as thresholds on the raw accumulator, once per threshold this thread meets (images often share one)
                qt = tnns_thr::make(tq, p.alpha, bias_f, next_tern);
                qe = e2m1_rule(qt);
                qt_t = tq;
                qt_set = true;
            }
            // rows16: the four rows of the quadrant this thread stores (8*h + lane/4), each mapped to its output pixel
            float* yrow0[4] = {nullptr, nullptr, nullptr, nullptr};
            if (rows16) {
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int r = m_tile * TILE_M + (int)rank * BM + q * 32 + 8 * h + (lane >> 2);
                    if (r < p.Mv) {
                        const int ni = (int)p.div_hpwp.div((uint32_t)r);
                        const int rm = r - ni * p.HpWp;
                        const int y2 = (int)p.div_wp.div((uint32_t)rm), x2 = rm - y2 * p.Wp;
                        if (y2 < p.OH && x2 < p.OW) yrow0[h] = p.y + ((size_t)ni * OHW + (size_t)(y2 * p.OW + x2)) * p.KN;
                    }
                }
            }
            if (!mbar_wait(bar_tfull + 8 * buf, (lt / NBUF) & 1, abort_flag, p.status, 5)) goto done;
            tc_fence_after();
            int start = 0;
            if (OVL && buf == 0 && ecol == EPW - 1) start = NSL - 1;
#pragma unroll 1
            for (int i = slice0; i < NSL; i += slice_step) {
                const int cb = ecol * ECOLS + ((i + start) % NSL) * 32;
                uint32_t v[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * ACC_OFF + cb);
                if (rows16) {
                    tmem_ld_16x256b_x4(taddr, v);
                    tmem_ld_16x256b_x4(taddr + (16u << 16), v + 16);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (OVL ? (i == 0) : (i == NSL - 1)) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if (CG == 2 && rank != 0) mbar_arrive_cluster(bar_release + (OVL ? 0 : 8 * buf));
                            else mbar_arrive(OVL ? bar_tempty : bar_tempty + 8 * buf);
                        }
                    }
                    float f[32];
                    prelu32_f4(v, f, alpha_in_unit, p.acc_bias, bias_f, p.alpha, p.zero_passes);
                    const int c0 = n0 + cb;
                    float* const yrow[4] = {yrow0[0] ? yrow0[0] + c0 : nullptr, yrow0[1] ? yrow0[1] + c0 : nullptr,
                                            yrow0[2] ? yrow0[2] + c0 : nullptr, yrow0[3] ? yrow0[3] + c0 : nullptr};
                    if (SINGLE) store_rows16_single(f, yrow, p.KN - c0, lane);
                    else store_rows16_at(f, yrow, p.KN - c0, lane);
                    continue;
                }
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                      "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
                      "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
                      "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(taddr)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (OVL ? (i == 0) : (i == NSL - 1)) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 2 && rank != 0) mbar_arrive_cluster(bar_release + (OVL ? 0 : 8 * buf));
                        else mbar_arrive(OVL ? bar_tempty : bar_tempty + 8 * buf);
                    }
                }
                const int c0 = n0 + cb;
                if (by_thr && p.next_format >= 2 && c0 + 32 <= p.KN) {
                    if (e_out) {
                        uint32_t w4[4];
                        if (next_tern) quantise32_e2m1<true>(v, qe, w4);
                        else quantise32_e2m1<false>(v, qe, w4);
                        const uint32_t padw = next_tern ? 0u : 0x22222222u;
                        e_out[c0 >> 5] = valid ? make_uint4(w4[0], w4[1], w4[2], w4[3]) : make_uint4(padw, padw, padw, padw);
                    }
                } else if (valid) {
                    float f[32];
                    uint32_t sg = 0, nz = 0;
                    if (by_thr) {
                        if (next_tern) {
                            uint32_t above = 0;
#pragma unroll
                            for (int j = 31; j >= 0; j--) {
                                sg = push_sign(sg, __uint_as_float(v[j]) + qt.n1);
                                above = push_sign(above, qt.t2 - __uint_as_float(v[j]));
                            }
                            nz = sg | above;
                        } else {
#pragma unroll
                            for (int j = 31; j >= 0; j--) sg = push_sign(sg, __uint_as_float(v[j]) + qt.n1);
                        }
                    } else
                    // (the run-time choices are taken outside the unrolled loops: left inside, every element pays for
                    // both sides of each -- the epilogue warps share their schedulers with the MMA-issuing threads)
                    if (alpha_in_unit && p.acc_bias) {
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const float a = __uint_as_float(v[j]) + bias_f;
                            f[j] = fmaxf(a, fmaf(a, p.alpha, 0.0f));
                        }
                    } else if (alpha_in_unit) {
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const float a = __uint_as_float(v[j]);
                            f[j] = fmaxf(a, fmaf(a, p.alpha, 0.0f));
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++) {
                            const float ac = (p.acc_bias ? __uint_as_float(v[j]) + bias_f : __uint_as_float(v[j])) + 0.0f;
                            f[j] = ac * ((p.zero_passes ? ac >= 0.f : ac > 0.f) ? 1.0f : p.alpha);
                        }
                    }
                    const bool full = c0 + 32 <= p.KN;
                    if (img_out) {
                        if (c0 < p.cp_next * 64) {
                            const bool tern = next_tern;
                            if (!by_thr) {
                                if (tern) quantise32_ternary(f, tq, sg, nz);
                                else sg = quantise32_binary(f, tq);
                            }
                            const int have = p.KN - c0;
                            const uint32_t vmask = have >= 32 ? 0xFFFFFFFFu : (have > 0 ? (1u << have) - 1u : 0u);
                            if (p.next_format >= 2) {
                                // the 32 channels as 16 bytes of e2m1 operands; channels past KN: ternary 0, binary +1
                                uint32_t w4[4];
                                tnns_expand32_f4(sg & vmask, tern ? ~(nz & vmask) : 0u, w4);
                                e_out[c0 >> 5] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                            } else {
                                const int planes = tern ? 2 : 1;
                                const size_t lanes = (size_t)p.cp_next * 2;
                                uint32_t* px = p.pimg + ((size_t)n_img * planes * OHW + opix) * lanes + (c0 >> 5);
                                px[0] = sg & vmask;
                                if (tern) px[(size_t)OHW * lanes] = ~(nz & vmask);
                            }
                        }
                    } else if (p.layout == TNNS_NHWC) {
                        if (full && p.y_vec == 4) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4)
                                __stcs(reinterpret_cast<float4*>(ybase + c0 + j), make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (c0 + j < p.KN) __stcs(ybase + c0 + j, f[j]);
                        }
                    } else {
                        float* yc = ybase + (size_t)c0 * OHW;
                        if (full) {
#pragma unroll
                            for (int j = 0; j < 32; j++, yc += OHW) __stcs(yc, f[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++, yc += OHW)
                                if (c0 + j < p.KN) __stcs(yc, f[j]);
                        }
                    }
                } else if (e_out && c0 < p.cp_next * 64) {
                    const uint32_t padw = p.next_binary ? 0x22222222u : 0u;
                    e_out[c0 >> 5] = make_uint4(padw, padw, padw, padw);
                }
            }
        }
    }

done:
    __syncwarp();
    if (*abort_flag && warp == WARP_TMA && lane == 0) {
        // a wait gave up: give the copies already issued time to land before shared memory is released
        for (int i = 0; i < 1000; i++) __nanosleep(1000);
    }
    tc_fence_before();
    if (CG == 2) cluster_sync_all(); else __syncthreads();
    if (warp == WARP_MMA) {
        tc_fence_after();
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
    if (QF && p.q_self_clean && warp == WARP_TMA) {
        // the block that leaves last zeroes the synchronisation words for the next launch on the stream
        unsigned int left = 0;
        if (lane == 0) {
            __threadfence();
            left = atomicAdd(p.q_sync + 1, 1u);
        }
        left = __shfl_sync(0xFFFFFFFFu, left, 0);
        if (left == gridDim.x - 1) {
            __threadfence();
            for (int i = lane; i < Q_FLAG0 + p.qN; i += 32) p.q_sync[i] = 0;
        }
    }
}

template <int BN, int CG, int TAPS, bool QF, bool SINGLE = false, int GRP = 1, bool IMG = false>
int launch_slab(tnns_cuda_ctx* ctx, const SlabArgs& a, size_t smem, cudaStream_t stream, const CUtensorMap* tmap_a, const CUtensorMap* tmap_b,
                const CUtensorMap* tmap_q) {
    using Cfg = SlabCfg<BN, CG, TAPS, QF, IMG>;
    auto kern = gemm_slab_kernel<BN, CG, TAPS, QF, SINGLE, GRP, IMG>;
    const auto maps = tensor_maps<maps_of(CG, QF)>(tmap_a, tmap_b, tmap_q);
    static bool smem_set[64] = {false};  // once per kernel and device
    if (!smem_set[ctx->device & 63]) {
        TNNS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_MAX));
        smem_set[ctx->device & 63] = true;
    }
    const long long tiles = (long long)((a.Mv + CG * BM - 1) / (CG * BM)) * ((a.KN + BN - 1) / BN);
    cudaLaunchAttribute attr[2];
    int nattr = 0;
    attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[nattr].val.programmaticStreamSerializationAllowed = 1;
    nattr++;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(!QF && Cfg::NSETS > 1 && tiles <= ctx->sm_count ? 32 * (Cfg::WARP_EPI0 + 4 * ONE_TILE_GROUPS) : Cfg::NTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    if (CG == 1) {
        cfg.gridDim = dim3((int)std::min<long long>(tiles, ctx->sm_count));
    } else {
        attr[nattr].id = cudaLaunchAttributeClusterDimension;
        attr[nattr].val.clusterDim.x = CG;
        attr[nattr].val.clusterDim.y = 1;
        attr[nattr].val.clusterDim.z = 1;
        nattr++;
        static int max_pairs[64] = {0};  // per device; measured with the largest shared-memory request
        int& mp = max_pairs[ctx->device & 63];
        if (mp == 0) {
            cfg.gridDim = dim3(CG * (ctx->sm_count / CG));
            cfg.dynamicSmemBytes = Cfg::SMEM_MAX;
            cfg.attrs = attr;
            cfg.numAttrs = nattr;
            int n = 0;
            TNNS_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
            if (n <= 0) return tnns_fail(TNNS_ERR_CUDA, "no block pair of the slab-fed GEMM fits this device");
            mp = std::min(n, ctx->sm_count / CG);
            cfg.dynamicSmemBytes = smem;
        }
        cfg.gridDim = dim3(CG * (int)std::min<long long>(tiles, mp));
    }
    cfg.attrs = attr;
    cfg.numAttrs = nattr;
    TNNS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a, maps));
    tnns_count_launch();
    TNNS_CUDA_TRY(cudaGetLastError());
    return TNNS_OK;
}

struct SlabPlan {
    int taps, rb, G, T, Wp, Hp, slab_rows, ncopies, copy_rows, slab_bytes, bn;
};

bool make_plan(const tnns_cuda_weights* w, const TnnsGeom& g, SlabPlan* pl) {
    if (!w->d_f4 || w->Kp >= 65536) return false;
    if (g.SH != 1 || g.SW != 1) return false;                      // the virtual lattice is the padded input lattice
    if (g.Cp != 1 && g.Cp != 2 && g.Cp % 4 != 0) return false;     // a pixel = 32, 64 or a multiple of 128 bytes
    pl->taps = g.Cp == 1 ? 4 : (g.Cp == 2 ? 2 : 1);
    pl->rb = 128 / pl->taps;
    pl->G = g.Cp >= 4 ? g.Cp / 4 : 1;
    pl->T = g.KH * g.KW;
    if (pl->T > SL_TAPMAX) return false;
    pl->Wp = g.W + 2 * g.PW;
    pl->Hp = g.H + 2 * g.PH;
    if ((long long)g.N * pl->Hp * pl->Wp >= 0x7FFFFFFFLL - 4096) return false;  // virtual rows are 32-bit
    pl->slab_rows = BM + (g.KH - 1) * pl->Wp + (g.KW - 1);
    pl->ncopies = (pl->slab_rows + 255) / 256;                     // a tensor copy moves at most 256 rows
    if (pl->ncopies > 4) return false;
    // every copy starts on a whole swizzle atom (eight rows) of the slab buffer
    pl->copy_rows = (((pl->slab_rows + pl->ncopies - 1) / pl->ncopies) + 7) & ~7;
    pl->slab_bytes = (pl->ncopies * pl->copy_rows * pl->rb + 1023) & ~1023;
    pl->bn = tnns_i8_tile_n(w->KN);
    return true;
}

}  // namespace

namespace {
struct SlabChoice {
    SlabPlan pl;
    bool pairs;
    bool loaders;
    int b_stage, fixed, grp, Mv, ntn;
    SlabRings rings;
    size_t smem;
};
// The form a launch takes: single blocks or block pairs (pairs_req 0 = by size, 1, 2), ring depths.
bool choose_form(int sm_count, const tnns_cuda_weights* w, const TnnsGeom& g, int pairs_req, bool fused, bool image_out, SlabChoice* ch) {
    if (!make_plan(w, g, &ch->pl)) return false;
    const SlabPlan& pl = ch->pl;
    ch->Mv = g.N * pl.Hp * pl.Wp;
    ch->ntn = (w->KN + pl.bn - 1) / pl.bn;
    const long long pair_tiles = (long long)((ch->Mv + 2 * BM - 1) / (2 * BM)) * ch->ntn;
    if (pairs_req == 2 && pl.bn != 256) return false;
    ch->pairs = pl.bn == 256 && (pairs_req == 2 || (pairs_req == 0 && pair_tiles >= sm_count / 2));
    // Slab loaders (SlabCfg::LOADER) where 32- or 64-byte pixels become an image.  fp32 outputs keep the tensor copies: the loaders'
    // pieces would queue behind the output's stores in the same unit (256 x 64x56x56 -> 64 fp32 out, copies / loaders: 52 / 60 us).
    ch->loaders = image_out && pl.taps > 1 && !ch->pairs && !fused;
    ch->b_stage = (pl.bn / (ch->pairs ? 2 : 1)) * KCH;
    ch->fixed = 1024 + SL_BAR_BYTES + (fused ? Q_STG * Q_PIX * 64 * 4 + 128 : 0);
    auto rings = [&]() {
        const SlabFeed feed = !ch->loaders ? SLAB_COPIES : (ch->pl.bn == 64 && pl.T == 9 && g.KW == 3) ? SLAB_LOADERS_TWO : SLAB_LOADERS;
        return slab_rings(pl.slab_bytes, ch->b_stage, 232448 - ch->fixed, w->Kp / 4, ch->ntn == 1, feed, &ch->rings);
    };
    if (!rings()) return false;
    if (!ch->pairs && !fused) {
        // few tiles: narrower ones (what fits with the widest tile fits with these)
        const int bn = tile_n_for(sm_count, ch->Mv, w->KN, pl.bn);
        if (bn != pl.bn) {
            ch->pl.bn = bn;
            ch->ntn = (w->KN + bn - 1) / bn;
            ch->b_stage = bn * KCH;
            if (!rings()) return false;
        }
    }
    // three weight stages a slot (see the kernel's GRP) where two slots fit
    SlabRings& r = ch->rings;
    ch->grp = (pl.taps == 1 && g.KH == 3 && g.KW == 3 && !r.resident && !ch->pairs && !fused && ch->pl.bn <= 128 && r.nstg >= 6) ? 3 : 1;
    r.nstg -= r.nstg % ch->grp;
    ch->smem = (size_t)ch->fixed + (size_t)r.nslab * pl.slab_bytes + (size_t)r.nstg * ch->b_stage;
    return true;
}
}  // namespace

bool tnns_slab_supported(const tnns_cuda_ctx* ctx, const tnns_cuda_weights* w, const TnnsGeom& g, bool fused) {
    SlabChoice ch;
    return choose_form(ctx->sm_count, w, g, 0, fused, false, &ch);
}

size_t tnns_bordered_image_bytes(int N, int C, int H, int W, int PH, int PW) {
    if (N < 0 || C <= 0 || H <= 0 || W <= 0 || PH < 0 || PW < 0) return 0;
    return (size_t)N * (H + 2 * PH) * (W + 2 * PW) * ((C + TNNS_WORD_BITS - 1) / TNNS_WORD_BITS) * 32;
}

int tnns_launch_gemm_slab(tnns_cuda_ctx* ctx, const tnns_cuda_weights* w, const void* d_image, float* d_y, const TnnsGeom& g, float alpha, int layout,
                          cudaStream_t stream, int pairs, void* d_pimg, const float* d_thr_next, int next_format, int next_binary, int next_PH,
                          int next_PW, const TnnsFusedInput* fused) {
    if (g.N == 0) return TNNS_OK;
    SlabChoice ch;
    if (!choose_form(ctx->sm_count, w, g, pairs, fused != nullptr, d_pimg != nullptr, &ch))
        return tnns_fail(TNNS_ERR_UNSUPPORTED, "layer outside the slab-fed GEMM (stride 1; 64, 128 or 256*k channels; slab and weight ring within shared memory)");
    const SlabPlan& pl = ch.pl;
    if (reinterpret_cast<uintptr_t>(d_image) & 127) return tnns_fail(TNNS_ERR_INVALID, "bordered image must be 128-byte aligned");
    const bool act_binary = w->type == BTN || w->type == BNN;
    const int Mv = ch.Mv;
    const bool use_pairs = ch.pairs;
    const size_t smem = ch.smem;
    SlabArgs a = {};
    a.nslab = ch.rings.nslab; a.nstg = ch.rings.nstg; a.b_resident = ch.rings.resident;
    a.Bimg = reinterpret_cast<const unsigned char*>(w->d_f4);
    a.y = d_y;
    a.Mv = Mv;
    a.KN = w->KN;
    a.nchunks = w->Kp / 4;
    a.b_rows = tnns_i8_tile_n(w->KN);
    a.b_shift = a.b_rows == 64 ? 6 : a.b_rows == 128 ? 7 : 8;
    a.div_ntn = tnns_fastdiv((uint32_t)ch.ntn);
    a.y_vec = tnns_row_vec(d_y, w->KN);
    a.OH = g.OH; a.OW = g.OW; a.Wp = pl.Wp; a.HpWp = pl.Hp * pl.Wp;
    a.KW = g.KW; a.T = pl.T; a.G = pl.G;
    a.Aimg = reinterpret_cast<const unsigned char*>(d_image);
    a.slab_rows = pl.slab_rows;
    a.slab_bytes = pl.slab_bytes; a.copy_rows = pl.copy_rows; a.ncopies = pl.ncopies;
    a.layout = (g.OH * g.OW == 1) ? TNNS_NHWC : layout;  // one pixel per image: both layouts are the same memory, the pixel-major epilogue stores 16 bytes per lane
    a.zero_passes = w->type != TNN;
    // BNN counts its products: pad words are never multiplied here, absent channels (+1 x +1) are
    a.acc_bias = (w->type == BNN) ? w->K_unpack - 64 * w->Kw : 0;
    a.alpha = alpha;
    a.status = ctx->d_status;
    a.pimg = reinterpret_cast<uint32_t*>(d_pimg);
    a.thr_next = d_thr_next;
    a.next_format = next_format;
    a.next_binary = next_binary;
    a.cp_next = (w->KN + TNNS_WORD_BITS - 1) / TNNS_WORD_BITS;
    a.o_PH = next_PH; a.o_PW = next_PW; a.o_Hp = g.OH + 2 * next_PH; a.o_Wp = g.OW + 2 * next_PW;
    if (d_pimg && next_format == 3 && (a.o_Hp != pl.Hp || a.o_Wp != pl.Wp))
        return tnns_fail(TNNS_ERR_UNSUPPORTED, "a bordered output image needs the next layer's padded size (%d x %d) to equal this layer's (%d x %d)",
                         a.o_Hp, a.o_Wp, pl.Hp, pl.Wp);
    a.Cp = g.Cp;
    a.div_hpwp = tnns_fastdiv((uint32_t)a.HpWp);
    a.div_wp = tnns_fastdiv((uint32_t)pl.Wp);
    // the bordered image as rows of pixels: (bytes of a pixel) x (all padded pixels of the batch)
    alignas(64) CUtensorMap map_a, map_b, map_q;
    int rc = ch.loaders ? TNNS_OK : tnns_tensor_map_2d(&map_a, 1, d_image, (unsigned long long)g.Cp * 32, (unsigned long long)Mv, (unsigned long long)g.Cp * 32, pl.rb,
                                pl.copy_rows, pl.rb);
    if (rc) return rc;
    if (use_pairs && (rc = tnns_tensor_map_2d(&map_b, 1, w->d_f4, KCH, w->f4_bytes / KCH, KCH, KCH, pl.bn / 2))) return rc;
    if (fused) {
        if (!fused->d_x || !fused->d_thr || !fused->d_sync) return tnns_fail(TNNS_ERR_INVALID, "NULL argument");
        if (!tnns_quantise_tma_supported(fused->d_x, g.H, g.W, layout))
            return tnns_fail(TNNS_ERR_UNSUPPORTED, "fused quantisation needs NCHW input with H*W a multiple of four and a 16-byte aligned base");
        const unsigned long long HW = (unsigned long long)g.H * g.W;
        if ((rc = tnns_tensor_map_nchw(&map_q, fused->d_x, g.N, g.C, (long long)HW, Q_PIX, 64))) return rc;
        unsigned int* words = nullptr;
        int self_clean = 0;
        if ((rc = tnns_fused_sync_prepare(ctx, g.N, stream, fused->d_sync, &words, &self_clean))) return rc;
        a.qthr = fused->d_thr;
        a.qimg = reinterpret_cast<uint4*>(const_cast<void*>(d_image));
        a.q_sync = words;
        a.q_self_clean = self_clean;
        a.qN = fused->starve ? 0 : g.N; a.qC = g.C; a.q_H = g.H; a.q_W = g.W; a.q_PH = g.PH; a.q_PW = g.PW;
        a.q_nbands = (g.H * g.W + Q_PIX - 1) / Q_PIX;
        a.q_binary = act_binary ? 1 : 0;
    }
    auto go = [&](auto taps_c) -> int {
        constexpr int T = decltype(taps_c)::value;
        if (fused) {
            if (use_pairs) return launch_slab<256, 2, T, true>(ctx, a, smem, stream, &map_a, &map_b, &map_q);
            switch (pl.bn) {
                case 64: return launch_slab<64, 1, T, true>(ctx, a, smem, stream, &map_a, nullptr, &map_q);
                case 128: return launch_slab<128, 1, T, true>(ctx, a, smem, stream, &map_a, nullptr, &map_q);
                default: return launch_slab<256, 1, T, true>(ctx, a, smem, stream, &map_a, nullptr, &map_q);
            }
        }
        const CUtensorMap* ma = ch.loaders ? nullptr : &map_a;
        if (d_pimg) {
            if (use_pairs) return launch_slab<256, 2, T, false, false, 1, true>(ctx, a, smem, stream, ma, &map_b, nullptr);
            if constexpr (T == 1)
                if (ch.grp == 3) return pl.bn == 64 ? launch_slab<64, 1, T, false, false, 3, true>(ctx, a, smem, stream, ma, nullptr, nullptr)
                                                    : launch_slab<128, 1, T, false, false, 3, true>(ctx, a, smem, stream, ma, nullptr, nullptr);
            switch (pl.bn) {
                case 64: return launch_slab<64, 1, T, false, false, 1, true>(ctx, a, smem, stream, ma, nullptr, nullptr);
                case 128: return launch_slab<128, 1, T, false, false, 1, true>(ctx, a, smem, stream, ma, nullptr, nullptr);
                default: return launch_slab<256, 1, T, false, false, 1, true>(ctx, a, smem, stream, ma, nullptr, nullptr);
            }
        }
        const bool single = single_floats(a.layout, a.y_vec, d_pimg);
        if (use_pairs) return single ? launch_slab<256, 2, T, false, true>(ctx, a, smem, stream, &map_a, &map_b, nullptr)
                                     : launch_slab<256, 2, T, false>(ctx, a, smem, stream, &map_a, &map_b, nullptr);
        if constexpr (T == 1)
            if (ch.grp == 3) {
                if (pl.bn == 64) return single ? launch_slab<64, 1, T, false, true, 3>(ctx, a, smem, stream, &map_a, nullptr, nullptr)
                                               : launch_slab<64, 1, T, false, false, 3>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
                return single ? launch_slab<128, 1, T, false, true, 3>(ctx, a, smem, stream, &map_a, nullptr, nullptr)
                              : launch_slab<128, 1, T, false, false, 3>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
            }
        if (single) {
            switch (pl.bn) {
                case 64: return launch_slab<64, 1, T, false, true>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
                case 128: return launch_slab<128, 1, T, false, true>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
                default: return launch_slab<256, 1, T, false, true>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
            }
        }
        switch (pl.bn) {
            case 64: return launch_slab<64, 1, T, false>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
            case 128: return launch_slab<128, 1, T, false>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
            default: return launch_slab<256, 1, T, false>(ctx, a, smem, stream, &map_a, nullptr, nullptr);
        }
    };
    if (pl.taps == 4) return go(std::integral_constant<int, 4>());
    if (pl.taps == 2) return go(std::integral_constant<int, 2>());
    return go(std::integral_constant<int, 1>());
}
