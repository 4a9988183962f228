// Quantise-only kernels for inputs the copy engine cannot fetch (the thresholding half of t2r_p2_opt / b2r,
// reference: src/tnns/ternarize2row_avx2.c:438-452, src/tnns/binarize2row_avx2.c:15-22), and the launcher that
// picks a quantise kernel for a tensor.
//
// The copy engine wants rows of a multiple of 16 bytes.  NCHW images with H*W no multiple of four, pixel-major
// images whose channel count is none, unaligned bases and tiny tensors are read here with plain loads:
//
//   quantise_px_kernel   (NCHW)  a warp owns 32 neighbouring pixels and 32 channels: every load is 128 contiguous
//                        bytes at whatever alignment, sixteen of them in flight per lane.  Pixels are numbered
//                        through the whole batch, so small odd images leave no ragged ends per image.
//   quantise_row_kernel  (NHWC)  a warp owns 32 consecutive (pixel, 32 channels) pieces: lane = channel, two
//                        ballots make a piece's plane words, lane j keeps piece j, and all 32 lanes store at
//                        once -- 512 contiguous bytes of the 4-bit image.
//
// Both are bound by the 4 bytes read per value.  Work is cut so finely (32 pixels x 32 channels) that a layer of a
// few thousand pixels still fills the chip.  Measured inside the layer call against the band-per-block kernel that
// read such tensors before (quantise part, us): 8 x 320x15x23 17 -> 6, 14 x 256x35x35 15 -> 6, 128 x 96x27x27
// 31 -> 17 (2.8 TB/s), NHWC 63 x 262x21x20 229 -> 24, NHWC binary 86 x 3x224x224 726 -> 314.
#include <algorithm>
#include <type_traits>

#include "internal.h"

namespace {

constexpr int QA_THREADS = 256;

// where pixel `pix` of image n sits in the image, in pixels (plain image: Wp = W, HpWp = H*W, off0 = 0)
struct QaGeom {
    int C, HW, Cp, pitch;  // channels, pixels per image, 64-channel words per pixel, words per pixel of the 4-bit image
    int W, Wp, HpWp, off0, H, PH, PW;
    int N;
    FastDiv div_hw, div_w, div_halves;
    long long pixels;      // N * HW
};

__device__ __forceinline__ uint32_t push_bit(uint32_t acc, float d) { return __funnelshift_l(__float_as_uint(d), acc, 1); }

__device__ __forceinline__ uint32_t image_of(const QaGeom& g, long long P) {
    return P < 0xFFFFFFFFLL ? g.div_hw.div((uint32_t)P) : (uint32_t)(P / g.HW);
}

// 32 channels (half h of the pixel's words) of pixel `pix` of image n
template <bool TERNARY, int IMG>
__device__ __forceinline__ void store_half(const QaGeom& g, void* out, uint32_t n, int pix, int h, uint32_t sg, uint32_t nz) {
    if (!TERNARY) nz = 0xFFFFFFFFu;  // the binary alphabet has no zero; absent channels read +1
    if (IMG == TNNS_IMG_E2M1) {
        uint32_t w[4];
        tnns_expand32_f4(sg, ~nz, w);
        const int y = (int)g.div_w.div((uint32_t)pix), x = pix - y * g.W;
        uint4* dst = reinterpret_cast<uint4*>(out) + ((size_t)n * g.HpWp + (size_t)y * g.Wp + x + g.off0) * g.pitch * 2 + h;
        *dst = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
        uint32_t* img = reinterpret_cast<uint32_t*>(out);
        const size_t planes = TERNARY ? 2 : 1;
        const size_t at = ((size_t)n * planes * g.HW + pix) * (2 * g.Cp) + h;
        img[at] = sg;
        if (TERNARY) img[at + (size_t)g.HW * (2 * g.Cp)] = ~nz;
    }
}

// the frame of a bordered image: only its pixels are visited (two bands of PH rows, then PW columns on either side)
template <bool TERNARY>
__device__ __forceinline__ void fill_frame(const QaGeom& g, void* out) {
    const uint32_t padw = TERNARY ? 0u : 0x22222222u;
    const uint4 pad4 = make_uint4(padw, padw, padw, padw);
    // (whole warps dealt out over the blocks)
    tnns_fill_frame(reinterpret_cast<uint4*>(out), pad4, g.N, g.H, g.W, g.PH, g.PW, g.pitch * 2, 2 * g.Cp,
                    ((long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31), (long long)gridDim.x * QA_THREADS);
}

template <bool TERNARY, int IMG>
__global__ void __launch_bounds__(QA_THREADS)
quantise_px_kernel(const float* __restrict__ x, const float* __restrict__ thr, void* __restrict__ out, QaGeom g) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the input may be the output of the launch before
    if (IMG == TNNS_IMG_E2M1 && g.HpWp != g.HW) fill_frame<TERNARY>(g, out);
    const int lane = threadIdx.x & 31;
    const int halves = 2 * g.Cp;
    const long long units = ((g.pixels + 31) / 32) * halves;
    for (long long u = (long long)blockIdx.x * (QA_THREADS / 32) + (threadIdx.x >> 5); u < units; u += (long long)gridDim.x * (QA_THREADS / 32)) {
        const long long pb = u < 0xFFFFFFFFLL ? (long long)g.div_halves.div((uint32_t)u) : u / halves;
        const int h = (int)(u - pb * halves);
        const long long P = pb * 32 + lane;
        if (P >= g.pixels) continue;
        const uint32_t n = image_of(g, P);
        const int pix = (int)(P - (long long)n * g.HW);
        const int nch = min(32, g.C - 32 * h);
        const float t = __ldg(thr + n) + 0.0f;  // + 0.0f: a threshold of -0 behaves as +0
        const float* p = x + ((size_t)n * g.C + 32 * (size_t)h) * g.HW + pix;
        uint32_t sg = 0, nz = 0;
        // channel b ends at bit b: visit downwards and shift left; the predicates are read off sign bits
        // (v < -t <=> signbit(v + t); |v| > t <=> signbit(t - |v|); binary v < t <=> signbit(v - t))
        if (nch == 32) {
#pragma unroll
            for (int b0 = 16; b0 >= 0; b0 -= 16) {
                float v[16];
#pragma unroll
                for (int b = 0; b < 16; b++) v[b] = __ldg(p + (size_t)(b0 + b) * g.HW);
#pragma unroll
                for (int b = 15; b >= 0; b--) {
                    if (TERNARY) {
                        sg = push_bit(sg, v[b] + t);
                        nz = push_bit(nz, t - fabsf(v[b]));
                    } else {
                        sg = push_bit(sg, (v[b] + 0.0f) - t);
                    }
                }
            }
        } else {
            // ragged group: sixteen or eight loads at once, the last channel's again for those past it, their bits masked off (as a
            // loop over the channels its remainder ran one load at a time: 843 x 30x15x79 71 us, 1371 x 30x27x27 binary 66; now 38 and 36)
            auto load = [&](auto count, int b0) {
                constexpr int COUNT = decltype(count)::value;
                float v[COUNT];
#pragma unroll
                for (int b = 0; b < COUNT; b++) v[b] = __ldg(p + (size_t)min(b0 + b, nch - 1) * g.HW);
#pragma unroll
                for (int b = COUNT - 1; b >= 0; b--) {
                    if (TERNARY) {
                        sg = push_bit(sg, v[b] + t);
                        nz = push_bit(nz, t - fabsf(v[b]));
                    } else {
                        sg = push_bit(sg, (v[b] + 0.0f) - t);
                    }
                }
            };
            for (int b0 = nch > 16 ? 16 : 0; b0 >= 0 && nch > 0; b0 -= 16) {
                if (nch - b0 > 8) load(std::integral_constant<int, 16>(), b0);
                else load(std::integral_constant<int, 8>(), b0);
            }
            sg &= tnns_low_bits(nch);  // channels at or past nch: sign 0, non-zero 0
            nz &= tnns_low_bits(nch);
        }
        store_half<TERNARY, IMG>(g, out, n, pix, h, sg, nz);
    }
}

template <bool TERNARY, int IMG>
__global__ void __launch_bounds__(QA_THREADS)
quantise_row_kernel(const float* __restrict__ x, const float* __restrict__ thr, void* __restrict__ out, QaGeom g) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (IMG == TNNS_IMG_E2M1 && g.HpWp != g.HW) fill_frame<TERNARY>(g, out);
    const int lane = threadIdx.x & 31;
    const int halves = 2 * g.Cp;
    const long long pieces = g.pixels * halves;
    for (long long u = (long long)blockIdx.x * (QA_THREADS / 32) + (threadIdx.x >> 5); u * 32 < pieces; u += (long long)gridDim.x * (QA_THREADS / 32)) {
        const long long i0 = u * 32;
        long long P = i0 < 0xFFFFFFFFLL ? (long long)g.div_halves.div((uint32_t)i0) : i0 / halves;
        int h = (int)(i0 - P * halves);
        uint32_t n = image_of(g, P);
        int pix = (int)(P - (long long)n * g.HW);
        float t = __ldg(thr + n) + 0.0f;
        const float* px = x + (size_t)P * g.C;  // all warp-uniform: the piece walk below keeps them up to date
        uint32_t my_s = 0, my_z = 0;
#pragma unroll 1
        for (int j0 = 0; j0 < 32; j0 += 8) {
            float v[8], tj[8];
            bool ok[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int c = 32 * h + lane;
                ok[j] = c < g.C && i0 + j0 + j < pieces;
                v[j] = ok[j] ? __ldg(px + c) : 0.f;
                tj[j] = t;
                if (++h == halves) {
                    h = 0;
                    px += g.C;
                    if (++pix == g.HW) {
                        pix = 0;
                        if (++n < (uint32_t)g.N) t = __ldg(thr + n) + 0.0f;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint32_t s = __ballot_sync(0xFFFFFFFFu, ok[j] && v[j] < (TERNARY ? -tj[j] : tj[j]));
                const uint32_t z = TERNARY ? __ballot_sync(0xFFFFFFFFu, ok[j] && fabsf(v[j]) > tj[j]) : 0u;
                if (lane == j0 + j) { my_s = s; my_z = z; }
            }
        }
        const long long i = i0 + lane;
        if (i < pieces) {
            const long long Pl = i < 0xFFFFFFFFLL ? (long long)g.div_halves.div((uint32_t)i) : i / halves;
            const uint32_t nl = image_of(g, Pl);
            store_half<TERNARY, IMG>(g, out, nl, (int)(Pl - (long long)nl * g.HW), (int)(i - Pl * halves), my_s, my_z);
        }
    }
}

}  // namespace

// Quantise only: fp32 tensor -> packed image (bit planes) or 4-bit operand image, plain or bordered by PH rows / PW
// columns of the padding value.  pitch_words: 64-channel words from one pixel of the 4-bit image to the next (0: the
// pixel's own; words past those are left as they are).
int tnns_launch_quantise(tnns_cuda_ctx* ctx, bool ternary, const float* d_x, const float* d_thr, void* d_image, int N, int C, int H,
                         int W, int layout, cudaStream_t stream, int format, int PH, int PW, int pitch_words) {
    if (N == 0) return TNNS_OK;
    if (format != TNNS_IMG_PLANES && format != TNNS_IMG_E2M1) return tnns_fail(TNNS_ERR_INVALID, "unknown image format %d", format);
    if ((PH || PW || pitch_words) && format != TNNS_IMG_E2M1) return tnns_fail(TNNS_ERR_INVALID, "only the 4-bit image has a border or a pitch");
    if (layout != TNNS_NCHW && layout != TNNS_NHWC) return tnns_fail(TNNS_ERR_INVALID, "unknown layout %d", layout);
    if (tnns_quantise_tma_supported(d_x, H, W, layout))
        return tnns_launch_quantise_tma(ctx, ternary, d_x, d_thr, d_image, N, C, H, W, stream, format, PH, PW, TNNS_NCHW, pitch_words);
    // (a 1x1 image is the same memory in both layouts: fully connected layers are read as pixel-major)
    const bool rows = layout == TNNS_NHWC || H * W == 1;
    if (rows && tnns_quantise_tma_nhwc_supported(d_x, N, C, H, W))
        return tnns_launch_quantise_tma(ctx, ternary, d_x, d_thr, d_image, N, C, H, W, stream, format, PH, PW, TNNS_NHWC, pitch_words);
    QaGeom g;
    g.N = N; g.C = C; g.H = H; g.W = W; g.HW = H * W; g.PH = PH; g.PW = PW;
    g.Cp = (C + TNNS_WORD_BITS - 1) / TNNS_WORD_BITS;
    g.pitch = pitch_words ? pitch_words : g.Cp;
    g.Wp = W + 2 * PW; g.HpWp = (H + 2 * PH) * g.Wp; g.off0 = PH * g.Wp + PW;
    g.pixels = (long long)N * g.HW;
    g.div_hw = tnns_fastdiv((uint32_t)g.HW);
    g.div_w = tnns_fastdiv((uint32_t)W);
    g.div_halves = tnns_fastdiv((uint32_t)(2 * g.Cp));
    const long long units = rows ? (g.pixels * 2 * g.Cp + 31) / 32 : ((g.pixels + 31) / 32) * 2 * g.Cp;
    const int grid = (int)std::min<long long>((units + QA_THREADS / 32 - 1) / (QA_THREADS / 32), (long long)ctx->sm_count * 8);
    auto launch = [&](auto kern) -> int {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(QA_THREADS);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        TNNS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, d_x, d_thr, d_image, g));
        tnns_count_launch();
        TNNS_CUDA_TRY(cudaGetLastError());
        return TNNS_OK;
    };
    const bool e2m1 = format == TNNS_IMG_E2M1;
    if (rows) {
        if (e2m1) return ternary ? launch(quantise_row_kernel<true, TNNS_IMG_E2M1>) : launch(quantise_row_kernel<false, TNNS_IMG_E2M1>);
        return ternary ? launch(quantise_row_kernel<true, TNNS_IMG_PLANES>) : launch(quantise_row_kernel<false, TNNS_IMG_PLANES>);
    }
    if (e2m1) return ternary ? launch(quantise_px_kernel<true, TNNS_IMG_E2M1>) : launch(quantise_px_kernel<false, TNNS_IMG_E2M1>);
    return ternary ? launch(quantise_px_kernel<true, TNNS_IMG_PLANES>) : launch(quantise_px_kernel<false, TNNS_IMG_PLANES>);
}
