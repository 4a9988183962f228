// Layers with few input channels (the first layer of an image network: C = 3) as a dense GEMM.
//
// The reference pads every filter tap to 64 channels (`C_pack = ceil(C/64)`, plane word
// `j = (kh*KW + kw)*C_pack + ic`, src/tnns/ternarize2row_avx2.c:285-313), so a 7x7 filter over 3 channels
// is a row of 49 plane words = 3136 positions of which 147 can be non-zero, and every route that follows
// that layout multiplies (and fetches) the 2989 zeros as well.  Zeros contribute nothing to the sum, so
// the same output comes from a row that holds only the real positions: element `e = (kh*KW + kw)*C + c`,
// K = KH*KW*C, rounded up to a channel count the tensor-core GEMM takes (64, 128 or a multiple of 256).
// Two small kernels make that a layer the existing GEMMs run unchanged:
//   * repack_weights_dense_kernel (once per weight upload) writes the packed kernel of a VIRTUAL layer
//     -- 1x1 filter, K' channels -- in the reference's own packed format; the ordinary upload path then
//     builds its operand images;
//   * dense_quantise_kernel (per call) quantises the fp32 input with the reference's rule
//     (src/tnns/ternarize2row_avx2.c:438-452) and writes, per output pixel, the K' positions of its window
//     as the 4-bit image of that virtual layer (positions outside the input or past K: zero).
// The GEMM is then the copy-engine fed one on a 1x1, stride-1 layer over N x OH x OW "pixels" of K'
// "channels", with every epilogue it has.  Ternary activations only (TNN, TBN): a binary window pads
// with +1, which the zero positions of this form cannot express.
#include <algorithm>
#include <cmath>

#include "internal.h"

namespace {

// bit `c` of plane word (tap, c / 64) of the parent row -> bit e % 64 of virtual plane word e / 64
__global__ void repack_weights_dense_kernel(const uint64_t* __restrict__ packed, uint64_t* __restrict__ out, int KN, int Kp, int Cp, int C,
                                            int T, int two_planes, int Kp_out) {
    const long long total = (long long)KN * Kp_out;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int kn = (int)(i / Kp_out), jo = (int)(i - (long long)kn * Kp_out);
        const uint64_t* row = packed + (size_t)kn * Kp * (two_planes ? 2 : 1);
        uint64_t sign = 0, zero = ~0ull;  // positions past K: ternary 0 (a binary plane reads +1 there; the activations are 0)
        for (int b = 0; b < 64; b++) {
            const int e = jo * 64 + b;
            if (e >= T * C) break;
            const int tap = e / C, c = e - tap * C;
            const int j = tap * Cp + (c >> 6), bit = c & 63;
            if (two_planes) {
                const uint64_t s = row[(j >> 2) * 8 + (j & 3)], z = row[(j >> 2) * 8 + 4 + (j & 3)];
                sign |= ((s >> bit) & 1ull) << b;
                zero = (zero & ~(1ull << b)) | (((z >> bit) & 1ull) << b);
            } else {
                sign |= ((row[j] >> bit) & 1ull) << b;
            }
        }
        if (two_planes) {
            uint64_t* orow = out + (size_t)kn * Kp_out * 2;
            orow[(jo >> 2) * 8 + (jo & 3)] = sign;
            orow[(jo >> 2) * 8 + 4 + (jo & 3)] = zero;
        } else {
            out[(size_t)kn * Kp_out + jo] = sign;
        }
    }
}

// A block makes a unit: a band of output rows (and a segment of output columns) of one image.
//   1. The input values its windows cover are quantised once, into two bit rows per input row in shared memory (sign,
//      non-zero): bit (x - x0)*C + c.  Positions outside the input are the reference's padding, zero whatever the threshold.
//      A warp makes a word with one load per lane and two ballots (COLUMNS false), or, NCHW from twelve channels on, a lane
//      reads all channels of one column and the lanes put their bits together by shuffles (true): with a lane per bit a load
//      touches C rows of the input, 12 or more sectors, and each sector again for the next words -- from L2 where the GEMM
//      in front or behind leaves little L1 (layer call, us, per bit / per column: 32 x 16x75x111 -> 64 7x7 s2 78 / 43,
//      32 x 12x75x111 -> 25 3x3 s2 42 / 22; below twelve channels most of its eight or sixteen loads would be repeats:
//      4 x 4x224x224 7x7 s2 25 / 47).
//   2. In that order the KW*C positions of a window's filter row are CONSECUTIVE bits, starting at ow*SW*C: a thread
//      collects positions of its output pixel with one funnel shift per filter row (and 32 positions) and plane, and stores
//      16 bytes of operands for every 32 of them; positions past K are zero.  Where the unit has few pixels, several warps
//      share them, each with its own sectors of the rows.
// Bound by instructions and by the latencies of one unit, so both steps keep their loops free of divisions and every lane
// on the same path, and units are single blocks, scheduled as SMs come free (a resident grid that walks them ran a
// nearly empty second wave wherever their number was a little above it: 24 x 3x224x224 -> 64 7x7 s2 51 us per layer call,
// 43 so).  Six of them fit an SM, five with a column's sixteen values in registers (40 and 48 registers, no spills).  Layer
// call, one load per position of every window / now: 8 x 3x224x224 -> 64 7x7 s2 31 / 24, 32 x 15x75x111 -> 96 7x7 s2 62 / 45.
constexpr int DQ_THREADS = 256;
constexpr int DQ_SMEM = 48 * 1024;
constexpr int DQ_ROWS = 8;      // loads in flight per lane (one bit per lane)
constexpr int DQ_COLUMN_C = 12; // channels from which on a lane reads a column

struct DenseQ {
    int N, C, H, W, OH, OW, KH, KW, SH, SW, PH, PW;
    int R, groups32;                 // positions of one filter row; 32-position pieces of an image row
    int band, seg, rows, words;      // output rows and columns of a unit; input rows and words per bit row it holds
    int nbands, nsegs;
    FastDiv div_c, div_seg, div_r, div_nsegs, div_nbands;
};

__device__ __forceinline__ void store_sector(uint4* dst, const uint32_t (&lo)[4], const uint32_t (&hi)[4]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(hi[0]),
                 "r"(hi[1]), "r"(hi[2]), "r"(hi[3])
                 : "memory");
}

template <bool NHWC, bool COLUMNS>
__global__ void __launch_bounds__(DQ_THREADS, COLUMNS ? 5 : 6)
dense_quantise_kernel(const float* __restrict__ x, const float* __restrict__ thr, uint4* __restrict__ img, DenseQ g) {
    extern __shared__ uint32_t sm_bits[];  // [rows][words] sign, then [rows][words] non-zero; one spare word behind
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the input may be the output of the launch before
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t* sm_s = sm_bits;
    uint32_t* sm_z = sm_bits + g.rows * g.words;
    const long long cstride = NHWC ? 1 : (long long)g.H * g.W, pstride = NHWC ? g.C : 1, rstride = pstride * g.W;
    const uint32_t nb = g.div_nsegs.div(blockIdx.x), n = g.div_nbands.div(nb);
    const int oh0 = (int)(nb - n * g.nbands) * g.band, ow0 = (int)(blockIdx.x - nb * g.nsegs) * g.seg;
    const int boh = min(g.band, g.OH - oh0), bow = min(g.seg, g.OW - ow0);
    const int y0 = oh0 * g.SH - g.PH, x0 = ow0 * g.SW - g.PW;
    const float t = __ldg(thr + n) + 0.0f;  // + 0.0f: a threshold of -0 behaves as +0 in every compare
    const float* src = x + (size_t)n * g.C * g.H * g.W;
    const int nrows = (boh - 1) * g.SH + g.KH;
    // (a position outside the input is NaN here: no compare holds, whatever the threshold)
    if (COLUMNS) {
        const int nchunks = ((bow - 1) * g.SW + g.KW + 31) / 32;
        const int first = (int)g.div_c.div((uint32_t)lane * 32), at0 = first * g.C - 32 * lane;  // column of word `lane`'s first bit, and where that column's bits start
        const uint32_t keep = (1u << g.C) - 1u;
        for (int k = warp; k < nrows * nchunks; k += DQ_THREADS / 32) {
            const int r = k / nchunks, ch = k - r * nchunks;
            const int ix = x0 + 32 * ch + lane, iy = y0 + r;
            const bool in = (unsigned)ix < (unsigned)g.W && (unsigned)iy < (unsigned)g.H;
            const float* p = src + (iy * rstride + ix);
            float v[16];
#pragma unroll
            for (int c = 0; c < 16; c++) v[c] = in ? __ldg(p + min(c, g.C - 1) * cstride) : NAN;  // past C (at most 16): the last one again, masked off
            uint32_t bits = 0;  // sign plane in the low half, non-zero in the high one
#pragma unroll
            for (int c = 0; c < 16; c++) bits |= (v[c] < -t ? 1u << c : 0u) | (fabsf(v[c]) > t ? 0x10000u << c : 0u);
            bits &= keep * 0x10001u;
            uint32_t ws = 0, wz = 0;
            int px = first, at = at0;
            for (int j = 0; j < 31 / g.C + 2; j++, px++, at += g.C) {  // a word holds bits of at most that many columns
                const uint32_t b = __shfl_sync(0xFFFFFFFFu, bits, px & 31);
                if (px < 32 && at < 32) {
                    ws |= at >= 0 ? (b & 0xFFFFu) << at : (b & 0xFFFFu) >> -at;
                    wz |= at >= 0 ? (b >> 16) << at : (b >> 16) >> -at;
                }
            }
            const int w = ch * g.C + lane;
            if (lane < g.C && w < g.words) {
                sm_s[r * g.words + w] = ws;
                sm_z[r * g.words + w] = wz;
            }
        }
    } else {
        const int nchunks = (nrows + DQ_ROWS - 1) / DQ_ROWS;
        for (int k = warp; k < g.words * nchunks; k += DQ_THREADS / 32) {
            // one word of up to DQ_ROWS rows: the lane's column and channel are worked out once for all of them
            const int w = k / nchunks, r0 = (k - w * nchunks) * DQ_ROWS;
            const uint32_t idx = (uint32_t)w * 32 + lane, xx = g.div_c.div(idx), c = idx - xx * g.C;
            const int ix = x0 + (int)xx, iy = y0 + r0;
            const bool col = (unsigned)ix < (unsigned)g.W;
            const float* p = src + (c * cstride + ix * (long long)pstride + iy * rstride);
            float v[DQ_ROWS];
#pragma unroll
            for (int r = 0; r < DQ_ROWS; r++) v[r] = (col && r0 + r < nrows && (unsigned)(iy + r) < (unsigned)g.H) ? __ldg(p + r * rstride) : NAN;
#pragma unroll
            for (int r = 0; r < DQ_ROWS; r++) {
                const uint32_t sgn = __ballot_sync(0xFFFFFFFFu, v[r] < -t), nz = __ballot_sync(0xFFFFFFFFu, fabsf(v[r]) > t);
                if (lane == 0 && r0 + r < nrows) {
                    sm_s[(r0 + r) * g.words + w] = sgn;
                    sm_z[(r0 + r) * g.words + w] = nz;
                }
            }
        }
    }
    __syncthreads();
    // a warp takes 32 pixels, or one of 2^parts_log2 parts of theirs: whole sectors of a row, an even number of pieces
    const int pixels = boh * bow, groups = (pixels + 31) / 32;
    int parts_log2 = 0;
    while (g.groups32 % (4 << parts_log2) == 0 && (groups << (parts_log2 + 1)) <= DQ_THREADS / 32) parts_log2++;
    const int pieces = g.groups32 >> parts_log2;
    for (int i = warp; i < groups << parts_log2; i += DQ_THREADS / 32) {
        const int grp0 = i >> parts_log2, first = (i - (grp0 << parts_log2)) * pieces, px = grp0 * 32 + lane;
        if (px >= pixels) continue;
        const int ohl = bow == g.seg ? (int)g.div_seg.div((uint32_t)px) : px / bow, owl = px - ohl * bow;
        int kh = (int)g.div_r.div((uint32_t)first * 32), off = first * 32 - kh * g.R;  // where the thread's first position lies
        const uint32_t* row_s = sm_s + (ohl * g.SH + kh) * g.words;
        const uint32_t* row_z = sm_z + (ohl * g.SH + kh) * g.words;
        uint4* dst = img + (((size_t)n * g.OH + oh0 + ohl) * g.OW + ow0 + owl) * g.groups32 + first;
        const uint32_t bit0 = (uint32_t)(owl * g.SW * g.C);
        uint64_t as = 0, az = 0;  // collected positions that are not stored yet; always fewer than 32 between two filter rows' pieces
        int have = 0, grp = 0;
        uint32_t s0 = 0, z0 = 0;  // an even piece waits for its neighbour: the two are stored as one 32-byte sector
        auto emit = [&]() {
            if (grp & 1) {
                uint32_t lo[4], hi[4];
                tnns_expand32_f4(s0, ~z0, lo);
                tnns_expand32_f4((uint32_t)as, ~(uint32_t)az, hi);
                store_sector(dst + grp - 1, lo, hi);
            } else {
                s0 = (uint32_t)as;
                z0 = (uint32_t)az;
            }
            grp++;
            as >>= 32;
            az >>= 32;
            have -= 32;
        };
        for (; kh < g.KH && grp < pieces; kh++, row_s += g.words, row_z += g.words, off = 0)
            for (; off < g.R && grp < pieces; off += 32) {
                const int take = min(g.R - off, 32);
                const uint32_t bit = bit0 + off, w = bit >> 5, keep = 0xFFFFFFFFu >> (32 - take);
                as |= (uint64_t)(__funnelshift_r(row_s[w], row_s[w + 1], bit & 31) & keep) << have;
                az |= (uint64_t)(__funnelshift_r(row_z[w], row_z[w + 1], bit & 31) & keep) << have;
                if ((have += take) >= 32) emit();
            }
        // what is left of the last piece, then zeros for positions past K (written even where they meet zero weights: the
        // GEMM reads whole rows, and sectors nobody wrote would come from HBM)
        while (grp < pieces) emit();
    }
}

}  // namespace

// K' of the virtual layer: the real positions rounded up to a pixel size the copy-engine fed GEMM takes
int tnns_dense_channels(int C, int KH, int KW) {
    const long long K = (long long)C * KH * KW;
    if (K <= 64) return 64;
    if (K <= 128) return 128;
    return (int)(((K + 255) / 256) * 256);
}

// Taken for ternary activations where at most a quarter of the padded row is real and the dense row stays short.
bool tnns_dense_eligible(int type, int C, int KH, int KW) {
    if (!(type == TNN || type == TBN) || C <= 0 || C > 16 || KH <= 0 || KW <= 0) return false;
    const long long K = (long long)C * KH * KW;
    return K <= 1024 && (long long)tnns_dense_channels(C, KH, KW) * 2 <= 64LL * KH * KW;
}

// Packed kernel of the virtual layer (device memory, the reference's layout for `w->type`, Kp_out plane words per row).
int tnns_launch_repack_weights_dense(tnns_cuda_ctx* ctx, const tnns_cuda_weights* w, uint64_t* d_out, int Kp_out) {
    (void)ctx;
    const bool two = (w->type == TNN || w->type == BTN);
    const long long total = (long long)w->KN * Kp_out;
    const int blocks = (int)std::min<long long>((total + 127) / 128, 4096);
    repack_weights_dense_kernel<<<blocks, 128>>>(w->d_packed, d_out, w->KN, w->Kp, w->Cp, w->C, w->KH * w->KW, two ? 1 : 0, Kp_out);
    tnns_count_launch();
    TNNS_CUDA_TRY(cudaGetLastError());
    return TNNS_OK;
}

int tnns_launch_dense_quantise(tnns_cuda_ctx* ctx, const float* d_x, const float* d_thr, void* d_img, const TnnsGeom& g, int Kd, int layout,
                               cudaStream_t stream) {
    const long long rows = (long long)g.N * g.OH * g.OW;
    if (rows == 0) return TNNS_OK;
    if (rows >= 0x7FFFFFFFLL || rows * (Kd / 32) >= 0xFFFFFFFFLL) return tnns_fail(TNNS_ERR_UNSUPPORTED, "too many output pixels for the dense first-layer form");
    DenseQ q;
    q.N = g.N; q.C = g.C; q.H = g.H; q.W = g.W; q.OH = g.OH; q.OW = g.OW; q.KH = g.KH; q.KW = g.KW; q.SH = g.SH; q.SW = g.SW; q.PH = g.PH; q.PW = g.PW;
    q.R = g.C * g.KW; q.groups32 = Kd / 32;
    // The unit: up to four output rows and 256 output columns, fewer where the chip would not get five units per SM (with
    // two: 8 x 3x224x224 -> 64 3x3 s2 20.9 us per layer call against 18.0, s1 43.3 against 37.7, 7x7 s2 24.1 against 23.2) and the
    // unit has more than two words for each warp, or where the bit rows would not fit shared memory (one output pixel
    // always does: K <= 1024 positions)
    q.band = std::min(4, g.OH);
    q.seg = std::min(256, g.OW);
    auto smem = [&]() -> size_t {
        q.rows = (q.band - 1) * g.SH + g.KH;
        q.words = (int)((((long long)(q.seg - 1) * g.SW + g.KW) * g.C + 31) / 32);
        return ((size_t)q.rows * q.words * 2 + 1) * sizeof(uint32_t);
    };
    auto units = [&]() -> long long { return (long long)g.N * ((g.OH + q.band - 1) / q.band) * ((g.OW + q.seg - 1) / q.seg); };
    auto split = [&](int& extent, int least) {  // halves one side of the unit while that is wanted
        while (extent > least && units() < 5LL * ctx->sm_count && smem() > 16 * 2 * sizeof(uint32_t)) extent = (extent + 1) / 2;
    };
    while (q.band > 1 && smem() > DQ_SMEM) q.band = (q.band + 1) / 2;
    while (q.seg > 1 && smem() > DQ_SMEM) q.seg = (q.seg + 1) / 2;
    split(q.seg, 64);  // columns first: a row split repeats KH - S rows of every band
    split(q.band, 1);
    split(q.seg, 16);
    const size_t bytes = smem();
    q.nbands = (g.OH + q.band - 1) / q.band;
    q.nsegs = (g.OW + q.seg - 1) / q.seg;
    q.div_c = tnns_fastdiv((uint32_t)g.C);
    q.div_seg = tnns_fastdiv((uint32_t)q.seg);
    q.div_r = tnns_fastdiv((uint32_t)q.R);
    q.div_nsegs = tnns_fastdiv((uint32_t)q.nsegs);
    q.div_nbands = tnns_fastdiv((uint32_t)q.nbands);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)units());  // at most one per output pixel
    cfg.blockDim = dim3(DQ_THREADS);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    uint4* img = reinterpret_cast<uint4*>(d_img);
    if (layout == TNNS_NHWC) TNNS_CUDA_TRY(cudaLaunchKernelEx(&cfg, dense_quantise_kernel<true, false>, d_x, d_thr, img, q));
    else if (g.C >= DQ_COLUMN_C) TNNS_CUDA_TRY(cudaLaunchKernelEx(&cfg, dense_quantise_kernel<false, true>, d_x, d_thr, img, q));
    else TNNS_CUDA_TRY(cudaLaunchKernelEx(&cfg, dense_quantise_kernel<false, false>, d_x, d_thr, img, q));
    tnns_count_launch();
    TNNS_CUDA_TRY(cudaGetLastError());
    return TNNS_OK;
}
