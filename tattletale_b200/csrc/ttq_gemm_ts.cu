// Linear layers of 9 / 17 to a few hundred activation rows: packed weights expanded straight into TENSOR MEMORY.
//
// y[M][N] = x . W^T with tcgen05.mma kind::f16 in the operand form whose M side (A) comes from tensor memory: the 128
// lanes are 128 WEIGHT rows, the N side (B, shared memory) are the activation rows.  A conversion warp reads its 16-row
// packed tile from a private ring of bulk copies, expands it in registers to fp16 and writes it with tcgen05.st in the
// 16x256b shape, whose register order is the fragment order of the packed layout: no shared-memory round trip of
// expanded weights (8 KB written and 8 KB read back per 2.3 KB packed tile), no swizzle arithmetic, and the row scales stay
// in registers for the whole tile.
//
// Work split.  An item is (128 weight rows, one 256-wide super-block, one block of nb <= 256 activation rows); the items of
// the matrix, K fastest, are cut into gridDim.x equal contiguous runs, one per CTA (one CTA per SM), whatever the shape.
// A run that covers a whole output tile writes it; otherwise the CTA parks its fp32 partial sums in its own workspace slot
// and counts the arrival, and the CTA that arrives last adds the slots in run order (deterministic) with all its threads.
//
// Roles (22 warps): 4 epilogue (thread = weight row), 16 conversion (two sets of 8 on alternating items, one 16-row tile
// each), one MMA warp, one warp that brings the activation slices.  Tensor memory: two or three A stages of 128 columns, the
// rest accumulators.  Every wait is bounded; tensor memory is always released.
//
// Bound.  A conversion warp's chain (wait, scale records, four slices of about 350 cycles, hand-over) gives an item about
// 1700 cycles per SM, twice the HBM time of its 18 KB; from about 100 rows the activation slices (nb x 512 bytes per item out
// of L2) and from 192 the tensor cores.  A fixed 9 us per linear go to the launch, the first tiles' latency and the sum of the
// pieces.  Measured (4096 -> 28672 / 14336 -> 4096 / 4096 -> 6144 / 4096 -> 4096, us; the shared-memory GEMM in brackets):
// 17 rows 30.7 / 20.0 / 12.8 / 11.3 (65.3 / 41.8 / 27.0 / 18.9), 64 rows 35.0 / 26.4 / 15.6 / 14.2 (65.6 / 42.9 / 30.0 / 20.0), 137 rows 56.0 / 37.6 / 23.2 / 21.0
// (128 rows: 68.9 / 45.9 / 34.4 / 22.7); Q8_0 and Q6_K, 4096 -> 28672, 12 rows: 31.7 (69.5) and 38.3 (78.2).
//
// Exact form (Q8_0, Q6_K, one block of 16 rows): every weight as its fp16 rounding plus the remainder, two products into the same
// accumulator, activations exact after a power of two per row, weights beyond fp16 brought into it by a power of two
// per weight row (ts_row_power); half an item per A stage.  4096 -> 28672, 5 to 8 rows: Q8_0 45.6
// us, Q6_K 56 (integer decode kernel: 77 and 95); error against 64 bits as the integer kernel's or below.
#include <cmath>

#include "ttq_devutil.cuh"

namespace ttq {

namespace {

constexpr int TS_EPI_WARPS = 4, TS_CONV_WARPS = 16;
constexpr int TS_MMA_WARP = TS_EPI_WARPS + TS_CONV_WARPS, TS_B_WARP = TS_MMA_WARP + 1;
constexpr int TS_WARPS = TS_B_WARP + 1, TS_THREADS = TS_WARPS * 32;
constexpr int TS_ROWS = 128, TS_GROUP_TILES = TS_ROWS / TILE_ROWS;
// What a launch is: one matrix, many (mixture of experts), or one matrix with its weights as exact pairs of fp16 values.
enum TsMode { TS_DENSE, TS_GROUPED, TS_PRECISE };
// bytes of a row's scale record, and of a conversion warp's 16 records (the exact Q6_K form holds every scale as a pair)
__host__ __device__ constexpr int ts_hdr_row(int fmt, int mode) { return mode == TS_PRECISE && fmt == TTQ_FMT_Q6_K ? 144 : 80; }
__host__ __device__ constexpr int ts_hdr_bytes(int fmt, int mode) { return 16 * ts_hdr_row(fmt, mode); }
constexpr int TS_MAX_RING = 4, TS_MAX_BSLOTS = 12;
constexpr int TS_MAX_A = 3;  // A stages in tensor memory
constexpr int TS_BAR_BYTES = (TS_CONV_WARPS * TS_MAX_RING + 2 * TS_MAX_BSLOTS + 2 * TS_MAX_A + 4) * 8 + 32;
constexpr int TS_SMEM_MAX = 227 * 1024;
constexpr int TS_A_COLS = 128, TS_TMEM_COLS = 512;

struct TsParams {
    const uint8_t *tiles;
    int64_t N, NT;
    int SBp;
    const __half *xh;  // activation images, see launch_xh_images
    int M, Mp;         // activation rows; image rows
    int nb;            // rows per block (a multiple of 16, at most 256); one block, grouped: one per row tile
    const void *bias;
    int bias_dt;
    void *y;
    int y_dt;
    int64_t ldy;
    float *ws;           // slot s: [nb][128] fp32, two slots per CTA
    unsigned *counters;  // arrivals per output tile, zero between launches
    int *status;
    int ring, bslots;  // stages of the packed rings, activation slots
    int spb;           // 64-wide slices per activation slot: 4 (a whole item), 2 or 1
    int64_t T;  // items (grouped: per row tile)
    // grouped (mixture-of-experts) mode, group_tiles != nullptr: a block of activation rows is a row tile of the routed row
    // space and belongs to one of many weight matrices of one shape; tables and the number of row tiles are on the device
    const uint8_t *const *group_tiles;
    const int *mt_group, *mt_row0, *n_mt;
    int64_t mt_cap;
    const float *row_scale;  // exact form: the outputs of activation row m are multiplied by row_scale[m]
    const float *top;        // exact form: Weight::top
};

// kind::f16: D = f32, A = B = f16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t ts_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24); }
__device__ __forceinline__ void ts_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void ts_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
// 16 lanes x 32 columns: registers 4 i .. 4 i + 3 of lane (g, t) = columns 8 i + 2 t, + 1 of row g, then of row g + 8
__device__ __forceinline__ void ts_st_16x256b(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ uint32_t ts_h2(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ __half2 ts_as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

// ---- one packed 16-row tile -> fp16 in tensor memory -------------------------------------------------------------
// Lane (g, t), register sl of a chunk: row g + 8 (sl & 1), group u = (t >> 1) + 2 (sl >> 1), weights 4 (t & 1) .. + 3 of an
// 8-wide window.  Every register gives two runs of four fp16 values (K order 0 2 1 3); run `hi` of register sl goes to
// columns 8 (2 (sl >> 1) + hi) + 2 t, + 1 of its row, i.e. to 16-byte slot p = 4 (sl >> 1) + 2 hi + (t >> 1) of the 64-wide
// slice.  launch_xh_images lays the activations out with the same slot -> K mapping.
//   Q4_K  slice n = window n; run hi = sub-block 2 u + hi
//   Q8_0  slice n = window n; run 0 = block u (chunk n), run 1 = block 4 + u (chunk 4 + n)
//   Q6_K  slice 2 s' + n = window n of sets s' (run 0) and s' + 2 (run 1)

// Exact form: where the weights of a matrix leave fp16 (a block's scale goes up to 65504, its weights to 128 times that in Q8_0 and 4096
// times in Q6_K) those of every row are divided by a power of two 2^s that brings the row's largest below 2^15.  To ask costs a launch
// up to 1 us (Q8_0, 4096 -> 28672 at 5 rows 44.5 -> 45.6, Q6_K 56.2 -> 56.2); out of line the rare case would cost nothing here but take the
// registers that let the next linear's activation pass in beside this kernel.
template <int FMT>
__device__ __forceinline__ bool ts_wide(float top) { return top > (FMT == TTQ_FMT_Q8_0 ? 65504.f / 128 : 65504.f / 32); }  // `top` of Q6_K has the sub-block scale in it
// 2^s of row n (sign 1), 2^-s (sign -1).
template <int FMT>
__device__ __forceinline__ float ts_row_power(const float *top, int64_t n, int sign) {
    const float row = __ldcg(top + 1 + n);
    const int s = ((__float_as_int(row) >> 23) & 255) - 127 + (FMT == TTQ_FMT_Q8_0 ? 7 : 5) - 14;
    return ts_wide<FMT>(row) ? __int_as_float((127 + sign * s) << 23) : 1.f;
}

// Writes the scale records of the tile's 16 rows (lane (r, h): half h of row r).  `shrink` (exact form): 2^-s, see ts_row_power.
template <int FMT, int MODE>
__device__ __forceinline__ void ts_header(uint32_t stage, uint32_t hdr, int lane, float shrink) {
    constexpr int TS_HDR_ROW = ts_hdr_row(FMT, MODE);
    const int r = lane & 15, h = lane >> 4;
    if constexpr (FMT == TTQ_FMT_Q4_K) {
        // sub-blocks 4h..4h+3: {scale, scale, offset, offset} halves, w = scale * (q - 8) + offset (high nibbles arrive as
        // 16 * (q - 8))
        const uint4 hv = lds128<2048>(stage + (uint32_t)r * 16);
        const __half2 dd = ts_as_h2(hv.x);
        const float d = __low2float(dd), dmin = __high2float(dd);
        uint32_t scw, mw;
        q4k_scale_words(hv, h, scw, mw);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float sc = d * (float)((scw >> (8 * i)) & 0xff);
            const float off = fmaf(8.f, sc, -dmin * (float)((mw >> (8 * i)) & 0xff));
            w[2 * i] = ts_h2(__float2half2_rn((i & 1) ? sc * 0.0625f : sc));
            w[2 * i + 1] = ts_h2(__float2half2_rn(off));
        }
        const uint32_t dst = hdr + (uint32_t)(r * TS_HDR_ROW + h * 32);
        sts128<0>(dst, w[0], w[1], w[2], w[3]);
        sts128<16>(dst, w[4], w[5], w[6], w[7]);
    } else if constexpr (FMT == TTQ_FMT_Q8_0) {
        const uint2 hv = lds64<4096>(stage + (uint32_t)(r * 16 + h * 8));
        uint32_t w[4] = {__byte_perm(hv.x, 0, 0x1010), __byte_perm(hv.x, 0, 0x3232), __byte_perm(hv.y, 0, 0x1010), __byte_perm(hv.y, 0, 0x3232)};
        if (MODE == TS_PRECISE && shrink != 1.f) {
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = ts_h2(__hmul2(ts_as_h2(w[i]), __float2half2_rn(shrink)));
        }
        sts128<0>(hdr + (uint32_t)(r * TS_HDR_ROW + h * 16), w[0], w[1], w[2], w[3]);
    } else {
        // 16-wide sub-blocks 8h..8h+7: d * sc as fp16, duplicated into both halves
        const uint2 hv = lds64<3072>(stage + (uint32_t)(r * 16 + h * 8));
        uint16_t dbits;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(dbits) : "r"(stage + 3328u + (uint32_t)r * 2));
        const float d = __half2float(__ushort_as_half(dbits)) * (MODE == TS_PRECISE ? shrink : 1.f);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float sc = d * (float)(int)(int8_t)(((i < 4 ? hv.x : hv.y) >> (8 * (i & 3))) & 0xff);
            w[i] = ts_h2(__float2half2_rn(sc));
        }
        const uint32_t dst = hdr + (uint32_t)(r * TS_HDR_ROW + h * 32);
        sts128<0>(dst, w[0], w[1], w[2], w[3]);
        sts128<16>(dst, w[4], w[5], w[6], w[7]);
        if constexpr (MODE == TS_PRECISE) {
            // what the rounding left out: d * sc has at most 19 significant bits
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float sc = d * (float)(int)(int8_t)(((i < 4 ? hv.x : hv.y) >> (8 * (i & 3))) & 0xff);
                w[i] = ts_h2(__float2half2_rn(sc - __low2float(ts_as_h2(w[i]))));
            }
            sts128<64>(dst, w[0], w[1], w[2], w[3]);
            sts128<80>(dst, w[4], w[5], w[6], w[7]);
        }
    }
}

// PRECISE: two slices from slice n0 on, the rounded weights in columns 0..63 and what the rounding left out in columns 64..127
// of the stage (w = q * scale: one fused multiply-add gives the remainder exactly); otherwise the four slices of the item.
template <int FMT, int MODE>
__device__ __forceinline__ void ts_expand(uint32_t stage, uint32_t hdr, int lane, uint32_t taddr, int n0) {
    constexpr int TS_HDR_ROW = ts_hdr_row(FMT, MODE), SLICES = MODE == TS_PRECISE ? 2 : 4;
    static_assert(MODE != TS_PRECISE || FMT != TTQ_FMT_Q4_K, "the exact form serves formats without an offset");
    // (the four slices are a loop, not unrolled: a quarter of the code to fetch at the start of every launch, and few enough
    // registers that the activation pass of the next linear can be resident beside this kernel)
    const int g = lane >> 2, t = lane & 3;
    const uint32_t sa = stage + (uint32_t)lane * 16;
    uint32_t mask_lo = 0x000f000fu, mask_hi = 0x00f000f0u, mask_b = 0x00ff00ffu, k1024 = 0x64006400u;
    asm volatile("" : "+r"(mask_lo), "+r"(mask_hi), "+r"(mask_b), "+r"(k1024));
    if constexpr (FMT == TTQ_FMT_Q4_K) {
        const __half2 k1032 = __float2half2_rn(1032.f), k1152 = __float2half2_rn(1152.f);
        uint4 so[4];  // register sl: {scale, offset} of sub-blocks 2u (low nibbles) and 2u + 1 (high nibbles)
        const uint32_t ha = hdr + (uint32_t)(g * TS_HDR_ROW + (t >> 1) * 16);
        so[0] = lds128<0>(ha);
        so[1] = lds128<8 * TS_HDR_ROW>(ha);
        so[2] = lds128<32>(ha);
        so[3] = lds128<8 * TS_HDR_ROW + 32>(ha);
#pragma unroll 1
        for (int n = 0; n < 4; n++) {
            const uint4 qa = lds128<0>(sa + n * 512);
            const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w};
            uint32_t r[16];
#pragma unroll
            for (int sl = 0; sl < 4; sl++) {
                const int o = 8 * (sl >> 1) + 2 * (sl & 1);
                const uint32_t x = wa[sl], x8 = x >> 8;
                const __half2 sl_ = ts_as_h2(so[sl].x), ol = ts_as_h2(so[sl].y), sh = ts_as_h2(so[sl].z), oh = ts_as_h2(so[sl].w);
                r[o + 0] = ts_h2(__hfma2(__hsub2(ts_as_h2(and_or(x, mask_lo, k1024)), k1032), sl_, ol));
                r[o + 1] = ts_h2(__hfma2(__hsub2(ts_as_h2(and_or(x8, mask_lo, k1024)), k1032), sl_, ol));
                r[o + 4] = ts_h2(__hfma2(__hsub2(ts_as_h2(and_or(x, mask_hi, k1024)), k1152), sh, oh));
                r[o + 5] = ts_h2(__hfma2(__hsub2(ts_as_h2(and_or(x8, mask_hi, k1024)), k1152), sh, oh));
            }
            ts_st_16x256b(taddr + n * 32, r);
        }
    } else if constexpr (FMT == TTQ_FMT_Q8_0) {
        const __half2 k1152 = __float2half2_rn(1152.f);
        uint32_t s0[4], s1[4];  // scales of blocks u and 4 + u per register
        const uint32_t ha = hdr + (uint32_t)(g * TS_HDR_ROW + (t >> 1) * 4);
        s0[0] = lds32<0>(ha);
        s0[1] = lds32<8 * TS_HDR_ROW>(ha);
        s0[2] = lds32<8>(ha);
        s0[3] = lds32<8 * TS_HDR_ROW + 8>(ha);
        s1[0] = lds32<16>(ha);
        s1[1] = lds32<8 * TS_HDR_ROW + 16>(ha);
        s1[2] = lds32<24>(ha);
        s1[3] = lds32<8 * TS_HDR_ROW + 24>(ha);
#pragma unroll 1
        for (int z = 0; z < SLICES; z++) {
            const int n = n0 + z;
            const uint4 qa = lds128<0>(sa + n * 512), qb = lds128<2048>(sa + n * 512);
            const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w};
            const uint32_t wb[4] = {qb.x, qb.y, qb.z, qb.w};
            uint32_t r[16], lo[16];
#pragma unroll
            for (int sl = 0; sl < 4; sl++) {
                // int8 -> fp16: flip the sign bit (q + 128 in 0..255), OR into the mantissa of 1024, subtract 1152
                const int o = 8 * (sl >> 1) + 2 * (sl & 1);
                const uint32_t x = wa[sl] ^ 0x80808080u, y = wb[sl] ^ 0x80808080u;
                const uint32_t v[4] = {and_or(x, mask_b, k1024), and_or(x >> 8, mask_b, k1024), and_or(y, mask_b, k1024), and_or(y >> 8, mask_b, k1024)};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int at = o + (e & 1) + 4 * (e >> 1);
                    const __half2 q = __hsub2(ts_as_h2(v[e]), k1152), sc = ts_as_h2(e < 2 ? s0[sl] : s1[sl]);
                    const __half2 w = __hmul2(q, sc);
                    r[at] = ts_h2(w);
                    if constexpr (MODE == TS_PRECISE) lo[at] = ts_h2(__hfma2(q, sc, __hneg2(w)));
                }
            }
            ts_st_16x256b(taddr + z * 32, r);
            if constexpr (MODE == TS_PRECISE) ts_st_16x256b(taddr + 64 + z * 32, lo);
        }
    } else {
        const __half2 k1056 = __float2half2_rn(1056.f);
#pragma unroll 1
        for (int z = 0; z < SLICES; z++) {
            const int n = n0 + z, sp = n >> 1;  // set of the low nibbles; the high nibbles are set sp + 2
            uint32_t s0[4], s1[4], t0[4], t1[4];
            const uint32_t ha = hdr + (uint32_t)(g * TS_HDR_ROW + (t >> 1) * 4 + sp * 16);
            s0[0] = lds32<0>(ha);
            s0[1] = lds32<8 * TS_HDR_ROW>(ha);
            s0[2] = lds32<8>(ha);
            s0[3] = lds32<8 * TS_HDR_ROW + 8>(ha);
            s1[0] = lds32<32>(ha);
            s1[1] = lds32<8 * TS_HDR_ROW + 32>(ha);
            s1[2] = lds32<40>(ha);
            s1[3] = lds32<8 * TS_HDR_ROW + 40>(ha);
            if constexpr (MODE == TS_PRECISE) {
                t0[0] = lds32<64>(ha);
                t0[1] = lds32<8 * TS_HDR_ROW + 64>(ha);
                t0[2] = lds32<72>(ha);
                t0[3] = lds32<8 * TS_HDR_ROW + 72>(ha);
                t1[0] = lds32<96>(ha);
                t1[1] = lds32<8 * TS_HDR_ROW + 96>(ha);
                t1[2] = lds32<104>(ha);
                t1[3] = lds32<8 * TS_HDR_ROW + 104>(ha);
            }
            const uint4 qa = lds128<0>(sa + n * 512), qb = lds128<2048>(sa + (n & 1) * 512);
            const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
            uint32_t r[16], lo[16];
#pragma unroll
            for (int sl = 0; sl < 4; sl++) {
                // 6-bit quant = nibble | (two plane bits << 4); OR-ed into the mantissa of 1024, minus 1024 + 32
                const int o = 8 * (sl >> 1) + 2 * (sl & 1);
                const uint32_t x = wa[sl], x8 = x >> 8;
                const uint32_t pl = wb[sl] >> (2 * sp), ph = wb[sl] >> (2 * sp + 4);
                const uint32_t v[4] = {and_or(x, mask_lo, k1024) | ((pl << 4) & 0x00300030u), and_or(x8, mask_lo, k1024) | ((pl >> 4) & 0x00300030u),
                                       and_or(x >> 4, mask_lo, k1024) | ((ph << 4) & 0x00300030u),
                                       and_or(x8 >> 4, mask_lo, k1024) | ((ph >> 4) & 0x00300030u)};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int at = o + (e & 1) + 4 * (e >> 1);
                    const __half2 q = __hsub2(ts_as_h2(v[e]), k1056), sc = ts_as_h2(e < 2 ? s0[sl] : s1[sl]);
                    const __half2 w = __hmul2(q, sc);
                    r[at] = ts_h2(w);
                    if constexpr (MODE == TS_PRECISE)
                        lo[at] = ts_h2(__hfma2(q, ts_as_h2(e < 2 ? t0[sl] : t1[sl]), __hfma2(q, sc, __hneg2(w))));
                }
            }
            ts_st_16x256b(taddr + z * 32, r);
            if constexpr (MODE == TS_PRECISE) ts_st_16x256b(taddr + 64 + z * 32, lo);
        }
    }
}

// Position of an item: tile = outer * ni + inner, super-block.  Dense: outer = 128 weight rows, ni = 1; grouped: outer = row tile,
// inner = 128 weight rows of its expert.
struct TsCursor {
    int64_t outer;
    int inner, sb;
    __device__ __forceinline__ void init(int64_t item, int SBp, int ni) {
        const int64_t tile = item / SBp;
        sb = (int)(item - tile * SBp);
        outer = tile / ni;
        inner = (int)(tile - outer * ni);
    }
    __device__ __forceinline__ void advance(int by, int SBp, int ni) {
        sb += by;
        while (sb >= SBp) {
            sb -= SBp;
            if (++inner == ni) {
                inner = 0;
                outer++;
            }
        }
    }
};

// (The mode is a template parameter: the tables cost the registers that let the activation pass sit beside the dense form)
template <int FMT, int MODE>
__global__ void __launch_bounds__(TS_THREADS, 1) gemm_ts_kernel(const TsParams p) {
    constexpr int TB = tile_bytes(FMT), TS_HDR_BYTES = ts_hdr_bytes(FMT, MODE);
    extern __shared__ uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const int nb = p.nb, SBp = p.SBp, ring = p.ring, bslots = p.bslots;
    const uint32_t slice_bytes = (uint32_t)nb * 128u;
    const int spb = p.spb;
    const uint32_t b_u32 = base, ring_u32 = b_u32 + bslots * spb * slice_bytes, hdr_u32 = ring_u32 + TS_CONV_WARPS * ring * TB;
    const uint32_t bars = hdr_u32 + TS_CONV_WARPS * TS_HDR_BYTES;
    const uint32_t ring_full = bars, b_full = ring_full + 8 * TS_CONV_WARPS * TS_MAX_RING;
    const uint32_t b_empty = b_full + 8 * TS_MAX_BSLOTS;
    const uint32_t a_full = b_empty + 8 * TS_MAX_BSLOTS, a_empty = a_full + 8 * TS_MAX_A, d_full = a_empty + 8 * TS_MAX_A, d_empty = d_full + 16;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(base_ptr + (d_empty + 16 - base));
    volatile int64_t *last_tile = reinterpret_cast<volatile int64_t *>(base_ptr + (d_empty + 32 - base));  // [2]
    // tensor memory: `na` stages of expanded weights, `nd` accumulator sets behind them
    const int na = nb <= 64 ? 3 : 2, nd = nb <= 128 ? 2 : 1, d_col = na * TS_A_COLS;
    constexpr bool grouped = MODE == TS_GROUPED, precise = MODE == TS_PRECISE;
    int64_t T = p.T;
    if (grouped) {
        grid_dependency_wait();  // the tables are written by preceding kernels
        const int64_t used = *p.n_mt;
        T *= used < p.mt_cap ? used : p.mt_cap;
    }
    int64_t G = gridDim.x;
    if (grouped) {
        if (T < G) G = T;
        if ((int64_t)blockIdx.x >= G) return;  // fewer items than CTAs: the last ones have none
    }
    const int ni = grouped ? (int)((p.N + TS_ROWS - 1) / TS_ROWS) : 1;
    auto group_of = [&](const TsCursor &c) -> int64_t { return grouped ? (int64_t)c.inner : c.outer; };
    // first image row of a block
    auto row0_of = [&](const TsCursor &c) -> int { return grouped ? p.mt_row0[c.outer] : 0; };
    const int rows = grouped ? nb : p.M;  // of a block's rows, those that exist
    const int64_t i0 = (int64_t)blockIdx.x * T / G;
    const int n_items = (int)(((int64_t)blockIdx.x + 1) * T / G - i0);
    const int64_t first_tile = i0 / SBp;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < bslots; i++) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < na; i++) {
            mbar_init(a_full + 8 * i, TS_GROUP_TILES);  // one arrival per conversion warp of the item's set
            mbar_init(a_empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(d_full + 8 * i, 1);
            mbar_init(d_empty + 8 * i, TS_EPI_WARPS);
        }
        last_tile[0] = last_tile[1] = -1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int cw = warp - TS_EPI_WARPS;  // conversion warp: set cw >> 3; its tile = its tensor-memory lanes
    const int set = cw >> 3, tau = 2 * (warp & 3) + ((cw >> 2) & 1);
    const uint32_t my_ring = ring_u32 + (uint32_t)(cw * ring * TB), my_bar = ring_full + (uint32_t)(cw * TS_MAX_RING * 8);
    const int my_count = cw >= 0 && cw < TS_CONV_WARPS && n_items > set ? (n_items - set + 1) / 2 : 0;
    // The ring's state is kept by the whole warp and one elected lane issues: with warp-uniform operands a bulk copy (or an
    // MMA) is one instruction, from a branch on the lane number the compiler makes a loop of about 100 cycles of it.
    TsCursor src = {0, 0, 0};
    const uint8_t *src_ptr = nullptr;  // the next tile (nullptr: rows beyond the matrix)
    int issued = 0, i_stage = 0;
    auto locate = [&]() {
        const int64_t rt = group_of(src) * TS_GROUP_TILES + tau;
        src_ptr = nullptr;
        if (rt < p.NT && (!grouped || src.outer * ni * SBp < T)) src_ptr = (grouped ? p.group_tiles[p.mt_group[src.outer]] : p.tiles) + (rt * SBp + src.sb) * (int64_t)TB;
    };
    auto issue_next = [&]() {
        const uint32_t bar = my_bar + 8 * i_stage;
        if (elect_one()) {
            if (src_ptr != nullptr) {
                mbar_expect_tx(bar, TB);
                bulk_g2s(my_ring + (uint32_t)(i_stage * TB), src_ptr, TB, bar);
            } else {
                mbar_arrive(bar);
            }
        }
        issued++;
        if (++i_stage == ring) i_stage = 0;
        if (src.sb + 2 < SBp) {
            src.sb += 2;
            if (src_ptr != nullptr) src_ptr += 2 * TB;
        } else {
            src.advance(2, SBp, ni);
            locate();
        }
    };
    const float top = precise ? __ldcg(p.top) : 0.f;  // on its way beside the first packed tiles, first looked at with them
    if (my_count > 0) {
        // the packed weights depend on no preceding kernel: the ring fills while that one drains
        if (elect_one()) {
            for (int s = 0; s < ring; s++) mbar_init(my_bar + 8 * s, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            fence_async_shared();
        }
        __syncwarp();
        src.init(i0, SBp, ni);
        src.advance(set, SBp, ni);
        locate();
        for (int s = 0; s < ring && s < my_count; s++) issue_next();
    }
    if (warp == TS_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_slot)),
                     "r"((uint32_t)TS_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < TS_EPI_WARPS) {
        // ---------------------------------------------------------------- epilogue: thread = weight row of the group
        grid_dependency_wait();  // outputs, workspace and counters may still be in use by the preceding kernel
        bool alive = true;
        TsCursor c;
        c.init(i0, SBp, ni);
        int left = n_items, seg = 0;
        const int r = warp * 32 + lane;
        while (left > 0) {
            const int run = SBp - c.sb < left ? SBp - c.sb : left;  // items of this CTA inside the tile
            const bool whole = run == SBp;
            const int buf = seg % nd, use = seg / nd;
            const int64_t tile = c.outer * ni + c.inner;
            const int row0 = row0_of(c);
            unsigned others = 0;  // CTAs besides this one that hold a piece of the tile
            if (!whole && threadIdx.x == 0) others = (unsigned)(((tile + 1) * SBp * G - 1) / T - ((tile * SBp + 1) * G - 1) / T);
            if (alive) alive = tc_wait_warp(d_full + 8 * buf, (uint32_t)(use & 1), p.status, lane);
            tc_fence_after();
            const int64_t n = group_of(c) * TS_ROWS + r;
            const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(d_col + buf * nb);
            const int slot = 2 * (int)blockIdx.x + (tile == first_tile ? 0 : 1);
            float *wsp = p.ws + (size_t)slot * nb * TS_ROWS + r;
            const float grow = precise && n < p.N && ts_wide<FMT>(top) ? ts_row_power<FMT>(p.top, n, 1) : 1.f;
            const float bias = whole && p.bias != nullptr && n < p.N ? load_as_float(p.bias, p.bias_dt, n) : 0.f;
#pragma unroll 1
            for (int c0 = 0; c0 < rows; c0 += 16) {
                uint32_t v[16];
                ts_ld16(taddr + c0, v);
                if (whole) {
                    if (n < p.N) {
                        const int64_t at = (int64_t)(row0 + c0) * p.ldy + n;
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c0 + i < rows) store_from_float(p.y, p.y_dt, at + i * p.ldy, (precise ? __uint_as_float(v[i]) * p.row_scale[c0 + i] * grow : __uint_as_float(v[i])) + bias);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c0 + i < rows) __stcg(wsp + (c0 + i) * TS_ROWS, __uint_as_float(v[i]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty + 8 * buf);
            if (!whole) {
                named_barrier(1, TS_EPI_WARPS * 32);
                if (threadIdx.x == 0) {
                    __threadfence();  // (cumulative: covers the stores of the 128 threads behind the barrier)
                    const unsigned old = atomicAdd(p.counters + tile, 1u);
                    if (old == others) {
                        p.counters[tile] = 0u;  // ready for the next launch
                        __threadfence();
                        last_tile[tile == first_tile ? 0 : 1] = tile;
                    }
                }
            }
            left -= run;
            seg++;
            c.advance(run, SBp, ni);
        }
    } else if (warp < TS_MMA_WARP) {
        // ---------------------------------------------------------------- expansion into tensor memory
        const uint32_t hdr = hdr_u32 + (uint32_t)(cw * TS_HDR_BYTES);
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32 + ((cw >> 2) & 1) * 16) << 16);
        int as = precise ? 2 * set : set, a_round = 0;  // A stage of the item, how often the stages have been filled before
        TsCursor c;
        c.init(i0, SBp, ni);
        c.advance(set, SBp, ni);
        bool alive = true;
        int s = 0;
        uint32_t rpar = 0;
        for (int k = 0; k < my_count; k++) {
            const uint32_t stage = my_ring + (uint32_t)(s * TB);
            const bool have = group_of(c) * TS_GROUP_TILES + tau < p.NT;
            if (alive) alive = mbar_wait_bounded(my_bar + 8 * s, rpar, p.status);
            alive = __all_sync(0xffffffffu, alive);
            if (have) {
                float shrink = 1.f;
                if (precise && ts_wide<FMT>(top)) shrink = ts_row_power<FMT>(p.top, (group_of(c) * TS_GROUP_TILES + tau) * TILE_ROWS + (lane & 15), -1);
                ts_header<FMT, MODE>(stage, hdr, lane, shrink);
            }
            __syncwarp();  // the records are written
            // (exact form: the item takes two A stages, each two slices as rounded weights and remainders)
#pragma unroll 1
            for (int half = 0; half < (precise ? 2 : 1); half++) {
                if (a_round >= 1 && alive) alive = tc_wait_warp(a_empty + 8 * as, (uint32_t)((a_round - 1) & 1), p.status, lane);
                tc_fence_after();
                if (have) {
                    ts_expand<FMT, MODE>(stage, hdr, lane, taddr + (uint32_t)(as * TS_A_COLS), 2 * half);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
                tc_fence_before();
                __syncwarp();  // also: every lane has read the stage and the records
                if (lane == 0) mbar_arrive(a_full + 8 * as);
                // the next stage of this set: two items on (dense); the item's second stage, then past the other set's two (exact)
                as += precise ? (half == 0 ? 1 : 3) : 2;
                while (as >= na) {
                    as -= na;
                    a_round++;
                }
            }
            if (alive && issued < my_count) issue_next();
            c.advance(2, SBp, ni);
            if (++s == ring) {
                s = 0;
                rpar ^= 1u;
            }
        }
    } else if (warp == TS_MMA_WARP) {
        // ---------------------------------------------------------------- MMA issue (the whole warp walks the items, one
        // elected lane issues: uniform operands, no per-instruction register moves)
        bool alive = true;
        const uint32_t idesc = ts_idesc(nb);
        int sb = (int)(i0 - first_tile * SBp), seg = 0, slot = 0, as = 0;
        uint32_t bpar = 0, apar = 0;
        bool fresh = true;  // the next product starts an accumulator
        const int step = precise ? 2 : spb;  // slices per hand-over (exact form: a whole item per activation slot, two A stages)
        for (int li = 0; li < n_items; li++) {
            const int buf = seg % nd, use = seg / nd;
            if (fresh && use >= 1 && alive) alive = tc_wait(d_empty + 8 * buf, (uint32_t)((use - 1) & 1), p.status);
            const uint32_t td = tmem_base + (uint32_t)(d_col + buf * nb);
            const bool done = sb + 1 == SBp || li == n_items - 1;
#pragma unroll 1
            for (int n = 0; n < 4; n += step) {
                if ((precise || n == 0) && alive) alive = tc_wait(a_full + 8 * as, apar, p.status);
                if ((!precise || n == 0) && alive) alive = tc_wait(b_full + 8 * slot, bpar, p.status);
                __syncwarp();
                tc_fence_after();
                if (elect_one()) {
                    uint64_t bd = smem_desc_sw128(b_u32 + (uint32_t)(slot * spb) * slice_bytes + (precise ? (uint32_t)n * slice_bytes : 0u));
                    uint32_t ta = tmem_base + (uint32_t)(as * TS_A_COLS + (precise ? 0 : n * 32));
                    for (int q = 0; q < step; q++) {
                        ts_mma(td, ta, bd, idesc, (fresh && n + q == 0) ? 0u : 1u);
#pragma unroll
                        for (int kk = 1; kk < 4; kk++) ts_mma(td, ta + 8 * kk, bd + (uint64_t)(2 * kk), idesc, 1u);
                        if (precise) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) ts_mma(td, ta + 64 + 8 * kk, bd + (uint64_t)(2 * kk), idesc, 1u);
                        }
                        ta += 32;
                        bd += (uint64_t)(slice_bytes >> 4);
                    }
                    if (!precise || n + step == 4) umma_commit(b_empty + 8 * slot);
                    if (precise || n + step == 4) umma_commit(a_empty + 8 * as);
                    if (n + step == 4 && done) umma_commit(d_full + 8 * buf);
                }
                __syncwarp();
                if ((!precise || n + step == 4) && ++slot == bslots) {
                    slot = 0;
                    bpar ^= 1u;
                }
                if ((precise || n + step == 4) && ++as == na) {
                    as = 0;
                    apar ^= 1u;
                }
            }
            fresh = done;
            if (done) {
                sb = 0;
                seg++;
            } else {
                sb++;
            }
        }
    } else {
        // ---------------------------------------------------------------- activation slices
        grid_dependency_wait();  // the images are written by the preceding kernel
        bool alive = true;
        TsCursor c;
        c.init(i0, SBp, ni);
        const int64_t it_stride = ((int64_t)p.Mp >> 3) << 10;
        const uint8_t *img = reinterpret_cast<const uint8_t *>(p.xh);
        int slot = 0, filled = 0;
        uint32_t par = 1;
        for (int li = 0; li < n_items; li++) {
            const uint8_t *from = img + (int64_t)c.sb * 4 * it_stride + (((int64_t)row0_of(c) >> 3) << 10);
            for (int n = 0; n < 4; n += spb, filled++) {
                if (filled >= bslots && alive) alive = __all_sync(0xffffffffu, tc_wait(b_empty + 8 * slot, par, p.status));
                const uint32_t dst = b_u32 + (uint32_t)(slot * spb) * slice_bytes, bar = b_full + 8 * slot;
                if (alive && elect_one()) {
                    mbar_expect_tx(bar, spb * slice_bytes);
                    if (!grouped) {
                        bulk_g2s(dst, from + n * it_stride, spb * slice_bytes, bar);  // the slices of one block are neighbours
                    } else {
                        for (int q = 0; q < spb; q++) bulk_g2s(dst + q * slice_bytes, from + (n + q) * it_stride, slice_bytes, bar);
                    }
                }
                if (++slot == bslots) {
                    slot = 0;
                    par ^= 1u;
                }
            }
            c.advance(1, SBp, ni);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TS_MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TS_TMEM_COLS) : "memory");
    }
    // ---- the tiles whose last piece came from this CTA: all threads add the pieces, four outputs each, in run order
#pragma unroll 1
    for (int which = 0; which < 2; which++) {
        const int64_t tile = last_tile[which];
        if (tile < 0) continue;
        const int64_t c_first = ((tile * SBp + 1) * G - 1) / T;
        const int pieces = (int)(((tile + 1) * SBp * G - 1) / T - c_first) + 1;
        TsCursor c;
        c.init(tile * SBp, SBp, ni);
        const int64_t group = group_of(c);
        const int row0 = row0_of(c);
        const size_t piece = (size_t)nb * TS_ROWS;
        // the first CTA of the tile parked its piece in its second slot, unless its own run starts inside the tile; every
        // other one in its first slot
        const float *w0 = p.ws + (size_t)(2 * c_first + (c_first * T / G / SBp == tile ? 0 : 1)) * piece;
        const float *w1 = p.ws + (size_t)(2 * (c_first + 1)) * piece;
        for (int idx = threadIdx.x; idx < rows * (TS_ROWS / 4); idx += TS_THREADS) {
            const int m = idx >> 5, v4 = (idx & 31) * 4;
            const size_t at = (size_t)m * TS_ROWS + v4;
            float4 acc = __ldcg(reinterpret_cast<const float4 *>(w0 + at));
            for (int c0 = 1; c0 < pieces; c0 += 6) {
                float4 q[6];  // six pieces requested at once
#pragma unroll
                for (int z = 0; z < 6; z++) {
                    q[z] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (c0 + z < pieces) q[z] = __ldcg(reinterpret_cast<const float4 *>(w1 + (size_t)(2 * (c0 + z - 1)) * piece + at));
                }
#pragma unroll
                for (int z = 0; z < 6; z++) {
                    acc.x += q[z].x;
                    acc.y += q[z].y;
                    acc.z += q[z].z;
                    acc.w += q[z].w;
                }
            }
            const int64_t n = group * TS_ROWS + v4;
            float o[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (precise) o[i] *= p.row_scale[m];
                if (precise && n + i < p.N && ts_wide<FMT>(top)) o[i] *= ts_row_power<FMT>(p.top, n + i, 1);
                if (p.bias != nullptr && n + i < p.N) o[i] += load_as_float(p.bias, p.bias_dt, n + i);
            }
            // four outputs in one store where they lie so (y may be host memory, where every store is a transfer of its own)
            const int64_t yi = (int64_t)(row0 + m) * p.ldy + n;
            uint8_t *yp = reinterpret_cast<uint8_t *>(p.y) + yi * (p.y_dt == TTQ_DT_F32 ? 4 : 2);
            const bool whole4 = n + 4 <= p.N;
            if (whole4 && p.y_dt == TTQ_DT_F32 && (reinterpret_cast<uintptr_t>(yp) & 15) == 0) {
                *reinterpret_cast<float4 *>(yp) = make_float4(o[0], o[1], o[2], o[3]);
            } else if (whole4 && p.y_dt != TTQ_DT_F32 && (reinterpret_cast<uintptr_t>(yp) & 7) == 0) {
                uint32_t w[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    if (p.y_dt == TTQ_DT_BF16) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
                        w[i] = *reinterpret_cast<const uint32_t *>(&h);
                    } else {
                        w[i] = ts_h2(__floats2half2_rn(o[2 * i], o[2 * i + 1]));
                    }
                }
                *reinterpret_cast<uint2 *>(yp) = make_uint2(w[0], w[1]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (n + i < p.N) store_from_float(p.y, p.y_dt, yi + i, o[i]);
            }
        }
    }
}

// CTAs of a dense launch.  One per SM, unless that cuts a tile into so many pieces that the CTA that adds them up works longer
// than the cut saves: an item takes about 0.9 + 0.0055 nb us, a piece nb / 160 us in that CTA, and a tile of SBp items in c pieces
// SBp / c items and c pieces.
int ts_grid(int64_t T, int64_t tiles, int SBp, int nb, int sms) {
    int64_t g = T < sms ? T : sms;
    const double c = sqrt((double)SBp * (0.9 + 0.0055 * nb) * 160.0 / nb);
    const int64_t most = (int64_t)((double)tiles * (c < 1.0 ? 1.0 : c));
    return (int)(g < most ? g : most);
}

template <int FMT, int MODE = TS_DENSE>
cudaError_t ts_launch(TsParams &p, int grid, cudaStream_t st) {
    constexpr int TB = tile_bytes(FMT), TS_HDR_BYTES = ts_hdr_bytes(FMT, MODE);
    static bool configured[64] = {};  // per device: the shared-memory opt-in belongs to the device's copy of the function
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(gemm_ts_kernel<FMT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    // Three ring stages of packed tiles cover the memory latency of narrow blocks.  From 80 rows the activation slices (latency times
    // rate out of L2) set the pace: two stages do, and the room holds more slices (4096 -> 28672 at 80 rows 44.7 -> 37.7 us, at 137
    // rows 71.3 -> 56.8).  A slot is a whole item while at least three of them fit.
    const int fixed = 1024 + TS_CONV_WARPS * TS_HDR_BYTES + TS_BAR_BYTES, slice = p.nb * 128;
    p.ring = p.nb > 64 ? 2 : 3;
    while (p.ring > 2 && fixed + TS_CONV_WARPS * p.ring * TB + 4 * slice > TS_SMEM_MAX) p.ring--;
    const int room = TS_SMEM_MAX - fixed - TS_CONV_WARPS * p.ring * TB;
    p.spb = room >= 12 * slice ? 4 : (room >= 6 * slice ? 2 : 1);
    p.bslots = room / (slice * p.spb);
    if (p.bslots > TS_MAX_BSLOTS) p.bslots = TS_MAX_BSLOTS;
    if (p.bslots < 2 || (MODE == TS_PRECISE && p.spb != 4)) return cudaErrorNotSupported;
    const size_t smem = (size_t)fixed + (size_t)TS_CONV_WARPS * p.ring * TB + (size_t)p.bslots * p.spb * slice;
    return launch_pdl(gemm_ts_kernel<FMT, MODE>, dim3((unsigned)grid), dim3(TS_THREADS), smem, st, p);
}

}  // namespace

// Activation images + the kernel above.  cudaErrorNotSupported: the caller takes another path (scratch too small).
cudaError_t launch_gemm_ts(int fmt, const LinearArgs &a, __half *xh, int64_t xh_capacity, int sms, int *status, unsigned *counters,
                           int64_t counters_cap, cudaStream_t st, int *launches) {
    *launches = 0;
    if (!gemm_supported(fmt) || a.M < 1 || a.M > 256) return cudaErrorNotSupported;
    TsParams p;
    p.M = (int)a.M;
    p.nb = p.Mp = (p.M + 15) / 16 * 16;
    p.tiles = a.tiles;
    p.N = a.N; p.NT = a.NT; p.SBp = (int)a.SBp;
    const int64_t groups = (a.N + TS_ROWS - 1) / TS_ROWS;
    p.T = groups * a.SBp;
    const int grid = ts_grid(p.T, groups, p.SBp, p.nb, sms);
    const int64_t Kp = a.SBp * TILE_K;
    const size_t xh_bytes = ((size_t)p.Mp * Kp * sizeof(__half) + 255) & ~(size_t)255;
    const size_t ws_bytes = (size_t)2 * grid * p.nb * TS_ROWS * sizeof(float);
    if (xh_bytes + ws_bytes > (size_t)xh_capacity * sizeof(__half) || groups > counters_cap) return cudaErrorNotSupported;
    p.xh = xh;
    p.ws = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(xh) + xh_bytes);
    p.counters = counters;
    p.bias = a.bias; p.bias_dt = a.bias_dt;
    p.y = a.y; p.y_dt = a.y_dt; p.ldy = a.ldy;
    p.status = status;
    p.row_scale = nullptr; p.top = nullptr;
    p.group_tiles = nullptr; p.mt_group = nullptr; p.mt_row0 = nullptr; p.n_mt = nullptr; p.mt_cap = 0;
    cudaError_t e = launch_xh_images(a, p.Mp, Kp, xh, sms, fmt == TTQ_FMT_Q4_K ? 2 : (fmt == TTQ_FMT_Q6_K ? 3 : 4), st);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (fmt == TTQ_FMT_Q4_K) e = ts_launch<TTQ_FMT_Q4_K>(p, grid, st);
    else if (fmt == TTQ_FMT_Q8_0) e = ts_launch<TTQ_FMT_Q8_0>(p, grid, st);
    else e = ts_launch<TTQ_FMT_Q6_K>(p, grid, st);
    if (e == cudaSuccess) ++*launches;
    return e;
}

namespace {

// Rows of the exact form: every row is brought by a power of two to a largest magnitude in [512, 1024), where a bf16 or f16
// value is exact in fp16 down to 2^-24 of 512; `scale[m]` undoes it.  One CTA per image row (rows beyond M: zeros).
__global__ void __launch_bounds__(512) xh_rows_kernel(const void *__restrict__ x, int x_dt, int M, int64_t K, int64_t Kp, int64_t ldx,
                                                      __half *__restrict__ xh, float *__restrict__ scale, int kmap) {
    __shared__ float red[16];
    grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = blockIdx.x;
    const int SBp = (int)(Kp >> 8);
    int s, slot;
    xh_place(kmap, lane, s, slot);
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 2)) & 15) == 0;
    grid_dependency_wait();
    auto load = [&](int sb, float (&v)[8]) {
        const int64_t k0 = (int64_t)sb * 256 + 8 * lane;
        if (m < M && aligned && k0 + 8 <= K) {
            xh_unpack(*reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(x) + m * ldx + k0), x_dt, v);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = m < M && k0 + i < K ? load_as_float(x, x_dt, m * ldx + k0 + i) : 0.f;
        }
    };
    float v[8], amax = 0.f;
    for (int sb = warp; sb < SBp; sb += 16) {
        load(sb, v);
#pragma unroll
        for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) red[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 16; w++) amax = fmaxf(amax, red[w]);
    // (two factors, so that neither leaves the range of a float: |9 - e| is at most 158)
    const int e = amax > 0.f && isfinite(amax) ? 9 - ilogbf(amax) : 0, e1 = e / 2, e2 = e - e1;
    const float f1 = ldexpf(1.f, e1), f2 = ldexpf(1.f, e2);
    if (threadIdx.x == 0) scale[m] = ldexpf(1.f, -e);
    for (int sb = warp; sb < SBp; sb += 16) {
        load(sb, v);
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int a = (q >> 1) * 4 + (q & 1);
            o[q] = ts_h2(__floats2half2_rn(v[a] * f1 * f2, v[a + 2] * f1 * f2));
        }
        const int64_t it = (int64_t)sb * 4 + s;
        const int64_t dst = ((it * (gridDim.x >> 3) + (m >> 3)) << 10) + ((m & 7) << 7) + ((slot ^ (m & 7)) << 4);
        *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(xh) + dst) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

}  // namespace

constexpr int TS_PRECISE_ROWS = 16;
int64_t gemm_ts_precise_halves(int64_t Kp, int sms) {
    return TS_PRECISE_ROWS * Kp + (256 + (int64_t)2 * sms * TS_PRECISE_ROWS * TS_ROWS * (int64_t)sizeof(float)) / (int64_t)sizeof(__half);
}

// Q8_0 / Q6_K, up to 16 rows, with weights and activations exact: the accuracy of the integer decode kernel at the rate of
// the tensor cores.  Not for the gated form, whose products would be rounded to fp16.
cudaError_t launch_gemm_ts_precise(int fmt, const LinearArgs &a, const float *top, __half *xh, int64_t xh_capacity, int sms, int *status, unsigned *counters,
                                   int64_t counters_cap, cudaStream_t st, int *launches) {
    *launches = 0;
    constexpr int NB = TS_PRECISE_ROWS;
    if ((fmt != TTQ_FMT_Q8_0 && fmt != TTQ_FMT_Q6_K) || a.M < 1 || a.M > NB || a.gated) return cudaErrorNotSupported;
    TsParams p;
    p.nb = NB;
    p.M = (int)a.M; p.Mp = NB;
    p.tiles = a.tiles;
    p.N = a.N; p.NT = a.NT; p.SBp = (int)a.SBp;
    const int64_t groups = (a.N + TS_ROWS - 1) / TS_ROWS;
    p.T = groups * a.SBp;
    const int grid = ts_grid(p.T, groups, p.SBp, NB, sms);
    const int64_t Kp = a.SBp * TILE_K;
    const size_t xh_bytes = (size_t)NB * Kp * sizeof(__half), ws_at = xh_bytes + 256;  // 256: the row scales
    if (gemm_ts_precise_halves(Kp, grid) > xh_capacity || groups > counters_cap) return cudaErrorNotSupported;
    float *scale = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(xh) + xh_bytes);
    p.xh = xh;
    p.ws = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(xh) + ws_at);
    p.row_scale = scale;
    p.top = top;
    p.counters = counters;
    p.bias = a.bias; p.bias_dt = a.bias_dt;
    p.y = a.y; p.y_dt = a.y_dt; p.ldy = a.ldy;
    p.status = status;
    p.group_tiles = nullptr; p.mt_group = nullptr; p.mt_row0 = nullptr; p.n_mt = nullptr; p.mt_cap = 0;
    cudaError_t e = launch_pdl(xh_rows_kernel, dim3(NB), dim3(512), 0, st, a.x, a.x_dt, (int)a.M, a.K, Kp, a.ldx, xh, scale, fmt == TTQ_FMT_Q6_K ? 3 : 4);
    if (e != cudaSuccess) return e;
    ++*launches;
    e = fmt == TTQ_FMT_Q8_0 ? ts_launch<TTQ_FMT_Q8_0, TS_PRECISE>(p, grid, st) : ts_launch<TTQ_FMT_Q6_K, TS_PRECISE>(p, grid, st);
    if (e == cudaSuccess) ++*launches;
    return e;
}

// Grouped form (Q4_K): row tile mt of the routed rows multiplies weight matrix mt_group[mt]; `xh` holds the images of the
// routed rows in the slot order of this kernel.
bool gemm_ts_grouped_fits(const GroupedArgs &g, int sms) {
    const int64_t groups = (g.N + TS_ROWS - 1) / TS_ROWS;
    return g.ts_ws != nullptr && g.BM % 16 == 0 && g.BM <= 256 && groups * g.mt_cap <= g.ts_counters_cap &&
           (size_t)2 * sms * g.BM * TS_ROWS * sizeof(float) <= g.ts_ws_bytes;
}

cudaError_t launch_gemm_ts_grouped(const GroupedArgs &g, const __half *xh, int sms, int *status, cudaStream_t st) {
    if (!gemm_ts_grouped_fits(g, sms)) return cudaErrorInvalidValue;
    TsParams p;
    p.nb = g.BM;
    p.M = (int)g.Mp; p.Mp = (int)g.Mp;
    p.tiles = nullptr;
    p.N = g.N; p.NT = g.NT; p.SBp = (int)g.SBp;
    p.T = (g.N + TS_ROWS - 1) / TS_ROWS * g.SBp;
    p.xh = xh;
    p.ws = g.ts_ws;
    p.counters = g.ts_counters;
    p.bias = nullptr; p.bias_dt = TTQ_DT_F32;
    p.y = g.y; p.y_dt = g.y_dt; p.ldy = g.ldy;
    p.status = status;
    p.row_scale = nullptr; p.top = nullptr;
    p.group_tiles = g.group_tiles; p.mt_group = g.mt_group; p.mt_row0 = g.mt_row0; p.n_mt = g.n_mt; p.mt_cap = g.mt_cap;
    return ts_launch<TTQ_FMT_Q4_K, TS_GROUPED>(p, sms, st);
}

}  // namespace ttq
