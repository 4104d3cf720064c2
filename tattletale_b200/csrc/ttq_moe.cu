// Routing and combination kernels of the mixture-of-experts layer built on the grouped Q4_K GEMM.
//
// A layer call routes every (token, choice) pair to a row of a padded, expert-sorted row space:
// expert e owns ceil(count_e / BM) consecutive BM-row tiles, so that each row tile of the grouped GEMM
// multiplies exactly one expert's matrices.  Nothing is copied to the host: tile counts and tables stay
// on the device and the GEMM reads them there.
//
//   route_count   histogram of the expert ids
//   route_plan    prefix over the experts -> first row of each expert, expert of each row tile, tile count
//   route_scatter slot of every pair (atomic cursor per expert), source token of every slot; `ordered` for the tensor-memory
//                 GEMM: slots in the order of the pairs
//   combine       y[t] = sum_j w[t][j] * o[slot(t, j)]   (fixed order over j)
//
// The result does not depend on the order in which the atomics handed out the slots: the shared-memory GEMM adds up every row in
// the same order wherever it lies.  The tensor-memory GEMM cuts each row tile along K at places of its own, so there a row's tile
// has to be the same in every call.
//
// The reference has no mixture-of-experts layer; the dataflow is the gated MLP of
// workspace/transformers/src/layers/mlp.nim:56-60 applied per expert, weighted and summed.
#include "ttq_internal.cuh"

namespace ttq {
namespace {

__global__ void __launch_bounds__(256) route_count_kernel(const int *__restrict__ ids, int64_t pairs, int E, int *__restrict__ counts) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += (int64_t)gridDim.x * blockDim.x) {
        const int e = ids[i];
        if (e >= 0 && e < E) atomicAdd(counts + e, 1);
    }
}

// One block.  Expert counts -> padded row ranges and the row-tile tables.  Fixed tile heights (64, 128, 256): an
// expert's rows are padded to whole tiles.  BM = 384: rows are padded to 128 and a tile holds up to three
// 128-row blocks of ONE expert, so that the expert's weight rows are expanded once for (almost always) all of
// its rows.  `mt_cap` bounds the tables (they cannot overflow when the capacity was sized as the launcher does;
// the check keeps a bad call from writing out of bounds).
__global__ void __launch_bounds__(1024) route_plan_kernel(const int *__restrict__ counts, int E, int BM, int mt_cap,
                                                          int *__restrict__ row_start, int *__restrict__ cursor,
                                                          int *__restrict__ mt_group, int *__restrict__ mt_row0,
                                                          int *__restrict__ mt_mh, int *__restrict__ n_mt) {
    extern __shared__ int plan_s[];  // tile_start [E + 1], row_begin [E + 1]
    int *tile_start = plan_s, *row_begin = plan_s + E + 1;
    const int unit = BM == 384 ? 128 : BM;
    // (the counts go to shared memory first: read one by one from global memory the prefix took 13 us for 128 experts)
    for (int e = threadIdx.x; e < E; e += blockDim.x) tile_start[e] = counts[e];
    __syncthreads();
    if (threadIdx.x == 0) {
        int tiles = 0, rows = 0;
        for (int e = 0; e < E; e++) {
            const int padded = (tile_start[e] + unit - 1) / unit * unit;
            tile_start[e] = tiles;
            row_begin[e] = rows;
            tiles += (padded + BM - 1) / BM;
            rows += padded;
        }
        tile_start[E] = tiles;
        row_begin[E] = rows;
        n_mt[0] = tiles < mt_cap ? tiles : mt_cap;
        n_mt[1] = rows;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        row_start[e] = row_begin[e];
        cursor[e] = 0;
        const int padded = row_begin[e + 1] - row_begin[e];
        for (int t = tile_start[e]; t < tile_start[e + 1] && t < mt_cap; t++) {
            const int off = (t - tile_start[e]) * BM;
            mt_group[t] = e;
            mt_row0[t] = row_begin[e] + off;
            const int left = padded - off;
            mt_mh[t] = BM == 384 ? (left >= 384 ? 3 : left / 128) : (BM > 128 ? BM / 128 : 1);
        }
    }
}

__global__ void __launch_bounds__(256) route_scatter_kernel(const int *__restrict__ ids, int64_t pairs, int top_k, int E, int64_t Mp,
                                                            const int *__restrict__ row_start, int *__restrict__ cursor,
                                                            int *__restrict__ slot_of, int *__restrict__ row_src) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += (int64_t)gridDim.x * blockDim.x) {
        const int e = ids[i];
        int slot = -1;
        if (e >= 0 && e < E) {
            slot = row_start[e] + atomicAdd(cursor + e, 1);
            if (slot < Mp) row_src[slot] = (int)(i / top_k);
            else slot = -1;
        }
        slot_of[i] = slot;
    }
}

// One block per expert: its pairs in ascending order, 1024 of all pairs a step.  (1500 tokens of 8 choices among 128 experts: 12 steps;
// a call with more rows per expert than the tensor-memory GEMM serves keeps the atomics.)
__global__ void __launch_bounds__(256) route_scatter_ordered_kernel(const int *__restrict__ ids, int64_t pairs, int top_k, int E, int64_t Mp,
                                                                    const int *__restrict__ row_start, int *__restrict__ slot_of,
                                                                    int *__restrict__ row_src) {
    __shared__ int warp_count[8];
    const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int base = row_start[e];
    const unsigned n = (unsigned)pairs;  // fewer than 2^30: 32-bit division (12000 pairs of 128 experts 12.7 -> 11.5 us; 3.9 with atomics)
    for (unsigned i0 = 0; i0 < n; i0 += 1024) {
        const unsigned i = i0 + 4 * threadIdx.x;
        int id[4], count = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            id[q] = i + q < n ? ids[i + q] : -1;
            count += id[q] == e ? 1 : 0;
            if (e == 0 && i + q < n && (id[q] < 0 || id[q] >= E)) slot_of[i + q] = -1;
        }
        int upto = count;  // of the warp's threads up to this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        if (lane == 31) warp_count[warp] = upto;
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            before += w < warp ? warp_count[w] : 0;
            total += warp_count[w];
        }
        int slot = base + before + upto - count;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (id[q] != e) continue;
            if (slot < Mp) row_src[slot] = (int)((i + q) / (unsigned)top_k);
            slot_of[i + q] = slot < Mp ? slot : -1;
            slot++;
        }
        base += total;
        __syncthreads();
    }
}

// 8 outputs per thread; o rows are fp16 or bf16 (16-byte aligned rows take the vector path)
__global__ void __launch_bounds__(256) combine_kernel(const void *__restrict__ o, int o_dt, int64_t ldo, const int *__restrict__ slot_of,
                                                      const float *__restrict__ w, int64_t T, int top_k, int64_t H, void *__restrict__ y,
                                                      int y_dt, int64_t ldy) {
    const int64_t per_row = (H + 7) / 8, total = T * per_row;
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = c / per_row, h0 = (c % per_row) * 8;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int j = 0; j < top_k; j++) {
            const int slot = slot_of[t * top_k + j];
            if (slot < 0) continue;
            const float wj = w[t * top_k + j];
            const bool vec = o_dt == TTQ_DT_F16 && h0 + 8 <= H &&
                             ((reinterpret_cast<uintptr_t>(o) + (size_t)((int64_t)slot * ldo + h0) * 2) & 15) == 0;
            if (vec) {
                const uint4 raw = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(o) + (int64_t)slot * ldo + h0);
                const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float2 v = __half22float2(h2[q]);
                    acc[2 * q] = fmaf(wj, v.x, acc[2 * q]);
                    acc[2 * q + 1] = fmaf(wj, v.y, acc[2 * q + 1]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (h0 + i < H) acc[i] = fmaf(wj, load_as_float(o, o_dt, (int64_t)slot * ldo + h0 + i), acc[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (h0 + i < H) store_from_float(y, y_dt, t * ldy + h0 + i, acc[i]);
    }
}

unsigned grid_of(int64_t items, int cap) {
    int64_t b = (items + 255) / 256;
    if (b < 1) b = 1;
    return (unsigned)(b < cap ? b : cap);
}

}  // namespace

cudaError_t launch_moe_route(const MoeRouting &r, const int *topk_ids, int64_t T, int top_k, int E, int BM, int64_t Mp,
                             int64_t mt_cap, bool ordered, cudaStream_t st, int *launches) {
    *launches = 0;
    const int64_t pairs = T * top_k;
    // (the arrival counters in front of the counts too: a call that gave up a wait may have left some behind)
    cudaError_t e = cudaMemsetAsync(r.arrivals, 0, (size_t)(reinterpret_cast<uint8_t *>(r.counts + E) - reinterpret_cast<uint8_t *>(r.arrivals)), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(r.row_src, 0xff, sizeof(int) * (size_t)Mp, st);  // every row is padding until a pair claims it
    if (e != cudaSuccess) return e;
    route_count_kernel<<<grid_of(pairs, device_sms() * 4), 256, 0, st>>>(topk_ids, pairs, E, r.counts);
    route_plan_kernel<<<1, 1024, 2 * sizeof(int) * (size_t)(E + 1), st>>>(r.counts, E, BM, (int)mt_cap, r.row_start, r.cursor, r.mt_group,
                                                                          r.mt_row0, r.mt_mh, r.n_mt);
    if (ordered)
        route_scatter_ordered_kernel<<<E, 256, 0, st>>>(topk_ids, pairs, top_k, E, Mp, r.row_start, r.slot_of, r.row_src);
    else
        route_scatter_kernel<<<grid_of(pairs, device_sms() * 4), 256, 0, st>>>(topk_ids, pairs, top_k, E, Mp, r.row_start, r.cursor, r.slot_of,
                                                                               r.row_src);
    *launches = 3;
    return cudaGetLastError();
}

cudaError_t launch_moe_combine(const MoeRouting &r, const void *o, int o_dt, int64_t ldo, const float *topk_w, int64_t T,
                               int top_k, int64_t H, void *y, int y_dt, int64_t ldy, cudaStream_t st) {
    combine_kernel<<<grid_of(T * ((H + 7) / 8), device_sms() * 16), 256, 0, st>>>(o, o_dt, ldo, r.slot_of, topk_w, T, top_k, H, y, y_dt, ldy);
    return cudaGetLastError();
}

}  // namespace ttq
