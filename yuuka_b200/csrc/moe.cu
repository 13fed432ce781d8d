// qwen35moe feed-forward block on the device (model/qwen35/forward.go:320-458):
// router logits -> top-k experts by repeated argmax (lowest index wins ties) ->
// softmax over the selected logits only -> grouping of the (row, slot) pairs by
// expert -> the combine  x += sum_slot w * expert_out + sigmoid(gate) * shared_out.
// The expert matrices themselves run through the grouped tiled GEMM.
#include <cfloat>

#include "gemm_tiled.cuh"
#include "layers.cuh"

namespace yk {

constexpr int ROUTE_THREADS = 256;
constexpr int ROUTE_MAX_EXPERTS = 1024;

struct RouteParams {
    const float * xn;       // [rows][hidden] normalised activations
    const float * router;   // [experts][hidden] f32
    const float * sh_gate;  // [hidden] f32 (shared-expert gate vector)
    int hidden, experts, used;
    int32_t * ids;          // [rows][used]
    float * weights;        // [rows][used]
    float * shared_gate;    // [rows]
};

constexpr int ROUTE_ROWS = 8;      // rows per CTA: a router row is read once per eight activation rows
constexpr int ROUTE_EXPERTS = 32;  // router rows per CTA: four per warp

// Logits as integers that order like them (0 for NaN, which no round selects), and back
__device__ __forceinline__ uint32_t logit_key(float v) {
    if (v != v) return 0u;
    const uint32_t b = __float_as_uint(v + 0.0f);  // (-0 -> +0: equal values are told apart by index alone)
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float key_logit(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k); }

// grid (row groups, expert groups). A warp takes four router rows and all eight activation rows: 16-byte
// weight loads shared by the rows, 32 accumulators per lane; a dot product is summed by lanes in a fixed
// order (the CPU reference sums sequentially, so logits agree to rounding, not bit for bit), the 32 of a warp at once, each
// exchange halving what a lane holds. Logits go to global memory; the last CTA of a row group to arrive (atomic counter, no
// waiting) selects the experts of its eight rows, one warp per row, logits in registers, a round in two warp reductions.
// All of it is latency: the router rows are asked into L2 before the kernel waits for its input, the activations arrive
// in one batch. EPL: logits per lane.
template <int EPL>
__global__ void __launch_bounds__(ROUTE_THREADS) moe_route_kernel(const RouteParams p, int rows, float * logits, int * counters) {
    extern __shared__ __align__(16) float sm[];
    float * x = sm;  // [ROUTE_ROWS][hidden]
    __shared__ int last_flag;
    const int r0 = blockIdx.x * ROUTE_ROWS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nr = min(ROUTE_ROWS, rows - r0);
    const int n_vec = p.experts + 1;  // index `experts` is the shared-expert gate vector
    const int e0 = blockIdx.y * ROUTE_EXPERTS + warp * 4;
    const float * w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int e = min(e0 + q, n_vec - 1);
        w[q] = e < p.experts ? p.router + (int64_t)e * p.hidden : p.sh_gate;
        if (e0 < n_vec)
            for (int i = lane * 32; i < p.hidden; i += 32 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(w[q] + i));
    }
    pdl_entry();
    const float4 * src = reinterpret_cast<const float4 *>(p.xn + (int64_t)r0 * p.hidden);
    const int live = nr * (p.hidden / 4);
    for (int i = threadIdx.x; i < ROUTE_ROWS * (p.hidden / 4); i += ROUTE_THREADS) {
        if (i < live)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(x + i * 4)), "l"(src + i) : "memory");
        else reinterpret_cast<float4 *>(x)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (e0 < n_vec) {
        float acc[4 * ROUTE_ROWS];
#pragma unroll
        for (int i = 0; i < 4 * ROUTE_ROWS; i++) acc[i] = 0.0f;
#pragma unroll 4
        for (int i = lane * 4; i < p.hidden; i += 128) {
            float4 wv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) wv[q] = __ldg(reinterpret_cast<const float4 *>(w[q] + i));
#pragma unroll
            for (int rr = 0; rr < ROUTE_ROWS; rr++) {
                const float4 xv = *reinterpret_cast<const float4 *>(x + rr * p.hidden + i);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float & s = acc[q * ROUTE_ROWS + rr];
                    s = fmaf(wv[q].x, xv.x, s);
                    s = fmaf(wv[q].y, xv.y, s);
                    s = fmaf(wv[q].z, xv.z, s);
                    s = fmaf(wv[q].w, xv.w, s);
                }
            }
        }
        // sums over the lanes, 16 apart, then 8, ...: afterwards lane i holds value i = 8 q + row
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool high = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < o; i++) {
                const float keep = high ? acc[i + o] : acc[i], send = high ? acc[i] : acc[i + o];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        const int e = e0 + (lane >> 3), rr = lane & 7;
        if (e < n_vec && rr < nr) {
            if (e < p.experts) __stcg(logits + (int64_t)(r0 + rr) * p.experts + e, acc[0]);
            else p.shared_gate[r0 + rr] = 1.0f / (1.0f + (float)exp((double)-acc[0]));
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_flag = atomicAdd(&counters[blockIdx.x], 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (!last_flag) return;
    __threadfence();
    if (threadIdx.x == 0) counters[blockIdx.x] = 0;
    if (warp >= nr) return;
    const int r = r0 + warp;
    uint32_t key[EPL];  // expert lane + 32 k
#pragma unroll
    for (int k = 0; k < EPL; k++) {
        const int e = lane + 32 * k;
        key[k] = e < p.experts ? logit_key(__ldcg(logits + (int64_t)r * p.experts + e)) : 0u;
    }
    // selectExperts (forward.go:393-439): `used` rounds of first-maximum argmax over the experts not yet taken
    int32_t * ids = p.ids + (int64_t)r * p.used;
    float * wts = p.weights + (int64_t)r * p.used;
    float my_logit = 0.0f;  // lane s keeps the logit of slot s (used <= 32)
    for (int slot = 0; slot < p.used; slot++) {
        uint32_t best = 0u;
#pragma unroll
        for (int k = 0; k < EPL; k++) best = max(best, key[k]);
        best = __reduce_max_sync(0xffffffffu, best);
        uint32_t at = 0xffffffffu;
#pragma unroll
        for (int k = EPL - 1; k >= 0; k--)
            if (key[k] == best) at = (uint32_t)(lane + 32 * k);
        at = best ? __reduce_min_sync(0xffffffffu, at) : 0u;  // (nothing but NaN left: expert 0)
        if (lane == slot) my_logit = best ? key_logit(best) : -INFINITY;
        if (lane == 0) ids[slot] = (int32_t)at;
#pragma unroll
        for (int k = 0; k < EPL; k++)
            if (at == (uint32_t)(lane + 32 * k)) key[k] = 0u;  // taken
    }
    // softmax over the selected logits: exp in double, sum in float in slot order
    float mx = lane < p.used ? my_logit : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float wt = lane < p.used ? (float)exp((double)(my_logit - mx)) : 0.0f;
    float total = 0.0f;
    for (int s = 0; s < p.used; s++) total += __shfl_sync(0xffffffffu, wt, s);
    if (lane < p.used) wts[lane] = total > 0.0f ? wt / total : wt;
}

struct GroupParams {
    const int32_t * ids;     // [pairs] expert of pair p = row * used + slot
    int pairs, used, experts, max_segments;
    int32_t * pos_of_pair;   // [pairs] position of the pair in the expert-sorted order
    int32_t * row_of_pos;    // [pairs] source row of the pair at a position
    GemmSegment * segments;  // [max_segments]
};

// One CTA. Stable counting sort of the pairs by expert, cut into segments of at most 8 rows. Every warp takes a run of the
// pairs: it counts them by expert in a row of its own, the rows are scanned over the warps and the experts (one warp), and
// then it walks its run again, 32 pairs at a time in order, __match_any_sync giving every pair its rank among the equal
// experts of its group and the warp's cursor of the expert carrying the ranks on. (One warp walking all pairs was a chain
// of 40 groups for 1280 of them.)
constexpr int GROUP_WARPS = 16;
__global__ void __launch_bounds__(GROUP_WARPS * 32) moe_group_kernel(const GroupParams p) {
    pdl_entry();
    extern __shared__ int cursor[];  // [GROUP_WARPS][experts] counts, then first ranks of the warp's pairs
    __shared__ int count[ROUTE_MAX_EXPERTS];
    __shared__ int pair_off[ROUTE_MAX_EXPERTS];
    __shared__ int seg_off[ROUTE_MAX_EXPERTS];
    __shared__ int total_segments;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int run = ((p.pairs + GROUP_WARPS - 1) / GROUP_WARPS + 31) / 32 * 32, i0 = warp * run, i1 = min(p.pairs, i0 + run);
    int * mine = cursor + warp * p.experts;
    for (int i = threadIdx.x; i < GROUP_WARPS * p.experts; i += GROUP_WARPS * 32) cursor[i] = 0;
    __syncthreads();
    for (int i = i0 + lane; i < i1; i += 32) atomicAdd(&mine[p.ids[i]], 1);
    __syncthreads();
    for (int e = threadIdx.x; e < p.experts; e += GROUP_WARPS * 32) {
        int before = 0;
#pragma unroll
        for (int k = 0; k < GROUP_WARPS; k++) {
            const int c = cursor[k * p.experts + e];
            cursor[k * p.experts + e] = before;
            before += c;
        }
        count[e] = before;
    }
    __syncthreads();
    if (warp == 0) {
        // exclusive scans of the pair counts and of the segment counts, 32 experts at a time
        int pairs_before = 0, segs_before = 0;
        for (int base = 0; base < p.experts; base += 32) {
            const int e = base + lane, c = e < p.experts ? count[e] : 0, sg = (c + GEMM_SEGMENT_ROWS - 1) / GEMM_SEGMENT_ROWS;
            int pr = c, sr = sg;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, pr, o), y = __shfl_up_sync(0xffffffffu, sr, o);
                if (lane >= o) {
                    pr += x;
                    sr += y;
                }
            }
            if (e < p.experts) {
                pair_off[e] = pairs_before + pr - c;
                seg_off[e] = segs_before + sr - sg;
            }
            pairs_before += __shfl_sync(0xffffffffu, pr, 31);
            segs_before += __shfl_sync(0xffffffffu, sr, 31);
        }
        if (lane == 0) total_segments = segs_before;
    }
    __syncthreads();
    for (int base = i0; base < i1; base += 32) {
        const int i = base + lane;
        const bool valid = i < i1;
        const int e = valid ? p.ids[i] : -1 - lane;  // (lanes past the end match nobody)
        const unsigned same = __match_any_sync(0xffffffffu, e);
        const int leader = __ffs(same) - 1, rank = __popc(same & ((1u << lane) - 1u));
        int start = 0;
        if (valid && lane == leader) {
            start = mine[e];
            mine[e] = start + __popc(same);
        }
        start = __shfl_sync(0xffffffffu, start, leader);
        __syncwarp();
        if (valid) {
            const int j = start + rank, c = count[e], pos = pair_off[e] + j;
            p.pos_of_pair[i] = pos;
            p.row_of_pos[pos] = i / p.used;
            if (j % GEMM_SEGMENT_ROWS == 0) {
                const int z = seg_off[e] + j / GEMM_SEGMENT_ROWS;
                if (z < p.max_segments) p.segments[z] = GemmSegment{e, pos, min(GEMM_SEGMENT_ROWS, c - j), 0};
            }
        }
    }
    for (int z = total_segments + threadIdx.x; z < p.max_segments; z += GROUP_WARPS * 32) p.segments[z] = GemmSegment{0, 0, 0, 0};
}

int moe_max_segments(int pairs, int experts) {
    const int by_rows = pairs / GEMM_SEGMENT_ROWS + (experts < pairs ? experts : pairs);
    return by_rows < pairs ? by_rows : pairs;
}

void launch_moe_route(cudaStream_t s, const float * xn, const float * router, const float * sh_gate, int hidden, int experts,
                      int used, int rows, int32_t * ids, float * weights, float * shared_gate, float * logits, int * counters) {
    YK_REQUIRE(hidden % 4 == 0, YUUKA_ERR_UNSUPPORTED, "moe: hidden size %d is not a multiple of 4", hidden);
    YK_REQUIRE(experts <= ROUTE_MAX_EXPERTS && used <= 32 && used <= experts, YUUKA_ERR_UNSUPPORTED,
               "moe: %d experts / %d used exceeds the router kernel's limits (%d / 32)", experts, used, ROUTE_MAX_EXPERTS);
    YK_REQUIRE(experts <= hidden, YUUKA_ERR_UNSUPPORTED, "moe: more experts (%d) than hidden columns (%d)", experts, hidden);
    RouteParams p{xn, router, sh_gate, hidden, experts, used, ids, weights, shared_gate};
    const size_t smem = sizeof(float) * (size_t)ROUTE_ROWS * (size_t)hidden;
    YK_REQUIRE(smem <= 200 * 1024, YUUKA_ERR_UNSUPPORTED, "moe: hidden size %d is too wide for the router kernel", hidden);
    auto kern = experts <= 256 ? moe_route_kernel<8> : moe_route_kernel<ROUTE_MAX_EXPERTS / 32>;
    YK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((rows + ROUTE_ROWS - 1) / ROUTE_ROWS, (experts + 1 + ROUTE_EXPERTS - 1) / ROUTE_EXPERTS);
    launch_k(kern, grid, ROUTE_THREADS, smem, s, p, rows, logits, counters);
    YK_CUDA(cudaGetLastError());
}

void launch_moe_group(cudaStream_t s, const int32_t * ids, int rows, int used, int experts, int32_t * pos_of_pair,
                      int32_t * row_of_pos, GemmSegment * segments, int max_segments) {
    GroupParams p{ids, rows * used, used, experts, max_segments, pos_of_pair, row_of_pos, segments};
    const size_t smem = sizeof(int) * (size_t)GROUP_WARPS * (size_t)experts;
    YK_CUDA(cudaFuncSetAttribute(moe_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_k(moe_group_kernel, 1, GROUP_WARPS * 32, smem, s, p);
    YK_CUDA(cudaGetLastError());
}

struct CombineParams {
    float * x;                 // [rows][hidden] residual stream, updated in place
    const float * expert_out;  // [pairs][hidden] in expert-sorted order
    const float * shared_out;  // [rows][hidden]
    const int32_t * pos_of_pair;
    const float * weights;     // [rows][used]
    const float * shared_gate; // [rows]
    int hidden, used;
};

// forward.go:370-389, same order of operations: tmp = sum over slots of w * out (slot order), then
// + gate * shared, then x += tmp; products and sums rounded separately as the reference does.
__global__ void moe_combine_kernel(const CombineParams p) {
    pdl_entry();
    const int r = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.hidden) return;
    float tmp = 0.0f;
    for (int s = 0; s < p.used; s++) {
        const int pos = p.pos_of_pair[r * p.used + s];
        tmp = __fadd_rn(tmp, __fmul_rn(p.weights[r * p.used + s], p.expert_out[(int64_t)pos * p.hidden + i]));
    }
    tmp = __fadd_rn(tmp, __fmul_rn(p.shared_gate[r], p.shared_out[(int64_t)r * p.hidden + i]));
    float * dst = p.x + (int64_t)r * p.hidden + i;
    *dst = __fadd_rn(*dst, tmp);
}

void launch_moe_combine(cudaStream_t s, float * x, const float * expert_out, const float * shared_out,
                        const int32_t * pos_of_pair, const float * weights, const float * shared_gate, int hidden, int used,
                        int rows) {
    CombineParams p{x, expert_out, shared_out, pos_of_pair, weights, shared_gate, hidden, used};
    dim3 grid((hidden + 255) / 256, rows);
    launch_k(moe_combine_kernel, grid, 256, 0, s, p);
    YK_CUDA(cudaGetLastError());
}

}  // namespace yk
