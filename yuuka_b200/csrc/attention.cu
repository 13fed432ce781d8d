// Paged attention of the verify rows: every row attends to the committed
// positions of its sequence and to its own ancestors among the rows of the
// step (chain or tree), flash-decoding style: key ranges are split over CTAs,
// partial (max, sum, output) triples are merged, and the sigmoid output gate of
// the Qwen3.5 layout is applied (model/qwen35/forward.go:188-220; replaces
// attention_prefill_paged_f32_kernel, kernels/hip/prefill/prefill.hip:683).
//
// attention_mma_kernel multiplies on tensor cores; attention_partial_kernel, fp32 arithmetic on CUDA cores over rows decoded
// from the pool format, takes its place with YUUKA_CUDA_ATTN_FP32=1.
#include <cuda_fp16.h>

#include <cfloat>
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "layers.cuh"
#include "quant.cuh"
#include "xprep.cuh"

namespace yk {

constexpr int ATT_WARPS = 8;
constexpr int ATT_R = 5;                     // query rows per warp
constexpr int ATT_QT = ATT_WARPS * ATT_R;    // query rows per CTA
constexpr int ATT_KT = 32;                   // keys per tile (one per lane)

struct AttnParams {
    float * partial;
    const float * q;
    int ldq;
    int heads, kv_heads, splits, key_split;
    RowMeta rows;
    KvPool pool;
};

__device__ __forceinline__ void kv_decode8(const uint8_t * row, int format, int e8, float w[8]) {
    if (format == YUUKA_KV_F16) {
        const uint4 raw = *reinterpret_cast<const uint4 *>(row + e8 * 16);
        const __half2 * h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __half22float2(h[i]);
            w[2 * i] = f.x;
            w[2 * i + 1] = f.y;
        }
    } else if (format == YUUKA_KV_F32) {
        const float4 * p = reinterpret_cast<const float4 *>(row + e8 * 32);
        float4 a = p[0], b = p[1];
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    } else {
        decode8<YUUKA_DTYPE_Q8_0>(row, e8, w);
    }
}

// The same of an F32 or a Q8_0 row (blocks of 34 bytes: two at a time).
template <bool F32> __device__ __forceinline__ void kv_read8(const uint8_t * row, int e8, float (&w)[8]) {
    if constexpr (F32) {
        const float4 * p = reinterpret_cast<const float4 *>(row + e8 * 32);
        const float4 a = __ldg(p), b = __ldg(p + 1);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    } else {
        const uint16_t * blk = reinterpret_cast<const uint16_t *>(row + (e8 >> 2) * 34);
        const float d = __half2float(__ushort_as_half(__ldg(blk)));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = __ldg(blk + 1 + (e8 & 3) * 4 + i);
            w[2 * i] = d * (float)(int8_t)(q & 0xffu);
            w[2 * i + 1] = d * (float)(int8_t)(q >> 8);
        }
    }
}

template <int HD>
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_partial_kernel(const AttnParams p) {
    pdl_entry();
    constexpr int KSTR = HD + 4;
    extern __shared__ __align__(16) float sm[];
    float * qs = sm;                       // [ATT_QT][HD]
    float * ks = qs + ATT_QT * HD;         // [ATT_KT][KSTR]
    float * vs = ks + ATT_KT * KSTR;       // [ATT_KT][HD]
    float * ps = vs + ATT_KT * HD;         // [ATT_QT][ATT_KT]

    const int seq = blockIdx.z;
    const int kvh = blockIdx.y % p.kv_heads, qt = blockIdx.y / p.kv_heads;
    const int split = blockIdx.x;
    const int G = p.heads / p.kv_heads, N = p.rows.nodes, live = rows_of_seq(p.rows, seq);
    const int sq = seq_of(p.rows, seq);
    const int pos0 = p.rows.pos0[sq];
    const int total = pos0 + live;
    const int k_begin = split * p.key_split;
    const int k_end = min(total, k_begin + p.key_split);
    const int nq = min(ATT_QT, G * live - qt * ATT_QT);
    if (k_begin >= k_end || nq <= 0) return;  // (the merge knows how many ranges hold keys)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float scale = (float)(1.0 / sqrt((double)HD));

    // query rows of this tile: local index qi -> (node, head)
    for (int i = threadIdx.x; i < nq * (HD / 4); i += blockDim.x) {
        int qi = i / (HD / 4), c = i - qi * (HD / 4);
        int gq = qt * ATT_QT + qi, node = gq / G, head = kvh * G + gq % G;
        const float4 * src = reinterpret_cast<const float4 *>(p.q + (int64_t)(seq * N + node) * p.ldq + (int64_t)head * 2 * HD);
        reinterpret_cast<float4 *>(qs + qi * HD)[c] = src[c];
    }

    float m[ATT_R], l[ATT_R], acc[ATT_R][HD / 32];
    uint64_t mask[ATT_R];
#pragma unroll
    for (int r = 0; r < ATT_R; r++) {
        m[r] = -INFINITY;
        l[r] = 0.0f;
#pragma unroll
        for (int j = 0; j < HD / 32; j++) acc[r][j] = 0.0f;
        int qi = warp * ATT_R + r;
        int node = qi < nq ? (qt * ATT_QT + qi) / G : 0;
        mask[r] = qi < nq ? p.rows.anc_mask[seq * N + node] : 0;
    }

    for (int k0 = k_begin; k0 < k_end; k0 += ATT_KT) {
        __syncthreads();
        for (int i = threadIdx.x; i < ATT_KT * (HD / 8); i += blockDim.x) {
            int j = i / (HD / 8), c8 = i - j * (HD / 8);
            int pos = k0 + j;
            float kw[8], vw[8];
            if (pos < k_end) {
                int block = p.pool.tables[(int64_t)sq * p.pool.table_stride + pos / p.pool.block_size];
                int64_t off = ((int64_t)block * p.pool.block_size + pos % p.pool.block_size) * p.pool.row_bytes;
                kv_decode8(p.pool.k + off, p.pool.format, kvh * (HD / 8) + c8, kw);
                kv_decode8(p.pool.v + off, p.pool.format, kvh * (HD / 8) + c8, vw);
            } else {
#pragma unroll
                for (int e = 0; e < 8; e++) kw[e] = vw[e] = 0.0f;
            }
            float4 * kd = reinterpret_cast<float4 *>(ks + j * KSTR + c8 * 8);
            float4 * vd = reinterpret_cast<float4 *>(vs + j * HD + c8 * 8);
            kd[0] = make_float4(kw[0], kw[1], kw[2], kw[3]);
            kd[1] = make_float4(kw[4], kw[5], kw[6], kw[7]);
            vd[0] = make_float4(vw[0], vw[1], vw[2], vw[3]);
            vd[1] = make_float4(vw[4], vw[5], vw[6], vw[7]);
        }
        __syncthreads();

        // scores: lane = key
        float s[ATT_R];
#pragma unroll
        for (int r = 0; r < ATT_R; r++) s[r] = 0.0f;
        const float4 * kr = reinterpret_cast<const float4 *>(ks + lane * KSTR);
#pragma unroll 4
        for (int d4 = 0; d4 < HD / 4; d4++) {
            float4 kv = kr[d4];
#pragma unroll
            for (int r = 0; r < ATT_R; r++) {
                float4 qv = reinterpret_cast<const float4 *>(qs + (warp * ATT_R + r) * HD)[d4];
                s[r] = fmaf(qv.x, kv.x, s[r]);
                s[r] = fmaf(qv.y, kv.y, s[r]);
                s[r] = fmaf(qv.z, kv.z, s[r]);
                s[r] = fmaf(qv.w, kv.w, s[r]);
            }
        }
        const int pos = k0 + lane;
#pragma unroll
        for (int r = 0; r < ATT_R; r++) {
            const int qi = warp * ATT_R + r;
            bool vis = pos < k_end && qi < nq && (pos < pos0 || ((mask[r] >> (pos - pos0)) & 1ull));
            float sv = vis ? s[r] * scale : -INFINITY;
            float mx = sv;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            float m_new = fmaxf(m[r], mx);
            float pr = 0.0f, corr = 1.0f;
            if (m_new != -INFINITY) {
                corr = expf(m[r] - m_new);
                pr = vis ? expf(sv - m_new) : 0.0f;
            }
            float ps_sum = pr;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ps_sum += __shfl_xor_sync(0xffffffffu, ps_sum, o);
            l[r] = l[r] * corr + ps_sum;
            m[r] = m_new;
#pragma unroll
            for (int j = 0; j < HD / 32; j++) acc[r][j] *= corr;
            ps[qi * ATT_KT + lane] = pr;
        }
        __syncwarp();
        // weighted values: lane owns dims lane + 32 j
#pragma unroll 4
        for (int kk = 0; kk < ATT_KT; kk++) {
            float vv[HD / 32];
#pragma unroll
            for (int j = 0; j < HD / 32; j++) vv[j] = vs[kk * HD + lane + 32 * j];
#pragma unroll
            for (int r = 0; r < ATT_R; r++) {
                float pr = ps[(warp * ATT_R + r) * ATT_KT + kk];
#pragma unroll
                for (int j = 0; j < HD / 32; j++) acc[r][j] = fmaf(pr, vv[j], acc[r][j]);
            }
        }
    }

#pragma unroll
    for (int r = 0; r < ATT_R; r++) {
        int qi = warp * ATT_R + r;
        if (qi >= nq) continue;
        int gq = qt * ATT_QT + qi, node = gq / G, head = kvh * G + gq % G;
        float * dst = p.partial + (((int64_t)(seq * N + node) * p.heads + head) * p.splits + split) * (HD + 2);
#pragma unroll
        for (int j = 0; j < HD / 32; j++) dst[lane + 32 * j] = acc[r][j];
        if (lane == 0) {
            dst[HD] = m[r];
            dst[HD + 1] = l[r];
        }
    }
}

// ---------------------------------------------------------------------------
// Tensor-core form of the partial kernel (mma.sync m16n8k16, fp16 operands, fp32 accumulate).
// A CTA covers RB blocks of 16 query rows of one KV head and one key range, two warps per block: each owns half of the
// head dimension, its queries in registers as fp16 hi + lo pairs (so scores keep fp32-level accuracy; keys are exact
// when the pool stores F16 rows, otherwise they are split the same way). The two build the 16 x 32 score tile together,
// each over its two quarters of the head dimension, exchange the sums of the quarters and add the four in one order,
// hence hold the same softmax statistics, and each multiplies the probabilities (fp16) with its half of V.
// K and V of an F16 pool arrive by cp.async, one or two tiles ahead.
// What bounds it: a warp's chain of loads, products and exchange from tile to tile. The form before had four warps per
// block, the queries in shared memory and the next tile in registers: 137 registers in twelve warps, one CTA per SM.
// 32 sequences x 17 rows at contexts of 256 to 3072 (head 256): 356 -> 231 us with the merge.
constexpr int AM_KT = 32;
constexpr int AM_RB_MAX = 5;

// Row blocks per CTA for q_rows query rows of one KV head: as many as there are when one CTA can hold them; beyond that
// the size of four or five that walks the keys with fewer row blocks in all.
static int attention_row_blocks(int q_rows) {
    const int blocks = (q_rows + 15) / 16;
    if (blocks <= AM_RB_MAX) return blocks;
    return (blocks + 4) / 5 * 5 < (blocks + 3) / 4 * 4 ? 5 : 4;
}
int attention_query_ctas(int q_rows) {
    const int per = 16 * attention_row_blocks(q_rows);
    return (q_rows + per - 1) / per;
}
// The key ranges of many sequences are cut for tiles of three or four row blocks, whichever needs fewer.
int attention_query_tiles(int q_rows) {
    const int t3 = (q_rows + 47) / 48, t4 = (q_rows + 63) / 64;
    return t3 * 3 < t4 * 4 ? t3 : t4;
}

__device__ __forceinline__ void mma16816h(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// v as fp16 hi (returned) and the fp16 of the remainder
__device__ __forceinline__ __half split_half(float v, __half & lo) {
    const __half hi = __float2half_rn(v);
    lo = __float2half_rn(v - __half2float(hi));
    return hi;
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __half * p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const __half * p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// Shared memory: stages of [K | K's low halves (KSPLIT) | V] tiles, then the exchange buffers
constexpr int AM_SX = 48 * 32;  // floats per row block
constexpr int attention_stages(bool ksplit, int rb) { return ksplit ? 1 : (rb <= 3 ? 2 : 3); }  // (up to three blocks: two CTAs per SM)
constexpr size_t attention_stage_halves(int hd, bool ksplit) { return (size_t)(ksplit ? 3 : 2) * AM_KT * (hd + 8); }

template <int HD, bool KSPLIT, int RB>
__global__ void __launch_bounds__(RB * 64, RB <= 3 ? 2 : 1) attention_mma_kernel(const AttnParams p) {
    constexpr int AM_ROWS = 16 * RB, THREADS = RB * 64;
    constexpr int STR = HD + 8;   // halves per shared-memory row: 16 bytes of padding spread the banks
    constexpr int DW = HD / 2;    // head dimensions per warp
    constexpr int NT_O = DW / 8;  // 8-column output tiles per warp
    constexpr int KQ = HD / 64;   // 16-dimension steps of a quarter of the head
    constexpr int STAGES = attention_stages(KSPLIT, RB);
    constexpr int CONVERT = RB == 4 ? 4 : 2;  // (five row blocks leave a thread 168 registers instead of 255)
    extern __shared__ __align__(16) uint8_t smraw[];
    __half * stage0 = reinterpret_cast<__half *>(smraw);
    constexpr size_t STAGE = attention_stage_halves(HD, KSPLIT);
    constexpr int V_AT = (KSPLIT ? 2 : 1) * AM_KT * STR;
    pdl_entry();

    const int seq = blockIdx.z;
    const int kvh = blockIdx.y % p.kv_heads, qt = blockIdx.y / p.kv_heads;
    const int split = blockIdx.x;
    const int G = p.heads / p.kv_heads, N = p.rows.nodes, live = rows_of_seq(p.rows, seq);
    const int sq = seq_of(p.rows, seq);
    const int pos0 = p.rows.pos0[sq];
    const int total = pos0 + live;
    const int k_begin = split * p.key_split;
    const int k_end = min(total, k_begin + p.key_split);
    const int nq = min(AM_ROWS, G * live - qt * AM_ROWS);
    if (k_begin >= k_end || nq <= 0) return;  // (the merge knows how many ranges hold keys)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int rb = warp >> 1, hw = warp & 1;  // row block; half of the head dimension
    const float scale = (float)(1.0 / sqrt((double)HD));

    // (block sizes are powers of two in practice: a shift and a mask instead of two integer divisions per piece)
    const int bsz = p.pool.block_size, bshift = (bsz & (bsz - 1)) == 0 ? __ffs(bsz) - 1 : -1;
    const int32_t * table = p.pool.tables + (int64_t)sq * p.pool.table_stride;
    auto row_offset = [&](int pos) {
        const int bi = bshift >= 0 ? pos >> bshift : pos / bsz, within = bshift >= 0 ? pos & (bsz - 1) : pos - bi * bsz;
        return ((int64_t)__ldg(table + bi) * bsz + within) * p.pool.row_bytes;
    };
    constexpr int PIECES = AM_KT * (HD / 8);  // 16-byte pieces (eight fp16 values) of a K or V tile
    auto fetch = [&](int tile) {  // F16 pool: cp.async, zeros beyond the range
        __half * st = stage0 + (size_t)(tile % STAGES) * STAGE;
        const int k0 = k_begin + tile * AM_KT;
#pragma unroll 4
        for (int i = threadIdx.x; i < PIECES; i += THREADS) {
            const int j = i / (HD / 8), c8 = i - j * (HD / 8), pos = k0 + j;
            const bool in = pos < k_end;
            const size_t off = in ? row_offset(pos) + (size_t)(kvh * HD + c8 * 8) * 2 : 0;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(st + j * STR + c8 * 8);
            const int bytes = in ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p.pool.k + off), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + V_AT * 2), "l"(p.pool.v + off), "r"(bytes) : "memory");
        }
    };
    // F32 or Q8_0 pool: by way of registers, the loads of CONVERT pieces in flight at once. (One after the other, each behind
    // the stores of the one before, a 9-row step over 16,000 F32 rows took 755 us in four layers instead of 644.)
    auto convert = [&](int tile, auto f32) {
        const int k0 = k_begin + tile * AM_KT;
        for (int i0 = threadIdx.x; i0 < PIECES; i0 += CONVERT * THREADS) {
            float kw[CONVERT][8], vw[CONVERT][8];
#pragma unroll
            for (int u = 0; u < CONVERT; u++) {
                const int i = min(i0 + u * THREADS, PIECES - 1), j = i / (HD / 8), e8 = kvh * (HD / 8) + i - j * (HD / 8);
                const int64_t off = row_offset(min(k0 + j, k_end - 1));
                kv_read8<decltype(f32)::value>(p.pool.k + off, e8, kw[u]);
                kv_read8<decltype(f32)::value>(p.pool.v + off, e8, vw[u]);
            }
#pragma unroll
            for (int u = 0; u < CONVERT; u++) {
                const int i = i0 + u * THREADS, j = i / (HD / 8), c8 = i - j * (HD / 8);
                if (i >= PIECES) continue;
                const bool in = k0 + j < k_end;
                __half hh[8], ll[8], vv[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    hh[e] = split_half(in ? kw[u][e] : 0.0f, ll[e]);
                    vv[e] = __float2half_rn(in ? vw[u][e] : 0.0f);
                }
                __half * at = stage0 + j * STR + c8 * 8;
                *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(hh);
                *reinterpret_cast<uint4 *>(at + AM_KT * STR) = *reinterpret_cast<const uint4 *>(ll);
                *reinterpret_cast<uint4 *>(at + V_AT) = *reinterpret_cast<const uint4 *>(vv);
            }
        }
    };
    const int tiles = (k_end - k_begin + AM_KT - 1) / AM_KT;
    if constexpr (!KSPLIT) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; s++) {
            if (s < tiles) fetch(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }

    // the two query rows of this lane (local rows rb * 16 + g and + 8): fragments of this warp's half of the head
    // dimension, zeros beyond nq; the rows' ancestor masks
    uint32_t qh[2 * KQ][4], ql[2 * KQ][4];
    uint64_t mask[2];
    int row_ok[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int qi = rb * 16 + g + 8 * h;
        row_ok[h] = qi < nq;
        const int gq = qt * AM_ROWS + (row_ok[h] ? qi : 0), node = gq / G, head = kvh * G + gq - node * G;
        mask[h] = row_ok[h] ? p.rows.anc_mask[seq * N + node] : 0ull;
        const float * src = p.q + (int64_t)(seq * N + node) * p.ldq + (int64_t)head * 2 * HD + hw * DW + 2 * t;
#pragma unroll
        for (int kk = 0; kk < 2 * KQ; kk++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float2 v = row_ok[h] ? *reinterpret_cast<const float2 *>(src + 16 * kk + 8 * e) : make_float2(0.f, 0.f);
                __half lx, ly;
                const __half hx = split_half(v.x, lx), hy = split_half(v.y, ly);
                const __half2 hi = __halves2half2(hx, hy), lo = __halves2half2(lx, ly);
                qh[kk][h + 2 * e] = *reinterpret_cast<const uint32_t *>(&hi);
                ql[kk][h + 2 * e] = *reinterpret_cast<const uint32_t *>(&lo);
            }
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
    float o[NT_O][4];
#pragma unroll
    for (int nt = 0; nt < NT_O; nt++)
#pragma unroll
        for (int c = 0; c < 4; c++) o[nt][c] = 0.0f;
    float4 * sx = reinterpret_cast<float4 *>(reinterpret_cast<float *>(stage0 + STAGES * STAGE) + rb * AM_SX) + lane;

    for (int tile = 0; tile < tiles; tile++) {
        const int k0 = k_begin + tile * AM_KT;
        const __half * ks = stage0 + (size_t)(tile % STAGES) * STAGE;
        if constexpr (!KSPLIT) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();  // the tile has landed, and the previous one has been consumed
            if (tile + STAGES - 1 < tiles) fetch(tile + STAGES - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
            __syncthreads();
            if (p.pool.format == YUUKA_KV_F32) convert(tile, std::true_type());
            else convert(tile, std::false_type());
            __syncthreads();
        }
        if (rb * 16 >= nq) continue;  // (both warps of the block)

        // scores of the block's 16 rows against the 32 keys: this warp's two quarters of the head dimension
        float s[2][4][4];
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int nt = 0; nt < 4; nt++)
#pragma unroll
                for (int c = 0; c < 4; c++) s[q][nt][c] = 0.0f;
        const __half * krow = ks + (8 * (lane >> 4) + (lane & 7)) * STR + hw * DW + 8 * ((lane >> 3) & 1);
#pragma unroll
        for (int kk = 0; kk < 2 * KQ; kk++) {
            const int q = kk / KQ;
#pragma unroll
            for (int n2 = 0; n2 < 2; n2++) {
                uint32_t b[4];
                ldmatrix4(b, krow + 16 * n2 * STR + 16 * kk);
                mma16816h(s[q][2 * n2], qh[kk], b[0], b[1]);
                mma16816h(s[q][2 * n2 + 1], qh[kk], b[2], b[3]);
                mma16816h(s[q][2 * n2], ql[kk], b[0], b[1]);
                mma16816h(s[q][2 * n2 + 1], ql[kk], b[2], b[3]);
                if constexpr (KSPLIT) {
                    uint32_t bl[4];
                    ldmatrix4(bl, krow + AM_KT * STR + 16 * n2 * STR + 16 * kk);
                    mma16816h(s[q][2 * n2], qh[kk], bl[0], bl[1]);
                    mma16816h(s[q][2 * n2 + 1], qh[kk], bl[2], bl[3]);
                }
            }
        }
        // the four quarters meet, always as ((q0 + q1) + q2) + q3
        if (hw == 0) {
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
#pragma unroll
                for (int c = 0; c < 4; c++) s[0][nt][c] = s[0][nt][c] + s[1][nt][c];
                sx[nt * 32] = make_float4(s[0][nt][0], s[0][nt][1], s[0][nt][2], s[0][nt][3]);
            }
        } else {
#pragma unroll
            for (int nt = 0; nt < 4; nt++) {
                sx[(4 + nt) * 32] = make_float4(s[0][nt][0], s[0][nt][1], s[0][nt][2], s[0][nt][3]);
                sx[(8 + nt) * 32] = make_float4(s[1][nt][0], s[1][nt][1], s[1][nt][2], s[1][nt][3]);
            }
        }
        asm volatile("bar.sync %0, 64;" ::"r"(rb + 1) : "memory");
        float sc[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; nt++) {
            if (hw == 0) {
                const float4 q2 = sx[(4 + nt) * 32], q3 = sx[(8 + nt) * 32];
                sc[nt][0] = (s[0][nt][0] + q2.x) + q3.x;
                sc[nt][1] = (s[0][nt][1] + q2.y) + q3.y;
                sc[nt][2] = (s[0][nt][2] + q2.z) + q3.z;
                sc[nt][3] = (s[0][nt][3] + q2.w) + q3.w;
            } else {
                const float4 q01 = sx[nt * 32];
                sc[nt][0] = (q01.x + s[0][nt][0]) + s[1][nt][0];
                sc[nt][1] = (q01.y + s[0][nt][1]) + s[1][nt][1];
                sc[nt][2] = (q01.z + s[0][nt][2]) + s[1][nt][2];
                sc[nt][3] = (q01.w + s[0][nt][3]) + s[1][nt][3];
            }
        }
        // mask, online softmax; sc[nt][0,1] -> row g, keys 8 nt + 2 t + {0,1}; sc[nt][2,3] -> row g + 8
        uint32_t pa[2][4];  // probabilities as A fragments of the two 16-key steps
        float corr[2];
        // a tile that lies entirely in the committed context is visible to every row: no mask, no range test
        const bool plain_tile = k0 + AM_KT <= min(pos0, k_end);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float sv[4][2];
            float mx = -INFINITY;
            if (plain_tile) {
#pragma unroll
                for (int nt = 0; nt < 4; nt++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        sv[nt][e] = row_ok[h] ? sc[nt][2 * h + e] * scale : -INFINITY;
                        mx = fmaxf(mx, sv[nt][e]);
                    }
            } else {
#pragma unroll
                for (int nt = 0; nt < 4; nt++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int pos = k0 + 8 * nt + 2 * t + e;
                        const bool vis = pos < k_end && row_ok[h] && (pos < pos0 || ((mask[h] >> (pos - pos0)) & 1ull));
                        sv[nt][e] = vis ? sc[nt][2 * h + e] * scale : -INFINITY;
                        mx = fmaxf(mx, sv[nt][e]);
                    }
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m[h], mx);
            float sum = 0.0f;
            float pr[4][2];
            corr[h] = m_new != -INFINITY ? __expf(m[h] - m_new) : 1.0f;
#pragma unroll
            for (int nt = 0; nt < 4; nt++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    // (ex2.approx: the value is rounded to fp16 on the next line, 2^-11 against the approximation's 2^-22)
                    const float pv = (m_new != -INFINITY && sv[nt][e] != -INFINITY) ? __expf(sv[nt][e] - m_new) : 0.0f;
                    pr[nt][e] = __half2float(__float2half_rn(pv));  // the value the tensor core will see
                    sum += pr[nt][e];
                }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[h] = l[h] * corr[h] + sum;
            m[h] = m_new;
            // A fragment registers: [0] row g / [1] row g+8 for keys 2t..; [2], [3] the same rows, keys 2t+8..
            pa[0][h] = pack_h2(pr[0][0], pr[0][1]);
            pa[0][2 + h] = pack_h2(pr[1][0], pr[1][1]);
            pa[1][h] = pack_h2(pr[2][0], pr[2][1]);
            pa[1][2 + h] = pack_h2(pr[3][0], pr[3][1]);
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.0f || corr[1] != 1.0f)) {  // (a maximum moved)
#pragma unroll
            for (int nt = 0; nt < NT_O; nt++) {
                o[nt][0] *= corr[0];
                o[nt][1] *= corr[0];
                o[nt][2] *= corr[1];
                o[nt][3] *= corr[1];
            }
        }
        // O += P V on this warp's half of the head dimension
        const __half * vrow = ks + V_AT + (lane & 15) * STR + hw * DW + 8 * (lane >> 4);
#pragma unroll
        for (int kk = 0; kk < 2; kk++)
#pragma unroll
            for (int nt = 0; nt < NT_O; nt += 2) {
                uint32_t b[4];
                ldmatrix4_trans(b, vrow + 16 * kk * STR + 8 * nt);
                mma16816h(o[nt], pa[kk], b[0], b[1]);
                mma16816h(o[nt + 1], pa[kk], b[2], b[3]);
            }
    }

#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!row_ok[h]) continue;
        const int gq = qt * AM_ROWS + rb * 16 + g + 8 * h, node = gq / G, head = kvh * G + gq % G;
        float * dst = p.partial + (((int64_t)(seq * N + node) * p.heads + head) * p.splits + split) * (HD + 2);
#pragma unroll
        for (int nt = 0; nt < NT_O; nt++) {
            float2 v = make_float2(o[nt][2 * h], o[nt][2 * h + 1]);
            *reinterpret_cast<float2 *>(dst + hw * DW + 8 * nt + 2 * t) = v;
        }
        if (hw == 0 && t == 0) {
            dst[HD] = m[h];
            dst[HD + 1] = l[h];
        }
    }
}

// float exp: the CPU reference evaluates exp in f64 and rounds; the difference is below 2e-7 relative
__device__ __forceinline__ float sigmoid_ref(float x) { return 1.0f / (1.0f + expf(-x)); }

// One CTA per (row, head): the split statistics are combined once in shared memory, then every thread
// sums its four output dims over the splits that saw a key (independent, coalesced loads), applies the
// sigmoid gate, and a 16-dim group leader writes the prepared form.
constexpr int MERGE_MAX_SPLITS = 1024;

template <int HD>
__global__ void __launch_bounds__(HD / 4 < 32 ? 32 : HD / 4) attention_merge_kernel(float * __restrict__ out, int ldo, const float * __restrict__ partial,
                                                                 const float * __restrict__ q, int ldq, int heads, int all_splits,
                                                                 int key_split, const RowMeta rows, XPrepOut prep) {
    pdl_entry();
    __shared__ float w_s[MERGE_MAX_SPLITS], l_s[MERGE_MAX_SPLITS];
    __shared__ float inv_l;
    const int r = blockIdx.x / heads, head = blockIdx.x - r * heads;
    const int tid = threadIdx.x;
    // the key ranges that hold keys of the row's sequence; the others have written nothing
    const int seq = r / rows.nodes, splits = (rows.pos0[seq_of(rows, seq)] + rows_of_seq(rows, seq) + key_split - 1) / key_split;
    const float * base = partial + ((int64_t)r * heads + head) * all_splits * (HD + 2);
    constexpr int THREADS = HD / 4 < 32 ? 32 : HD / 4;  // whole warps; threads beyond HD / 4 only help with the statistics
    const bool has_dims = tid < HD / 4;
    // the split's running maximum and sum, all splits in flight at once (one lane summing them straight from
    // global memory was a chain of dependent L2 round trips: 12 us of this kernel at 23 splits)
    for (int s = tid; s < splits; s += THREADS) {
        const float2 ml = *reinterpret_cast<const float2 *>(base + (size_t)s * (HD + 2) + HD);
        w_s[s] = ml.x;
        l_s[s] = ml.y;
    }
    __syncthreads();
    if (tid < 32) {
        float M = -INFINITY;
        for (int s = tid; s < splits; s += 32) M = fmaxf(M, w_s[s]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        // weights exp(m_s - M); the normaliser is summed in split order by one lane, as the serial form did
        for (int s = tid; s < splits; s += 32) {
            const float ms = w_s[s];
            w_s[s] = ms == -INFINITY ? 0.0f : expf(ms - M);
        }
        __syncwarp();
        if (tid == 0) {
            float L = 0.0f;
            for (int s = 0; s < splits; s++)
                if (w_s[s] != 0.0f) L += l_s[s] * w_s[s];
            inv_l = L > 0.0f ? 1.0f / L : 0.0f;
        }
    }
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const float * col = base + (has_dims ? tid : 0) * 4;
#pragma unroll 8
    for (int s = 0; s < splits; s++) {
        const float w = w_s[s];
        if (w == 0.0f) continue;
        const float2 lo = *reinterpret_cast<const float2 *>(col + (size_t)s * (HD + 2));
        const float2 hi = *reinterpret_cast<const float2 *>(col + (size_t)s * (HD + 2) + 2);
        acc.x = fmaf(lo.x, w, acc.x);
        acc.y = fmaf(lo.y, w, acc.y);
        acc.z = fmaf(hi.x, w, acc.z);
        acc.w = fmaf(hi.y, w, acc.w);
    }
    const float inv = inv_l;
    const float4 gate =
        *reinterpret_cast<const float4 *>(q + (int64_t)r * ldq + (int64_t)head * 2 * HD + HD + (has_dims ? tid : 0) * 4);
    float4 o;
    o.x = acc.x * inv * sigmoid_ref(gate.x);
    o.y = acc.y * inv * sigmoid_ref(gate.y);
    o.z = acc.z * inv * sigmoid_ref(gate.z);
    o.w = acc.w * inv * sigmoid_ref(gate.w);
    if (prep.hi_only()) {
        if (has_dims) xprep_store_hi4(prep.xh + (int64_t)r * heads * HD + head * HD + tid * 4, o.x, o.y, o.z, o.w);
        return;
    }
    if (has_dims) *reinterpret_cast<float4 *>(out + (int64_t)r * ldo + head * HD + tid * 4) = o;
    if (prep.xh) {
        // gather the 16-dim group in its first lane (four neighbouring threads hold it)
        float v[16];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[4 * k] = __shfl_sync(0xffffffffu, o.x, (tid & 28) + k);
            v[4 * k + 1] = __shfl_sync(0xffffffffu, o.y, (tid & 28) + k);
            v[4 * k + 2] = __shfl_sync(0xffffffffu, o.z, (tid & 28) + k);
            v[4 * k + 3] = __shfl_sync(0xffffffffu, o.w, (tid & 28) + k);
        }
        if ((tid & 3) == 0 && has_dims) {
            const int cols = heads * HD, gq = head * (HD / 16) + (tid >> 2);
            xprep_store16(prep.xh + (int64_t)r * cols + gq * 16, prep.xl + (int64_t)r * cols + gq * 16, prep.xs16 + (int64_t)r * (cols >> 4) + gq, v);
        }
    }
}

size_t attention_scratch_floats(int rows, int heads, int head_dim, int splits) {
    return (size_t)rows * heads * splits * (head_dim + 2);
}

template <int HD>
static int launch_attention_hd(cudaStream_t s, float * out, int ldo, const float * q, int ldq, int heads, int kv_heads,
                               const RowMeta & rows, const KvPool & pool, const AttnScratch & sc, XPrepOut prep) {
    AttnParams p;
    p.partial = sc.partial;
    p.q = q;
    p.ldq = ldq;
    p.heads = heads;
    p.kv_heads = kv_heads;
    p.splits = sc.splits;
    p.key_split = sc.key_split;
    p.rows = rows;
    p.pool = pool;
    const int G = heads / kv_heads;
    static const bool use_mma = [] { const char * e = getenv("YUUKA_CUDA_ATTN_FP32"); return !(e && e[0] == '1'); }();
    if (use_mma) {
        // tensor-core partials; keys are taken as they are from an F16 pool and split into hi + lo otherwise
        // (F32 and Q8_0 rows are converted on the way in: by eight warps at least, which have a tile's loads in flight all at
        // once. With the ten of a CTA of five row blocks a one-row step over 16,000 Q8_0 rows took 643 us in four layers, with
        // eight 545)
        const bool convert = pool.format != YUUKA_KV_F16;
        const int blocks = attention_row_blocks(G * rows.nodes), rb = convert ? std::max(blocks, 4) : blocks;
        const int qtiles = (G * rows.nodes + 16 * rb - 1) / (16 * rb);
        auto launch = [&](auto ksplit) {
            constexpr bool KS = decltype(ksplit)::value;
            auto with = [&](auto kern) {
                const size_t smem = sizeof(__half) * attention_stages(KS, rb) * attention_stage_halves(HD, KS) + sizeof(float) * AM_SX * rb;
                YK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                launch_k(kern, dim3(sc.splits, kv_heads * qtiles, rows.batch), rb * 64, smem, s, p);
            };
            if (rb == 5) with(attention_mma_kernel<HD, KS, 5>);
            else if (rb == 4) with(attention_mma_kernel<HD, KS, 4>);
            else if constexpr (!KS) {
                if (rb == 3) with(attention_mma_kernel<HD, KS, 3>);
                else if (rb == 2) with(attention_mma_kernel<HD, KS, 2>);
                else with(attention_mma_kernel<HD, KS, 1>);
            }
        };
        if (convert) launch(std::true_type());
        else launch(std::false_type());
        YK_CUDA(cudaGetLastError());
    } else {
        const int qtiles = (G * rows.nodes + ATT_QT - 1) / ATT_QT;
        size_t smem = sizeof(float) * ((size_t)ATT_QT * HD + ATT_KT * (HD + 4) + ATT_KT * HD + ATT_QT * ATT_KT);
        auto kern = attention_partial_kernel<HD>;
        YK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        dim3 grid(sc.splits, kv_heads * qtiles, rows.batch);
        launch_k(kern, grid, ATT_WARPS * 32, smem, s, p);
        YK_CUDA(cudaGetLastError());
    }
    YK_REQUIRE(sc.splits <= MERGE_MAX_SPLITS, YUUKA_ERR_UNSUPPORTED, "attention: %d key splits exceed the merge kernel's %d",
               sc.splits, MERGE_MAX_SPLITS);
    launch_k(attention_merge_kernel<HD>, rows_of_step(rows) * heads, HD / 4 < 32 ? 32 : HD / 4, 0, s, out, ldo, sc.partial, q, ldq, heads,
             sc.splits, sc.key_split, rows, prep);
    YK_CUDA(cudaGetLastError());
    return 2;
}

int launch_attention(cudaStream_t s, float * out, int ldo, const float * q, int ldq, int heads, int kv_heads,
                     int head_dim, const RowMeta & rows, const KvPool & pool, int max_total_keys,
                     const AttnScratch & scratch, XPrepOut prep) {
    YK_REQUIRE(rows.nodes <= 64, YUUKA_ERR_UNSUPPORTED, "attention: at most 64 rows per sequence");
    YK_REQUIRE((int64_t)scratch.splits * scratch.key_split >= max_total_keys, YUUKA_ERR_INTERNAL,
               "attention: key splits do not cover %d keys", max_total_keys);
    switch (head_dim) {
    case 64: return launch_attention_hd<64>(s, out, ldo, q, ldq, heads, kv_heads, rows, pool, scratch, prep);
    case 128: return launch_attention_hd<128>(s, out, ldo, q, ldq, heads, kv_heads, rows, pool, scratch, prep);
    case 256: return launch_attention_hd<256>(s, out, ldo, q, ldq, heads, kv_heads, rows, pool, scratch, prep);
    default: YK_REQUIRE(false, YUUKA_ERR_UNSUPPORTED, "attention: head_dim %d is not 64, 128 or 256", head_dim);
    }
    return 0;
}

}  // namespace yk
