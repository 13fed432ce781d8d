// On-device acceptance for a verify step.
//
// Greedy: first-maximum argmax of every logits row (argmaxLogit,
// engine/speculative.go:263-271) and the prefix walk of the accept loop
// (engine/speculative.go:193-202), generalised from a chain to a tree: at node
// cur the wanted token is argmax(logits[cur]); the lowest-numbered child of
// cur that carries it is accepted and becomes cur; otherwise the wanted token
// is emitted as the correction and the walk ends.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "layers.cuh"

namespace yk {

constexpr int ARGMAX_CHUNK = 4096;

// (value, index) with the reference's tie rule: larger value wins, equal
// values keep the lower index. NaNs never win against a number.
__device__ __forceinline__ void best_of(float & v, int & i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) {
        v = ov;
        i = oi;
    }
}

__global__ void __launch_bounds__(256) argmax_partial_kernel(const float * __restrict__ logits, int vocab,
                                                             float * __restrict__ val, int32_t * __restrict__ idx,
                                                             int chunks) {
    pdl_entry();
    const int r = blockIdx.y, c = blockIdx.x;
    const float * row = logits + (int64_t)r * vocab;
    const int begin = c * ARGMAX_CHUNK, end = min(vocab, begin + ARGMAX_CHUNK);
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    if (end - begin == ARGMAX_CHUNK && ((uintptr_t)(row + begin) & 15) == 0) {
        // a whole chunk: all of a thread's loads are in flight at once (bound by DRAM: 64 x 9 x 248320 logits)
        float4 v[ARGMAX_CHUNK / 1024];
#pragma unroll
        for (int u = 0; u < ARGMAX_CHUNK / 1024; u++) v[u] = __ldcs(reinterpret_cast<const float4 *>(row + begin) + u * 256 + threadIdx.x);
#pragma unroll
        for (int u = 0; u < ARGMAX_CHUNK / 1024; u++) {
            const int i = begin + (u * 256 + (int)threadIdx.x) * 4;
            best_of(bv, bi, v[u].x, i);
            best_of(bv, bi, v[u].y, i + 1);
            best_of(bv, bi, v[u].z, i + 2);
            best_of(bv, bi, v[u].w, i + 3);
        }
    } else {
        for (int i = begin + threadIdx.x; i < end; i += blockDim.x) best_of(bv, bi, row[i], i);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        best_of(bv, bi, ov, oi);
    }
    __shared__ float sv[8];
    __shared__ int si[8];
    if ((threadIdx.x & 31) == 0) {
        sv[threadIdx.x >> 5] = bv;
        si[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) best_of(bv, bi, sv[w], si[w]);
        val[(int64_t)r * chunks + c] = bv;
        idx[(int64_t)r * chunks + c] = bi;
    }
}

struct WalkParams {
    const float * val;
    const int32_t * idx;
    int chunks;
    RowMeta rows;
    AcceptOut out;
};

// one CTA per sequence: finish the argmax of each of its rows (a warp per row, lanes over the chunk maxima,
// combined with the same tie rule), then one thread walks the tree, whose tokens and parents wait in shared memory
constexpr int WALK_THREADS = 256;
__global__ void __launch_bounds__(WALK_THREADS) greedy_walk_kernel(const WalkParams p) {
    pdl_entry();
    __shared__ int want[64], tok_s[64], par_s[64];
    const int seq = blockIdx.x, N = p.rows.nodes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int node = threadIdx.x; node < N; node += blockDim.x) {
        tok_s[node] = p.rows.tokens[(int64_t)seq * N + node];
        par_s[node] = p.rows.parent[(int64_t)seq * N + node];
    }
    for (int node = warp; node < N; node += WALK_THREADS / 32) {
        const int r = seq * N + node;
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int c = lane; c < p.chunks; c += 32) best_of(bv, bi, p.val[(int64_t)r * p.chunks + c], p.idx[(int64_t)r * p.chunks + c]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            best_of(bv, bi, ov, oi);
        }
        if (lane == 0) want[node] = bi == 0x7fffffff ? 0 : bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t * path = p.out.path + (int64_t)seq * N;
        int32_t * emitted = p.out.emitted + (int64_t)seq * N;
        int cur = 0, a = 0;
        for (;;) {
            const int w = want[cur];
            int next = -1;
            for (int c = cur + 1; c < N; c++)
                if (par_s[c] == cur && tok_s[c] == w) { next = c; break; }
            emitted[a] = w;
            if (next < 0) break;
            path[a] = next;
            a++;
            cur = next;
        }
        for (int i = a; i < N; i++) path[i] = -1;
        for (int i = a + 1; i < N; i++) emitted[i] = -1;
        p.out.accepted[seq] = a;
    }
}

int launch_accept_greedy(cudaStream_t s, const float * logits, int vocab, const RowMeta & rows,
                         const ArgmaxScratch & scratch, const AcceptOut & out) {
    const int R = rows.batch * rows.nodes;
    const int chunks = (vocab + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
    YK_REQUIRE(chunks <= scratch.chunks, YUUKA_ERR_INTERNAL, "argmax scratch is too small");
    dim3 grid(chunks, R);
    launch_k(argmax_partial_kernel, grid, 256, 0, s, logits, vocab, scratch.val, scratch.idx, scratch.chunks);
    YK_CUDA(cudaGetLastError());
    WalkParams p{scratch.val, scratch.idx, scratch.chunks, rows, out};
    launch_k(greedy_walk_kernel, rows.batch, WALK_THREADS, 0, s, p);
    YK_CUDA(cudaGetLastError());
    return 2;
}

// ---------------------------------------------------------------------------
// Rejection-sampling acceptance over a draft tree (not in the reference, which
// verifies greedily only: engine/speculative.go:73-75). The rule is written so
// that every deciding quantity is an elementwise IEEE operation or an integer
// sum; the result does not depend on the order of the parallel reductions.
//
// At node cur (start: the root), with children in row order:
//   mx  = max_i L[cur][i];  e_i = exp_det((L[cur][i] - mx) / T);  w_i = (uint64)(e_i * 2^40)
//   r = w, R = sum w
//   child c (token x, draft distribution Q[c], uniform u = U[2c]):
//     accept iff (double)(u * Q[c][x]) * (double)R <= (double)r_x      -> cur = c, start over at c
//     else r_i = max(0, r_i - (uint64)((double)Q[c][i] * (double)R)), R = sum r  (R == 0: r = w again)
//   no child accepted: t = min((uint64)((double)U[2 cur + 1] * (double)R), R - 1);
//     emit the smallest j with sum_{i <= j} r_i > t.

// Packed fp32 pairs (fma / mul / add.rn.f32x2): the IEEE results of the scalar forms in half the instructions.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma_p(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long mul_p(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add_p(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
// Weights of two logits: w = (uint64)(exp_det((L - mx) / T) * 2^40) with
//   exp_det(x): n = rint(x * 1.44269504), r = x - n ln 2 in two parts, a degree-5 polynomial, times 2^n; 0 below -87.
// (the polynomial and the parts of ln 2 are those of expf in the Cephes library). rint is an addition and subtraction of
// 1.5 * 2^23 (|x log2 e| < 2^22), whose low bits are n; 2^n * 2^40 is one exact multiplication; x is clamped at -87, where
// the weight is 0 as well (anything below 2^-40 is). A logit of +infinity, or a 1 / T that overflows, makes x a NaN at the
// maximum: it passes the clamp and converts to 2^63, so that such a token takes all the weight.
__device__ __forceinline__ void target_weights2(float l0, float l1, float mx, float inv_t, unsigned long long & w0, unsigned long long & w1) {
    const float2 xs = unpack2(mul_p(add_p(pack2(l0, l1), pack2(-mx, -mx)), pack2(inv_t, inv_t)));
    const unsigned long long x = pack2(max_nan(xs.x, -87.0f), max_nan(xs.y, -87.0f));
    const unsigned long long shifted = add_p(mul_p(x, pack2(1.44269504f, 1.44269504f)), pack2(12582912.0f, 12582912.0f));
    const unsigned long long n = add_p(shifted, pack2(-12582912.0f, -12582912.0f));
    unsigned long long r = fma_p(n, pack2(-0.693359375f, -0.693359375f), x);
    r = fma_p(n, pack2(2.12194440e-4f, 2.12194440e-4f), r);
    unsigned long long q = fma_p(pack2(1.9875691500e-4f, 1.9875691500e-4f), r, pack2(1.3981999507e-3f, 1.3981999507e-3f));
    q = fma_p(q, r, pack2(8.3334519073e-3f, 8.3334519073e-3f));
    q = fma_p(q, r, pack2(4.1665795894e-2f, 4.1665795894e-2f));
    q = fma_p(q, r, pack2(1.6666665459e-1f, 1.6666665459e-1f));
    q = fma_p(q, r, pack2(5.0000001201e-1f, 5.0000001201e-1f));
    const unsigned long long e = add_p(fma_p(q, mul_p(r, r), r), pack2(1.0f, 1.0f));
    const float2 ns = unpack2(shifted);
    // (low bits of the shifted value + 127 + 40, moved into the exponent: the upper bits drop out)
    const float s0 = __uint_as_float((__float_as_uint(ns.x) + 167u) << 23), s1 = __uint_as_float((__float_as_uint(ns.y) + 167u) << 23);
    const float2 v = unpack2(mul_p(e, pack2(s0, s1)));
    w0 = (unsigned long long)v.x;
    w1 = (unsigned long long)v.y;
}

constexpr int REJ_THREADS = 512;
constexpr int REJ_WARPS = REJ_THREADS / 32;
constexpr int REJ_MAX_CLUSTER = 8;   // CTAs that share one sequence's vocabulary
constexpr int REJ_MAX_NODES = 64;
constexpr int REJ_KEEP = 2;       // rejected drafts of a node whose rows a pass reads again; at this many the weights are stored

struct RejectParams {
    const float * logits;   // [batch][nodes][vocab]
    const float * q;        // [batch][nodes][vocab]
    const float * u;        // [batch][nodes][2]
    unsigned long long * r; // [batch][vocab], for trees with many siblings (see REJ_STORE_SIBLINGS), else null
    int vocab;
    float inv_t;
    RowMeta rows;
    AcceptOut out;
};

__device__ __forceinline__ void st_cluster_u64(unsigned long long * p, unsigned rank, unsigned long long v) {
    const uint32_t local = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(v) : "memory");
}
// four consecutive values from p + i, `fill` beyond n (VEC: p is 16-byte aligned, i and n are multiples of four)
template <bool VEC>
__device__ __forceinline__ float4 load4(const float * p, int i, int n, float fill) {
    if (VEC) return i < n ? *reinterpret_cast<const float4 *>(p + i) : make_float4(fill, fill, fill, fill);
    return make_float4(i < n ? p[i] : fill, i + 1 < n ? p[i + 1] : fill, i + 2 < n ? p[i + 2] : fill, i + 3 < n ? p[i + 3] : fill);
}
__device__ __forceinline__ unsigned long long take_away(unsigned long long r, float q, double R) {
    const unsigned long long qr = (unsigned long long)__dmul_rn((double)q, R);
    return r > qr ? r - qr : 0ull;
}

// One sequence per cluster of CL CTAs; CTA c owns the vocabulary slice [c * slice, (c + 1) * slice), a warp of it a
// contiguous run of `run` tokens. All CTAs of a cluster walk the tree together: the deciding quantities (the
// maximum, R, r[x], the uniforms) are the same everywhere, so they take the same turns; rank 0 writes the path.
//
// The residual weights are not stored as long as a node has few children. They are elementwise functions of a row of
// logits and of the draft rows rejected at the node so far, so each pass recomputes them from those rows, which the first pass has left in L2:
// 4 bytes read per token and pass, where keeping them moved 16. What bounds the walk is then latency (two
// passes, two exchanges a node, each behind the one before), so the grid is chosen for one wave of all sequences
// (rejection_cluster), with two CTAs to an SM to overlap one's exchanges with another's passes.
// 64 sequences x 9 rows x 248,320 tokens at T = 0.7 (1.6 accepted a sequence): 361 -> 181 us, one sequence 39 us; all
// eight drafts accepted 262 us, of which 9 x 64 MB of logits are 90 us at the measured copy rate.
// Each pass after a rejection reads one draft row more, so a node with many children stores the weights from the second
// rejection on and each pass reads them and one draft row. One sequence, all drafts children of the root and rejected:
// eight drafts 224 -> 127 us, sixteen 634 -> 225, 63 7167 -> 963; with four 93 either way, so those go without the scratch.
// Sums and maxima cross the cluster by stores into every CTA's slots and one hardware barrier; slots alternate
// between two sets (a CTA can only be one exchange ahead of the slowest).
template <int CL, bool VEC, bool STORE>
__global__ void __launch_bounds__(REJ_THREADS, 2) rejection_walk_kernel(const RejectParams p, int slice, int run) {
    pdl_entry();
    __shared__ unsigned long long red[REJ_WARPS];
    __shared__ unsigned long long slots[2][CL];
    __shared__ int rejected[REJ_MAX_NODES];   // draft rows taken away from the weights at this node, in order
    __shared__ double rejected_R[REJ_MAX_NODES];
    const unsigned rank = CL == 1 ? 0u : cluster_cta_rank();
    const int seq = blockIdx.x / CL, N = p.rows.nodes, V = p.vocab, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int v1 = min(V, ((int)rank + 1) * slice);
    const int s0 = min(v1, (int)rank * slice + warp * run), s1 = min(v1, s0 + run);
    const int32_t * tokens = p.rows.tokens + (int64_t)seq * N;
    const int32_t * parent = p.rows.parent + (int64_t)seq * N;
    const float * U = p.u + (int64_t)seq * N * 2;
    const float * Q = p.q + (int64_t)seq * N * V;
    unsigned long long * r = STORE ? p.r + (int64_t)seq * V : nullptr;
    int32_t * path = p.out.path + (int64_t)seq * N;
    int32_t * emitted = p.out.emitted + (int64_t)seq * N;
    if constexpr (CL > 1) cluster_sync_all();  // every CTA of the cluster has started before another stores into it
    int turn = 0;
    // every warp's value (in all its lanes) -> red, every CTA's -> slots[turn ^ 1] after the return
    auto exchange = [&](unsigned long long v, bool is_max) {
        auto join = [&](unsigned long long x, unsigned long long y) {
            return is_max ? (unsigned long long)__float_as_uint(fmaxf(__uint_as_float((uint32_t)x), __uint_as_float((uint32_t)y))) : x + y;
        };
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = join(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) red[warp] = v;
        __syncthreads();
        if (warp == 0) {
            v = red[lane & (REJ_WARPS - 1)];
#pragma unroll
            for (int o = REJ_WARPS / 2; o > 0; o >>= 1) v = join(v, __shfl_xor_sync(0xffffffffu, v, o));
            if constexpr (CL == 1) {
                if (lane == 0) slots[turn][0] = v;
            } else {
                if (lane < CL) st_cluster_u64(&slots[turn][rank], (unsigned)lane, v);
            }
        }
        if constexpr (CL == 1) __syncthreads();
        else cluster_sync_all();
        turn ^= 1;
    };
    int cur = 0, a = 0;
    for (;;) {
        const float * L = p.logits + ((int64_t)seq * N + cur) * V;
        float mx = -INFINITY;
        for (int i0 = s0 + lane * 4; i0 < s1; i0 += 8 * 128) {
            float4 l[8];
#pragma unroll
            for (int u = 0; u < 8; u++) l[u] = load4<VEC>(L, i0 + u * 128, s1, -INFINITY);
#pragma unroll
            for (int u = 0; u < 8; u++) mx = fmaxf(mx, fmaxf(fmaxf(l[u].x, l[u].y), fmaxf(l[u].z, l[u].w)));
        }
        exchange((unsigned long long)__float_as_uint(mx), true);
#pragma unroll
        for (int c = 0; c < CL; c++) mx = fmaxf(mx, __uint_as_float((uint32_t)slots[turn ^ 1][c]));
        int n_rej = 0;
        bool stored = false;  // r holds the weights, and the list of rejected rows those that r does not know of yet
        // weights of tokens i .. i + 3, zero from `end` on
        auto weights_at4 = [&](int i, int end, unsigned long long (&w)[4]) {
            if (STORE && stored) {
#pragma unroll
                for (int e = 0; e < 4; e++) w[e] = i + e < end ? __ldcg(r + i + e) : 0ull;
            } else {
                const float4 l = load4<VEC>(L, i, end, -INFINITY);
                target_weights2(l.x, l.y, mx, p.inv_t, w[0], w[1]);
                target_weights2(l.z, l.w, mx, p.inv_t, w[2], w[3]);
            }
            for (int j = 0; j < n_rej; j++) {
                const float4 q = load4<VEC>(Q + (int64_t)rejected[j] * V, i, end, 0.0f);
                const double Rj = rejected_R[j];
                w[0] = take_away(w[0], q.x, Rj);
                w[1] = take_away(w[1], q.y, Rj);
                w[2] = take_away(w[2], q.z, Rj);
                w[3] = take_away(w[3], q.w, Rj);
            }
        };
        // sum of the weights of this warp's run
        auto run_sum = [&]() {
            unsigned long long sum = 0;
            if (STORE && stored) {  // and one row since
                const float * q = Q + (int64_t)rejected[0] * V;
                const double R0 = rejected_R[0];
                for (int i0 = s0 + lane; i0 < s1; i0 += 8 * 32) {
                    unsigned long long w[8];
                    float d[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int i = i0 + u * 32;
                        w[u] = i < s1 ? __ldcg(r + i) : 0ull;
                        d[u] = i < s1 ? q[i] : 0.0f;
                    }
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        w[u] = take_away(w[u], d[u], R0);
                        sum += w[u];
                        if (i0 + u * 32 < s1) __stcg(r + i0 + u * 32, w[u]);
                    }
                }
                return sum;
            }
            if (n_rej == 0) {
                for (int i0 = s0 + lane * 4; i0 < s1; i0 += 4 * 128) {
                    float4 l[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) l[u] = load4<VEC>(L, i0 + u * 128, s1, -INFINITY);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        unsigned long long w[4];
                        target_weights2(l[u].x, l[u].y, mx, p.inv_t, w[0], w[1]);
                        target_weights2(l[u].z, l[u].w, mx, p.inv_t, w[2], w[3]);
                        sum += (w[0] + w[1]) + (w[2] + w[3]);
                    }
                }
                return sum;
            }
            if (n_rej == 1) {  // (the usual case on its own: its row and its R stay in registers)
                const float * q = Q + (int64_t)rejected[0] * V;
                const double R0 = rejected_R[0];
                for (int i0 = s0 + lane * 4; i0 < s1; i0 += 4 * 128) {
                    float4 l[4], d[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        l[u] = load4<VEC>(L, i0 + u * 128, s1, -INFINITY);
                        d[u] = load4<VEC>(q, i0 + u * 128, s1, 0.0f);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        unsigned long long w0, w1;
                        target_weights2(l[u].x, l[u].y, mx, p.inv_t, w0, w1);
                        sum += take_away(w0, d[u].x, R0) + take_away(w1, d[u].y, R0);
                        target_weights2(l[u].z, l[u].w, mx, p.inv_t, w0, w1);
                        sum += take_away(w0, d[u].z, R0) + take_away(w1, d[u].w, R0);
                    }
                }
                return sum;
            }
            for (int i0 = s0 + lane * 4; i0 < s1; i0 += 128) {
                unsigned long long w[4];
                weights_at4(i0, s1, w);
                sum += (w[0] + w[1]) + (w[2] + w[3]);
                if (STORE) {
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (i0 + e < s1) __stcg(r + i0 + e, w[e]);
                }
            }
            return sum;
        };
        auto weight_at = [&](int x) {
            unsigned long long w, unused;
            if (STORE && stored) w = __ldcg(r + x);  // (another CTA's, perhaps: an exchange lies between)
            else target_weights2(L[x], mx, mx, p.inv_t, w, unused);
            for (int j = 0; j < n_rej; j++) w = take_away(w, Q[(int64_t)rejected[j] * V + x], rejected_R[j]);
            return w;
        };
        unsigned long long below, mine;
        auto total = [&]() {
            unsigned long long tot = 0;
            below = 0;
#pragma unroll
            for (int c = 0; c < CL; c++) {
                const unsigned long long x = slots[turn ^ 1][c];
                if (c < (int)rank) below += x;
                if (c == (int)rank) mine = x;
                tot += x;
            }
            return tot;
        };
        exchange(run_sum(), false);
        unsigned long long R = total();
        int next = -1;
        for (int c = cur + 1; c < N; c++) {
            if (parent[c] != cur) continue;
            const int32_t x = tokens[c];
            // (every thread of every CTA works this out for itself: no exchange)
            if (__dmul_rn((double)__fmul_rn(U[2 * c], Q[(int64_t)c * V + x]), (double)R) <= (double)weight_at(x)) {
                next = c;
                break;
            }
            if (STORE && CL > 1 && stored) cluster_sync_all();  // every CTA has read r[x], which its owner is about to replace
            else __syncthreads();                      // the list may still be in use
            if (tid == 0) {
                rejected[n_rej] = c;
                rejected_R[n_rej] = (double)R;
            }
            n_rej++;
            __syncthreads();
            exchange(run_sum(), false);
            R = total();
            if (STORE && n_rej >= (stored ? 1 : REJ_KEEP)) {
                stored = true;
                n_rej = 0;
            }
            if (R == 0) {  // nothing is left: the target's own weights again
                stored = false;
                n_rej = 0;
                exchange(run_sum(), false);
                R = total();
            }
        }
        if (next >= 0) {
            if (tid == 0 && rank == 0) {
                emitted[a] = tokens[next];
                path[a] = next;
            }
            a++;
            cur = next;
            continue;
        }
        // residual draw: the smallest j whose inclusive prefix sum over r exceeds t, by the warp whose run holds it
        unsigned long long t = (unsigned long long)__dmul_rn((double)U[2 * cur + 1], (double)R);
        if (t >= R) t = R - 1;
        if (t < below || t - below >= mine) break;  // (no exchange follows: every CTA may leave)
        t -= below;
        int owner = 0;
        unsigned long long before = 0;
        while (t - before >= red[owner]) before += red[owner++];
        t -= before;
        // the CTA shares out that warp's run, a few consecutive tokens to a thread: which thread's, then which token
        const int r0 = min(v1, (int)rank * slice + owner * run), r1 = min(v1, r0 + run);
        const int part = ((run + REJ_THREADS - 1) / REJ_THREADS + 3) & ~3;
        const int p0 = min(r1, r0 + tid * part), p1 = min(r1, p0 + part);
        unsigned long long own = 0;
        for (int i = p0; i < p1; i += 4) {
            unsigned long long w[4];
            weights_at4(i, p1, w);
            own += (w[0] + w[1]) + (w[2] + w[3]);
        }
        unsigned long long incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        __syncthreads();  // red has been read
        if (lane == 31) red[warp] = incl;
        __syncthreads();
        for (int w = 0; w < warp; w++) incl += red[w];
        if (incl - own <= t && t < incl) {  // exactly one thread: t is below the run's total
            unsigned long long acc = incl - own;
            for (int i = p0; i < p1; i += 4) {
                unsigned long long w[4];
                weights_at4(i, p1, w);
                int e = 0;
                for (; e < 4 && acc + w[e] <= t; e++) acc += w[e];
                if (e < 4) {
                    emitted[a] = i + e;
                    break;
                }
            }
        }
        break;
    }
    if (rank == 0) {
        for (int i = a + tid; i < N; i += REJ_THREADS) path[i] = -1;
        for (int i = a + 1 + tid; i < N; i += REJ_THREADS) emitted[i] = -1;
        if (tid == 0) p.out.accepted[seq] = a;
    }
}

// CTAs per sequence: as many as let all sequences run at once (two CTAs on each SM), as long as a CTA keeps
// at least 4,096 tokens (two loads per thread and pass; below that the exchanges cost more than the passes they cut).
static int rejection_cluster(int sms, int batch, int vocab) {
    int cl = REJ_MAX_CLUSTER;
    while (cl > 1 && (batch * cl > 2 * sms || vocab < cl * 4096)) cl >>= 1;
    return cl;
}

template <int CL>
static void launch_rejection(cudaStream_t s, const RejectParams & p) {
    const int slice = ((p.vocab + CL - 1) / CL + 3) & ~3, run = ((slice + REJ_WARPS - 1) / REJ_WARPS + 3) & ~3;
    const bool vec = (p.vocab & 3) == 0 && (((uintptr_t)p.logits | (uintptr_t)p.q) & 15) == 0;
    auto kern = p.r ? (vec ? rejection_walk_kernel<CL, true, true> : rejection_walk_kernel<CL, false, true>)
                    : (vec ? rejection_walk_kernel<CL, true, false> : rejection_walk_kernel<CL, false, false>);
    if (CL > 1) launch_k_cluster(kern, dim3(p.rows.batch * CL), REJ_THREADS, 0, s, CL, p, slice, run);
    else launch_k(kern, p.rows.batch, REJ_THREADS, 0, s, p, slice, run);
}

int rejection_siblings(const int32_t * parent, int batch, int nodes) {
    int most = 1;
    for (int b = 0; parent && b < batch; b++) {
        int children[REJ_MAX_NODES] = {};
        for (int i = 1; i < nodes; i++) most = std::max(most, ++children[parent[b * nodes + i]]);
    }
    return most;
}

int launch_accept_rejection(cudaStream_t s, int sms, const float * logits, const float * draft_probs, const float * uniforms, unsigned long long * residual,
                            int vocab, float temperature, const RowMeta & rows, const AcceptOut & out) {
    YK_REQUIRE(temperature > 0.0f, YUUKA_ERR_INVALID_ARGUMENT, "rejection sampling needs a temperature above zero");
    YK_REQUIRE(rows.nodes <= REJ_MAX_NODES, YUUKA_ERR_UNSUPPORTED, "rejection sampling: at most %d rows per sequence", REJ_MAX_NODES);
    RejectParams p{logits, draft_probs, uniforms, residual, vocab, 1.0f / temperature, rows, out};
    switch (rejection_cluster(sms, rows.batch, vocab)) {
    case 8: launch_rejection<8>(s, p); break;
    case 4: launch_rejection<4>(s, p); break;
    case 2: launch_rejection<2>(s, p); break;
    default: launch_rejection<1>(s, p); break;
    }
    YK_CUDA(cudaGetLastError());
    return 1;
}

__global__ void accept_all_kernel(RowMeta rows, AcceptOut out) {
    pdl_entry();
    const int seq = blockIdx.x, N = rows.nodes;
    if (threadIdx.x == 0) out.accepted[seq] = N - 1;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        out.path[(int64_t)seq * N + i] = i + 1 < N ? i + 1 : -1;
        out.emitted[(int64_t)seq * N + i] = i + 1 < N ? rows.tokens[(int64_t)seq * N + i + 1] : -1;
    }
}

void launch_accept_all(cudaStream_t s, const RowMeta & rows, const AcceptOut & out) {
    launch_k(accept_all_kernel, rows.batch, 64, 0, s, rows, out);
    YK_CUDA(cudaGetLastError());
}

int argmax_chunks(int vocab) { return (vocab + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK; }

}  // namespace yk

// ---------------------------------------------------------------------------
// Kernel-level entry point: acceptance over logits that are already on the device (the acceptance case of the
// kernel microbenchmark; hosts whose logits come from elsewhere). Row metadata and scratch live for the call.
extern "C" yuuka_status yuuka_accept_tree(yuuka_stream * stream, const yuuka_buffer * logits, int32_t batch, int32_t nodes,
                                          int32_t vocab, const int32_t * tokens, const int32_t * parent, uint32_t mode,
                                          float temperature, const yuuka_buffer * draft_probs, const float * uniforms,
                                          int32_t * accepted, int32_t * emitted, int32_t * path, yuuka_event * begin,
                                          yuuka_event * end) {
    using namespace yk;
    return guard([&] {
        YK_REQUIRE(stream && logits && tokens && accepted && emitted, YUUKA_ERR_INVALID_ARGUMENT, "accept_tree: null argument");
        YK_REQUIRE(batch > 0 && nodes > 0 && nodes <= 64 && vocab > 0, YUUKA_ERR_INVALID_ARGUMENT, "accept_tree: invalid shape");
        YK_REQUIRE(mode == YUUKA_ACCEPT_GREEDY || mode == YUUKA_ACCEPT_REJECTION, YUUKA_ERR_INVALID_ARGUMENT,
                   "accept_tree: unknown acceptance mode %u", mode);
        const uint64_t R = (uint64_t)batch * nodes, need = R * (uint64_t)vocab * sizeof(float);
        YK_REQUIRE(logits->bytes >= need, YUUKA_ERR_INVALID_ARGUMENT, "accept_tree: logits buffer holds fewer than %llu bytes",
                   (unsigned long long)need);
        if (mode == YUUKA_ACCEPT_REJECTION) {
            YK_REQUIRE(temperature > 0.0f && temperature == temperature, YUUKA_ERR_INVALID_ARGUMENT,
                       "accept_tree: rejection sampling needs a temperature above zero");
            YK_REQUIRE(uniforms && draft_probs && draft_probs->bytes >= need, YUUKA_ERR_INVALID_ARGUMENT,
                       "accept_tree: rejection sampling needs uniforms and a draft_probs buffer of %llu bytes", (unsigned long long)need);
            for (uint64_t i = 0; i < R * 2; i++)
                YK_REQUIRE(uniforms[i] >= 0.0f && uniforms[i] < 1.0f, YUUKA_ERR_INVALID_ARGUMENT,
                           "accept_tree: uniform draw %llu is outside [0, 1)", (unsigned long long)i);
        }
        // row metadata on the host
        std::vector<int32_t> par(R), dep(R);
        std::vector<unsigned long long> anc(R);
        for (int b = 0; b < batch; b++)
            for (int i = 0; i < nodes; i++) {
                const size_t r = (size_t)b * nodes + i;
                YK_REQUIRE(tokens[r] >= 0 && tokens[r] < vocab, YUUKA_ERR_INVALID_ARGUMENT, "token id %d is out of range", tokens[r]);
                const int p = parent ? parent[r] : i - 1;
                YK_REQUIRE((i == 0 && p == -1) || (i > 0 && p >= 0 && p < i), YUUKA_ERR_INVALID_ARGUMENT,
                           "parent[%d][%d] = %d is not a preceding row", b, i, p);
                par[r] = p;
                dep[r] = i == 0 ? 0 : dep[(size_t)b * nodes + p] + 1;
                anc[r] = (i == 0 ? 0ull : anc[(size_t)b * nodes + p]) | (1ull << i);
            }
        set_device(stream->dev);
        const int chunks = argmax_chunks(vocab);
        const bool reject = mode == YUUKA_ACCEPT_REJECTION;
        // inputs, filled by one copy: anc | uniforms | tokens | parent | depth; results, read by one copy: accepted |
        // path | emitted; then scratch: argmax val, idx or the residual weights
        const size_t o_anc = 0, o_uni = o_anc + R * 8, o_tok = o_uni + (reject ? R * 8 : 0), o_par = o_tok + R * 4, o_dep = o_par + R * 4,
                     o_acc = o_dep + R * 4, o_path = o_acc + (size_t)batch * 4, o_em = o_path + R * 4, staged = o_em + R * 4,
                     o_val = (staged + 255) / 256 * 256, o_idx = o_val + (reject ? 0 : R * chunks * 4), weights = (size_t)batch * vocab * 8;
        // (weights beyond what the stream's scratch keeps cost an allocation, about what 16 rejected siblings cost without them)
        const int siblings = reject ? rejection_siblings(parent, batch, nodes) : 0;
        const bool stores = siblings >= REJ_STORE_SIBLINGS && (o_val + weights <= StreamScratch::KEEP || siblings > 16);
        const size_t total = o_idx + (reject ? (stores ? weights : 0) : R * chunks * 4);
        std::lock_guard<std::mutex> lock(stream->scratch.mutex);
        StreamScratchUse use(stream->scratch, total, staged);
        uint8_t * d = use.device, * h = use.host;
        memcpy(h + o_anc, anc.data(), R * 8);
        memcpy(h + o_tok, tokens, R * 4);
        memcpy(h + o_par, par.data(), R * 4);
        memcpy(h + o_dep, dep.data(), R * 4);
        if (reject) memcpy(h + o_uni, uniforms, R * 8);
        cudaStream_t st = stream->s;
        YK_CUDA(cudaMemcpyAsync(d, h, o_acc, cudaMemcpyHostToDevice, st));
        RowMeta rows{(const int32_t *)(d + o_tok), (const int32_t *)(d + o_par), (const int32_t *)(d + o_dep),
                     (const uint64_t *)(d + o_anc), nullptr, batch, nodes};
        AcceptOut out{(int32_t *)(d + o_acc), (int32_t *)(d + o_path), (int32_t *)(d + o_em)};
        if (begin) YK_CUDA(cudaEventRecord(begin->e, st));
        if (!reject) {
            ArgmaxScratch sc{(float *)(d + o_val), (int32_t *)(d + o_idx), chunks};
            launch_accept_greedy(st, (const float *)logits->ptr, vocab, rows, sc, out);
        } else {
            launch_accept_rejection(st, stream->dev->sm_count, (const float *)logits->ptr, (const float *)draft_probs->ptr, (const float *)(d + o_uni),
                                    stores ? (unsigned long long *)(d + o_val) : nullptr, vocab, temperature, rows, out);
        }
        if (end) YK_CUDA(cudaEventRecord(end->e, st));
        YK_CUDA(cudaMemcpyAsync(h + o_acc, d + o_acc, staged - o_acc, cudaMemcpyDeviceToHost, st));
        YK_CUDA(cudaStreamSynchronize(st));
        memcpy(accepted, h + o_acc, (size_t)batch * 4);
        memcpy(emitted, h + o_em, R * 4);
        if (path) memcpy(path, h + o_path, R * 4);
    });
}
