// Gated DeltaNet over the rows of a verify step, with rollback by delta log.
//
// The scan never writes the recurrent state. For every row it emits what the
// state update needs -- the normalised key, d = beta * (v - S^T k) and the decay
// exp(alpha) -- and the commit kernel applies exactly the accepted rows'
// rank-one updates to the stored state. Rejected rows therefore cost nothing
// and no per-position copy of the 2 MiB/layer state is made.
//
// Math follows forwardRecurrent (model/qwen35/forward.go:245-287) and
// gdnPerTokenScan (model/qwen35/recurrent.go:56-105). Replaces
// conv1d_chunk / gdn_prepare_splitreg / gdn_chunk_prepared of the reference
// (kernels/hip/prefill/prefill.hip:274-521).
#include <cstdlib>

#include "layers.cuh"
#include "xprep.cuh"

namespace yk {

constexpr int GDN_COLS = 32;   // state columns per CTA
constexpr int GDN_WARPS = 4;   // each owns 8 of the 32 columns
constexpr int GDN_MAX_NODES = 64;

// float exp: the CPU reference evaluates exp in f64 and rounds; the difference is below 2e-7 relative
__device__ __forceinline__ float sigmoid_ref(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_ref(float x) { return x * sigmoid_ref(x); }
__device__ __forceinline__ float softplus_ref(float x) {
    if (x > 20.0f) return x;
    return log1pf(expf(x));
}

// One state update, the same expression in the scan and in the commit so both
// produce identical bits: S <- S * decay + k * d.
__device__ __forceinline__ float state_update(float s, float decay, float k, float d) {
    return fmaf(k, d, s * decay);
}

// Two fp32 lanes per instruction (fma.rn.f32x2 / mul.rn.f32x2): the same IEEE results as the scalar forms, half the
// instructions. The recurrence keeps its state, keys and queries as such pairs.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)),
          "l"(*reinterpret_cast<const unsigned long long *>(&c)));
    return *reinterpret_cast<const float2 *>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)));
    return *reinterpret_cast<const float2 *>(&d);
}
// state_update on a pair: S <- S * decay + k * d
__device__ __forceinline__ float2 state_update2(float2 s, float2 decay, float2 k, float2 d) { return fma2(k, d, mul2(s, decay)); }

struct ScanParams {
    GdnArgs a;
    RowMeta rows;
    int chain;       // front end only: the rows are chains (row i follows row i - 1), however many there are
    int block_rows;  // front end only: rows of a sequence per CTA
};

// ---------------------------------------------------------------------------
// Front end, parallel over (row, S-channel unit): depthwise causal conv over the row's ancestors and the stored
// history + SiLU (forward.go:253-268), L2 norm of the q and k units (forward.go:275-279, 484-493), beta = sigmoid,
// decay = exp(softplus(alpha + dt) * a) (forward.go:245-248).
// grid (2*groups + rank, row blocks, batch). A warp owns a row of a unit outright, S / 32 channels per lane: every tap of
// a row is in flight at once, the sums of squares close by shuffles (as many independent chains as channels), nothing
// meets at a barrier, and a warp goes on to its next row with its weights in registers. It is latency that bounds this
// kernel: one CTA per (row, unit) spent 39 us on 512 rows of 8192 channels (15 waves of CTAs, each a chain of waits)
// where its 40 MB take 6.
// KMAX: taps held in registers (4, or 8 for the longer kernels). SPLIT: a CTA of S / 32 warps per row, 32 channels each
// (few rows: the chain of a warp is shorter. With a warp per row a 9-row step of 24 such layers took 16 us more).
template <int S, int KMAX, bool SPLIT>
__global__ void __launch_bounds__(128) gdn_front_kernel(const ScanParams p) {
    // (releasing the scan from here, so that it could fetch its state while this kernel runs, measured 7 us
    // slower per layer: a dependent grid that starts early and really has to block in griddepcontrol.wait
    // is woken late; only triggers placed at the end of a kernel have paid)
    const GdnArgs & a = p.a;
    constexpr int G = SPLIT ? 1 : S / 32;
    const int N = p.rows.nodes, K = a.kernel, K1 = K - 1;
    const int u = blockIdx.x, seq = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int key_dim = a.groups * S, conv_dim = 2 * key_dim + a.rank * S;
    const int e0 = (SPLIT ? warp * 32 : 0) + lane;
    const int c0 = u * S + e0;  // q units, then k units, then v units: exactly the conv row order
    float w[G][KMAX];
#pragma unroll
    for (int i = 0; i < G; i++)
#pragma unroll
        for (int t = 0; t < KMAX; t++) w[i][t] = t < K ? a.conv_w[(int64_t)(c0 + 32 * i) * K + t] : 0.0f;
    int par0 = -1, par1 = -1;  // parents of rows lane and lane + 32
    if (!p.chain) {
        if (lane < N) par0 = p.rows.parent[seq * N + lane];
        if (lane + 32 < N) par1 = p.rows.parent[seq * N + lane + 32];
    }
    pdl_entry();
    const float * proj = a.proj + (int64_t)seq * N * a.ldp;
    const float * hist = a.conv_state + ((int64_t)seq_of(p.rows, seq) * conv_dim + c0) * K1;
    const int first = blockIdx.y * p.block_rows, last = min(N, first + p.block_rows);
    for (int node = first + (SPLIT ? 0 : warp); node < last; node += (SPLIT ? 1 : 4)) {
        const int r = seq * N + node;
        float taps[G][KMAX];
        int cur = node, hidx = K1 - 1;
#pragma unroll
        for (int t = KMAX - 1; t >= 0; t--) {
            if (t < K) {
                const float * src = cur >= 0 ? proj + (int64_t)cur * a.ldp + c0 : hist + hidx;
                const int stride = cur >= 0 ? 32 : 32 * K1;
#pragma unroll
                for (int i = 0; i < G; i++) taps[i][t] = src[i * stride];
                if (cur < 0) hidx--;
                else if (p.chain) cur--;
                else cur = __shfl_sync(0xffffffffu, cur < 32 ? par0 : par1, cur & 31);
            }
        }
        float v[G];
#pragma unroll
        for (int i = 0; i < G; i++) {
            float sum = 0.0f;
#pragma unroll
            for (int t = 0; t < KMAX; t++)
                if (t < K) sum += w[i][t] * taps[i][t];
            v[i] = silu_ref(sum);
        }
        if (u < 2 * a.groups) {
            double sq[G];
#pragma unroll
            for (int i = 0; i < G; i++) sq[i] = (double)v[i] * (double)v[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < G; i++) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
            double tot = 0;
            if constexpr (SPLIT) {
                __shared__ double red[S / 32];  // (one row per CTA)
                if (lane == 0) red[warp] = sq[0];
                __syncthreads();
#pragma unroll
                for (int i = 0; i < S / 32; i++) tot += red[i];
            } else {
#pragma unroll
                for (int i = 0; i < G; i++) tot += sq[i];
            }
            const float scale = (float)(1.0 / sqrt(tot + (double)a.eps));
            const bool is_q = u < a.groups;
            const float mul = is_q ? scale * (float)(1.0 / sqrt((double)S)) : scale;
            float * dst = (is_q ? a.qn + u * S : a.khat + (u - a.groups) * S) + (int64_t)r * key_dim + e0;
#pragma unroll
            for (int i = 0; i < G; i++) dst[32 * i] = v[i] * mul;
        } else {
            const int h = u - 2 * a.groups;
            float * dst = a.vconv + (int64_t)r * (a.rank * S) + h * S + e0;
#pragma unroll
            for (int i = 0; i < G; i++) dst[32 * i] = v[i];
            if (e0 == 0) {
                const float * row = a.proj + (int64_t)r * a.ldp;
                a.beta[(int64_t)r * a.rank + h] = sigmoid_ref(row[conv_dim + a.rank * S + h]);
                a.decay[(int64_t)r * a.rank + h] = expf(softplus_ref(row[conv_dim + a.rank * S + a.rank + h] + a.dt[h]) * a.a[h]);
            }
        }
    }
}

// One row per CTA while that is a resident wave of warps or less (24 per SM); beyond that one row per warp, and then as
// many rows per warp as keep the launch at one wave.
template <int S>
static void launch_gdn_front_s(cudaStream_t s, ScanParams & p) {
    const GdnArgs & a = p.a;
    const int units = 2 * a.groups + a.rank, N = p.rows.nodes;
    const int64_t wave = (int64_t)a.sms * 24;
    const int64_t unit_rows = (int64_t)units * N * p.rows.batch;
    if (unit_rows * (S / 32) <= wave) {
        p.block_rows = 1;
        launch_k(a.kernel <= 4 ? gdn_front_kernel<S, 4, true> : gdn_front_kernel<S, 8, true>, dim3(units, N, p.rows.batch), S, 0, s, p);
    } else {
        const int64_t per_warp = (unit_rows + wave - 1) / wave;
        const int blocks = (int)((N + 4 * per_warp - 1) / (4 * per_warp));
        p.block_rows = (N + blocks - 1) / blocks;
        launch_k(a.kernel <= 4 ? gdn_front_kernel<S, 4, false> : gdn_front_kernel<S, 8, false>,
                 dim3(units, (N + p.block_rows - 1) / p.block_rows, p.rows.batch), 128, 0, s, p);
    }
    YK_CUDA(cudaGetLastError());
}
static void launch_gdn_front(cudaStream_t s, const GdnArgs & a, const RowMeta & rows, bool chain) {
    YK_REQUIRE(a.kernel >= 2 && a.kernel <= 8, YUUKA_ERR_UNSUPPORTED, "gdn: conv kernel %d is outside 2..8", a.kernel);
    YK_REQUIRE(a.S == 64 || a.S == 128, YUUKA_ERR_UNSUPPORTED, "gdn: state size %d is not 64 or 128", a.S);
    ScanParams p{a, rows, chain ? 1 : 0, 0};
    if (a.S == 128) launch_gdn_front_s<128>(s, p);
    else launch_gdn_front_s<64>(s, p);
}

// ---------------------------------------------------------------------------
// Recurrence (recurrent.go:56-105) + gated RMSNorm (recurrent.go:39-50).
// grid (S/32 column blocks, rank, batch), the column blocks of a head forming one thread-block
// cluster; 4 warps. A warp owns 8 state columns outright: lane = (row quarter, column), S/4 state
// rows per lane in registers, and the two sums over the state rows close with two shuffles, so the
// rows of a step are walked without a CTA-wide barrier (an earlier form split the state rows over
// the warps and met at two barriers per row: 1 us more per layer). For the gated norm the column
// blocks exchange their sums of squares through distributed shared memory, and each finishes its
// own columns and emits them as f32 and in the prepared form the out-projection GEMM reads.
// Redoing the front end inside this kernel (every CTA its head's q and k group and its own v
// columns) to save the launch in between measured 9 us slower per layer: the front end is only
// cheap when spread over its 576 CTAs.
// TREE: the rows of a sequence may branch (the host staged parent pointers); they are then walked depth first.
template <int S, bool TREE>
__global__ void __launch_bounds__(GDN_WARPS * 32) gdn_scan_kernel(const ScanParams p) {
    pdl_entry();
    constexpr int RPL = S / 4;  // state rows per lane
    const GdnArgs & a = p.a;
    const int cb = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
    const int N = p.rows.nodes;
    const int kh = h % a.groups;
    const int key_dim = a.groups * S, inner = a.rank * S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rq = lane >> 3, cl = warp * 8 + (lane & 7);  // row quarter; column within the block
    const int col = cb * GDN_COLS + cl;

    extern __shared__ __align__(16) float sm[];
    // q and k rows are stored quarter by quarter with four words of padding after each (QP words per quarter): the
    // four row quarters of a warp read their 16-byte pieces from distinct banks (dense rows put all four on the
    // same ones: more bank conflicts than loads in the profile of the batched step)
    constexpr int QP = RPL + 4, SP4 = 4 * QP;
    float * qn = sm;                      // [N][4][QP]
    float * kn = qn + N * SP4;            // [N][4][QP]
    float * vv = kn + N * SP4;            // [N][GDN_COLS]
    float * dd = vv + N * GDN_COLS;       // [N][GDN_COLS]
    float * o_s = dd + N * GDN_COLS;      // [N][GDN_COLS] outputs of this column block
    float * dec = o_s + N * GDN_COLS;     // [N]
    float * bet = dec + N;                // [N]
    int * par = reinterpret_cast<int *>(bet + N);  // [N]
    // TREE: [S / 8][threads] pairs, the state after row 0 (8-byte aligned: the arrays before it hold 2 N (S + 16) + 99 N words)
    float * root_s = reinterpret_cast<float *>(par + N + (N & 1));
    __shared__ double ssq[GDN_MAX_NODES];
    __shared__ float scale_s[GDN_MAX_NODES];
    __shared__ int order_s[TREE ? GDN_MAX_NODES : 1];  // the rows depth first, worked out by the host when it staged the step

    // stored state: the longest fetch (HBM), issued first
    const float * s0 = a.state + ((int64_t)(seq_of(p.rows, seq) * a.rank + h) * S + rq * RPL) * S + col;
    float2 st[RPL / 2];  // state rows (2 i, 2 i + 1) of this lane's quarter, one column
#pragma unroll
    for (int i = 0; i < RPL / 2; i++) st[i] = make_float2(s0[(int64_t)(2 * i) * S], s0[(int64_t)(2 * i + 1) * S]);

    // the front-end kernel has left normalised q and k, the conv output of v, beta and decay in global memory
    // (16-byte loads, eight in flight per thread: with 64 rows of a prompt sub-chunk a scalar loop spent most
    // of the kernel waiting for one L2 round trip after another)
    constexpr int SQ = S / 4;
#pragma unroll 8
    for (int i = threadIdx.x; i < N * SQ; i += blockDim.x) {
        const int node = i / SQ, e4 = i - node * SQ;
        const int64_t at = (int64_t)(seq * N + node) * key_dim + kh * S + e4 * 4;
        const int spot = node * SP4 + (e4 / (RPL / 4)) * QP + (e4 % (RPL / 4)) * 4;
        *reinterpret_cast<float4 *>(qn + spot) = *reinterpret_cast<const float4 *>(a.qn + at);
        *reinterpret_cast<float4 *>(kn + spot) = *reinterpret_cast<const float4 *>(a.khat + at);
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < N * (GDN_COLS / 4); i += blockDim.x) {
        const int node = i / (GDN_COLS / 4), e4 = i - node * (GDN_COLS / 4);
        reinterpret_cast<float4 *>(vv)[i] =
            *reinterpret_cast<const float4 *>(a.vconv + (int64_t)(seq * N + node) * inner + h * S + cb * GDN_COLS + e4 * 4);
    }
    for (int node = threadIdx.x; node < N; node += blockDim.x) {
        par[node] = p.rows.parent[seq * N + node];
        bet[node] = a.beta[(int64_t)(seq * N + node) * a.rank + h];
        dec[node] = a.decay[(int64_t)(seq * N + node) * a.rank + h];
        if (TREE) order_s[node] = p.rows.order[seq * N + node];
    }
    __syncthreads();

    // gate values the last phase needs, up to ZPT per thread. The first three (a 9-row step needs 2.25) are fetched now, so
    // that the end of the kernel does not wait for them; a tree needs the registers
    constexpr int ZPT = GDN_MAX_NODES * GDN_COLS / (GDN_WARPS * 32), ZPRE = TREE ? 0 : 3;
    float z[ZPT];
    auto fetch_z = [&](int k) {
        const int i = threadIdx.x + k * (GDN_WARPS * 32);
        const int node = i / GDN_COLS, c = i - node * GDN_COLS;
        z[k] = i < N * GDN_COLS ? a.z[(int64_t)(seq * N + node) * a.ldz + h * S + cb * GDN_COLS + c] : 0.0f;
    };
#pragma unroll
    for (int k = 0; k < ZPRE; k++) fetch_z(k);

    // The rows are walked in depth-first order: a row then follows its parent directly unless it is a later
    // sibling, so a branch is replayed from the stored state only when the walk backtracks. In row order
    // (breadth first, as draft trees are numbered) almost every row of a tree switched branches: the 16-node
    // tree of the batched configuration cost 24 replayed updates on top of its 16, depth first it costs 2. (The order is
    // an input: one thread of every CTA working it out, its path kept in local memory, cost 56 us of a layer's 239 at
    // 32 sequences x 17 rows.)

    // ---- recurrence (recurrent.go:56-105) ----
    int cur = -1;  // node whose state st currently holds (-1: the stored state)
    for (int step = 0; step < N; step++) {
        const int node = TREE ? order_s[step] : step;
        const int pnode = par[node];
        if (pnode != cur) {
            // a sibling branch: rebuild the parent's state by replaying the log of its path, from the state after row 0
            // (every row of a step descends from row 0, the pending token; a tree keeps that state in shared memory)
            // or, failing that, from the stored one
            const int stop = TREE && pnode >= 0 ? 0 : -1;  // the row whose state the replay starts from
            int len = 0;
            for (int c = pnode; c > stop; c = par[c]) len++;
            if (TREE && pnode >= 0) {
#pragma unroll
                for (int i = 0; i < RPL / 2; i++) st[i] = reinterpret_cast<const float2 *>(root_s)[i * (GDN_WARPS * 32) + threadIdx.x];
            } else {
#pragma unroll
                for (int i = 0; i < RPL / 2; i++) st[i] = make_float2(s0[(int64_t)(2 * i) * S], s0[(int64_t)(2 * i + 1) * S]);
            }
            for (int j = len - 1; j >= 0; j--) {
                int c = pnode;
                for (int up = 0; up < j; up++) c = par[c];
                const float dc = dec[c], dv = dd[c * GDN_COLS + cl];
                const float2 dc2 = make_float2(dc, dc), dv2 = make_float2(dv, dv);
#pragma unroll
                for (int i = 0; i < RPL / 2; i++)
                    st[i] = state_update2(st[i], dc2, *reinterpret_cast<const float2 *>(kn + c * SP4 + rq * QP + 2 * i), dv2);
            }
        }
        // this lane's S/4 key and query values, fetched as float4 (a quarter of the shared-memory loads)
        float2 kx[RPL / 2], qx[RPL / 2];
#pragma unroll
        for (int i = 0; i < RPL; i += 4) {
            const float4 k4 = *reinterpret_cast<const float4 *>(kn + node * SP4 + rq * QP + i);
            const float4 q4 = *reinterpret_cast<const float4 *>(qn + node * SP4 + rq * QP + i);
            kx[i / 2] = make_float2(k4.x, k4.y); kx[i / 2 + 1] = make_float2(k4.z, k4.w);
            qx[i / 2] = make_float2(q4.x, q4.y); qx[i / 2 + 1] = make_float2(q4.z, q4.w);
        }
        const float dc = dec[node];
        const float2 dc2 = make_float2(dc, dc);
        // sk = (decay * S)^T k over this lane's rows (four partial sums: rows i mod 4), then over the four row quarters
        float2 sd[RPL / 2], sk01 = make_float2(0.0f, 0.0f), sk23 = sk01;
#pragma unroll
        for (int i = 0; i < RPL / 2; i++) {
            sd[i] = mul2(st[i], dc2);
            if (i & 1) sk23 = fma2(sd[i], kx[i], sk23);
            else sk01 = fma2(sd[i], kx[i], sk01);
        }
        float sk = (sk01.x + sk01.y) + (sk23.x + sk23.y);
        sk += __shfl_xor_sync(0xffffffffu, sk, 8);
        sk += __shfl_xor_sync(0xffffffffu, sk, 16);
        const float d = (vv[node * GDN_COLS + cl] - sk) * bet[node];
        const float2 d2 = make_float2(d, d);
        float2 o01 = make_float2(0.0f, 0.0f), o23 = o01;
#pragma unroll
        for (int i = 0; i < RPL / 2; i++) {
            st[i] = fma2(kx[i], d2, sd[i]);  // state_update with the product S * decay already at hand
            if (i & 1) o23 = fma2(st[i], qx[i], o23);
            else o01 = fma2(st[i], qx[i], o01);
        }
        float o = (o01.x + o01.y) + (o23.x + o23.y);
        o += __shfl_xor_sync(0xffffffffu, o, 8);
        o += __shfl_xor_sync(0xffffffffu, o, 16);
        if (rq == 0) {
            o_s[node * GDN_COLS + cl] = o;
            dd[node * GDN_COLS + cl] = d;
            a.dlog[(int64_t)(seq * N + node) * inner + h * S + col] = d;
        }
        if (TREE && node == 0) {
#pragma unroll
            for (int i = 0; i < RPL / 2; i++) reinterpret_cast<float2 *>(root_s)[i * (GDN_WARPS * 32) + threadIdx.x] = st[i];
        }
        __syncwarp();  // dd of this row is read by the other row quarters when a later branch replays it
        cur = node;
    }

    pdl_trigger_late();
    // ---- gated RMSNorm of the head (recurrent.go:39-50), sums of squares exchanged across the cluster ----
    // (the other gate values are fetched now, into the registers the state has left: the exchanges hide their latency)
#pragma unroll
    for (int k = ZPRE; k < ZPT; k++) fetch_z(k);
    const float norm_w = a.norm[cb * GDN_COLS + (threadIdx.x & (GDN_COLS - 1))];
    const bool hi_only = a.prep.hi_only();  // the out projection of a wide step reads nothing else
    __syncthreads();
    for (int node = warp; node < N; node += GDN_WARPS) {
        const double v = (double)o_s[node * GDN_COLS + lane];
        double sq = v * v;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) ssq[node] = sq;
    }
    cluster_sync_all();
    for (int node = threadIdx.x; node < N; node += blockDim.x) {
        double tot = 0;
        for (unsigned r = 0; r < gridDim.x; r++) tot += ld_cluster_f64(ssq + node, r);  // the cluster spans gridDim.x
        const float mean = (float)(tot / (double)S);
        scale_s[node] = (float)(1.0 / sqrt((double)(mean + a.eps)));
    }
    cluster_sync_all();  // scales visible to the CTA; no CTA leaves while another may still read its sums
#pragma unroll
    for (int k = 0; k < ZPT; k++) {
        const int i = threadIdx.x + k * (GDN_WARPS * 32);
        if (i < N * GDN_COLS) {
            float t = o_s[i];
            t *= scale_s[i / GDN_COLS] * norm_w;
            t *= silu_ref(z[k]);
            if (hi_only) a.prep.xh[(int64_t)(seq * N + i / GDN_COLS) * inner + h * S + cb * GDN_COLS + (i & (GDN_COLS - 1))] = __float2half_rn(t);
            else o_s[i] = t;
        }
    }
    if (hi_only) return;
    __syncthreads();
    for (int gi = threadIdx.x; gi < N * (GDN_COLS >> 4); gi += blockDim.x) {
        const int node = gi / (GDN_COLS >> 4), part = gi - node * (GDN_COLS >> 4);
        const int64_t r = seq * N + node;
        const int c0 = h * S + cb * GDN_COLS + part * 16;
        float g16[16];
#pragma unroll
        for (int i = 0; i < 16; i++) g16[i] = o_s[node * GDN_COLS + part * 16 + i];
        float4 * dst = reinterpret_cast<float4 *>(a.out + r * inner + c0);
#pragma unroll
        for (int i = 0; i < 4; i++) dst[i] = make_float4(g16[4 * i], g16[4 * i + 1], g16[4 * i + 2], g16[4 * i + 3]);
        if (a.prep.xh) xprep_store16(a.prep.xh + r * inner + c0, a.prep.xl + r * inner + c0, a.prep.xs16 + r * (inner >> 4) + (c0 >> 4), g16);
    }
}

int launch_gdn_scan(cudaStream_t s, const GdnArgs & a, const RowMeta & rows) {
    YK_REQUIRE(rows.nodes <= GDN_MAX_NODES, YUUKA_ERR_UNSUPPORTED, "gdn: at most %d rows per sequence", GDN_MAX_NODES);
    YK_REQUIRE(rows.chains || rows.order, YUUKA_ERR_INTERNAL, "gdn: a tree step needs its rows depth first");
    launch_gdn_front(s, a, rows, rows.chains != 0);
    ScanParams p{a, rows, 0, 0};
    const int N = rows.nodes;
    dim3 grid(a.S / GDN_COLS, a.rank, rows.batch);
    const size_t smem = sizeof(float) * ((size_t)2 * N * (a.S + 16) + 3 * N * GDN_COLS + 3 * N + (rows.chains ? 0 : (size_t)(a.S / 4) * GDN_WARPS * 32 + 1));
    auto launch = [&](auto kern) {
        YK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        launch_k_cluster(kern, grid, GDN_WARPS * 32, smem, s, grid.x, p);
    };
    if (a.S == 128) {
        if (rows.chains) launch(gdn_scan_kernel<128, false>);
        else launch(gdn_scan_kernel<128, true>);
    } else {
        if (rows.chains) launch(gdn_scan_kernel<64, false>);
        else launch(gdn_scan_kernel<64, true>);
    }
    YK_CUDA(cudaGetLastError());
    return 2;
}

// ---------------------------------------------------------------------------
// Chunkwise (WY-form) scan for chains whose rows are all committed: the sub-chunks of a prompt pass.
// gdnChunkedScan (model/qwen35/recurrent.go:107-351) expresses the rows of a chunk relative to the state S_0 at
// its start; here the same algebra is arranged so that every decay factor is a ratio exp(g_r - g_s) <= 1 (the
// reference scales the values by exp(-g), which overflows for strongly decaying heads over 64 rows). With g the
// cumulative log decay, gam_r = exp(g_r), and d_r = beta_r (v_r - (decayed state)^T k_r) the per-token delta:
//   (I + B) D = diag(beta) (V - diag(gam) K S_0),   B[r][s] = beta_r exp(g_r - g_s) (k_r . k_s)  for s < r
//   o_r = gam_r q_r S_0 + sum_{s <= r} exp(g_r - g_s) (q_r . k_s) d_s
//   S_C = gam_C S_0 + sum_s exp(g_C - g_s) k_s d_s^T
// Three launches take a whole pass. (1) The matrices B and A and the inverses of B's diagonal blocks depend on neither the
// state nor the column: one CTA per (chunk, key head) makes them for all chunks at once, K K^T and Q K^T shared by the
// value heads of a key head. (2) One CTA per (head, 32 columns) walks the chunks with its columns of the state in shared
// memory: K S_0 and Q S_0, the substitution, outputs and state update; the next chunk's q and k arrive meanwhile.
// (3) The gated norm of all rows, where a head's columns meet again.
// (One launch per chunk with all of this inside took 22.5 us per 64 rows of 32 heads: a chain of loads, barriers and
// cluster exchanges, and every column block made B and A again. 512 rows: 180 us then; now 12 + 68 + 9.)
//
// Every product is a tensor-core product, mma.sync m16n8k8 on tf32 operands, with both operands split into two
// tf32 parts (x = hi + lo, three products: lo hi, hi lo, hi hi), which keeps fp32-level accuracy: the two forms
// of the recurrence have to agree to 1e-4 (model/qwen35/recurrent_test.go:60-64). A first form of this kernel
// on fp32 FMAs with 4 x 4 register tiles was bound by shared-memory loads and latency chains (48 k cycles per
// 64-row chunk against 100 k for the row-by-row scan).
constexpr int GC_THREADS = 512;
constexpr int GC_WARPS = GC_THREADS / 32;
constexpr int GC_CP = GDN_COLS + 8;  // pitch of the [row][32 columns] arrays and of the state block: the four k rows
                                     // a B fragment reads fall on distinct banks (8 t + g)

// x = hi + lo with hi the leading 10 mantissa bits (the tensor core ignores the low 13 bits of a tf32 operand, so
// lo, exact in fp32, is used as it is: its own truncation is 2^-20 of x). Masking instead of cvt.rna.tf32: the
// conversion instruction issues at a fraction of the ALU rate and was the whole cost of this kernel's products.
__device__ __forceinline__ void tf32_split(float x, uint32_t & hi, uint32_t & lo) {
    hi = __float_as_uint(x) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// acc[j] += A (16 x 8 ksteps) * B (8 ksteps x 8, NT tiles side by side). fa(row, k) and fb(k, col) read one
// element of the operands; lane (g, t) of the warp holds rows g, g + 8 and k columns t, t + 4 of A, k rows t, t + 4
// and column g of B, and elements (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1) of each 16 x 8 result.
template <int NT, class FA, class FB>
__device__ __forceinline__ void warp_mma_3x(float (&acc)[NT][4], int ksteps, FA fa, FB fb, int g, int t) {
    for (int ks = 0; ks < ksteps; ks++) {
        const int k0 = ks * 8;
        uint32_t ah[4], al[4];
        tf32_split(fa(g, k0 + t), ah[0], al[0]);
        tf32_split(fa(g + 8, k0 + t), ah[1], al[1]);
        tf32_split(fa(g, k0 + t + 4), ah[2], al[2]);
        tf32_split(fa(g + 8, k0 + t + 4), ah[3], al[3]);
#pragma unroll
        for (int j = 0; j < NT; j++) {
            uint32_t bh[2], bl[2];
            tf32_split(fb(k0 + t, 8 * j + g), bh[0], bl[0]);
            tf32_split(fb(k0 + t + 4, 8 * j + g), bh[1], bl[1]);
            mma_tf32(acc[j], al, bh);
            mma_tf32(acc[j], ah, bl);
            mma_tf32(acc[j], ah, bh);
        }
    }
}

__device__ __forceinline__ void cp_async16(void * dst, const void * src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// What launch (1) leaves for a (chunk, head), pitches chosen for the fragment loads of launch (2) (banks 4 g + t)
constexpr int GC_ROWS = GDN_MAX_NODES;
constexpr int GC_NP = GC_ROWS + 4, GC_TP = 20;
struct ChunkPair {
    float B[GC_ROWS * GC_NP];  // beta_r w_rs (k_r . k_s), 16 x 16 blocks below the diagonal ones
    float A[GC_ROWS * GC_NP];  // w_rs (q_r . k_s), blocks up to the diagonal ones
    float T[GC_ROWS * GC_TP];  // inverses of the 16 x 16 diagonal blocks of I + B
    float beta[GC_ROWS], gam[GC_ROWS], tail[GC_ROWS];  // beta_r, exp(g_r), exp(g_C - g_r)
};
static_assert(sizeof(ChunkPair) % 16 == 0, "copied in 16-byte pieces");

struct ChunkParams {
    GdnArgs a;
    int rows;          // of the pass
    ChunkPair * pairs; // [chunks][rank]
};

// q and k rows [r0, r0 + n) of one key head -> shared memory, zero rows up to `padded`
template <int S>
__device__ __forceinline__ void chunk_fetch_rows(float * dst, const float * src, int key_dim, int n, int padded) {
    constexpr int KP = S + 4, SQ = S / 4;
    for (int i = threadIdx.x; i < padded * SQ; i += GC_THREADS) {
        const int node = i / SQ, e4 = i - node * SQ;
        if (node < n) cp_async16(dst + node * KP + e4 * 4, src + (int64_t)node * key_dim + e4 * 4);
        else *reinterpret_cast<float4 *>(dst + node * KP + e4 * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// (1) grid (chunks, groups)
constexpr int GC_HEADS = 4;  // value heads of a key head worked on together
template <int S>
__global__ void __launch_bounds__(GC_THREADS, 1) gdn_chunk_pairs_kernel(const ChunkParams p) {
    pdl_entry();
    const GdnArgs & a = p.a;
    const int kh = blockIdx.y, r0 = blockIdx.x * GC_ROWS, N = min(GC_ROWS, p.rows - r0);
    const int key_dim = a.groups * S, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    constexpr int KP = S + 4;            // pitch of a q / k row: the eight rows an A fragment reads fall on banks 4 g + t
    const int MT = (N + 15) >> 4;        // 16-row tiles
    const int NR = MT * 16;              // rows with padding (zero rows)
    extern __shared__ __align__(16) float sm[];
    float * qn = sm, * kn = qn + NR * KP;
    __shared__ float lg[GC_HEADS][GC_ROWS], bet[GC_HEADS][GC_ROWS];
    __shared__ float diag[GC_HEADS][GC_ROWS * 17];  // diagonal blocks of B
    chunk_fetch_rows<S>(qn, a.qn + (int64_t)r0 * key_dim + kh * S, key_dim, N, NR);
    chunk_fetch_rows<S>(kn, a.khat + (int64_t)r0 * key_dim + kh * S, key_dim, N, NR);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // K K^T and Q K^T on the lower triangle: 16 x 16 tiles up to the diagonal one, two per warp at most
    const int per_mat = MT * (MT + 1) / 2;
    constexpr int SLOTS = (4 * 5 + GC_WARPS - 1) / GC_WARPS;
    float acc[SLOTS][2][4];
    int tile_r[SLOTS], tile_c[SLOTS];
#pragma unroll
    for (int slot = 0; slot < SLOTS; slot++) {
        const int tile = warp + slot * GC_WARPS, mat = tile >= per_mat, rest = tile - mat * per_mat;
        int mt = 0;
        while ((mt + 1) * (mt + 2) / 2 <= rest) mt++;
        tile_r[slot] = mt;
        tile_c[slot] = rest - mt * (mt + 1) / 2;
        if (tile >= 2 * per_mat) continue;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[slot][j][e] = 0.0f;
        const float * arow = (mat ? qn : kn) + (16 * mt) * KP, * brow = kn + (16 * tile_c[slot]) * KP;
        warp_mma_3x<2>(acc[slot], S / 8, [&](int r, int k) { return arow[r * KP + k]; }, [&](int k, int c) { return brow[c * KP + k]; }, g, t);
    }
    for (int h0 = kh; h0 < a.rank; h0 += GC_HEADS * a.groups) {
        const int heads = min(GC_HEADS, (a.rank - h0 + a.groups - 1) / a.groups);
        __syncthreads();
        for (int i = threadIdx.x; i < heads * GC_ROWS; i += GC_THREADS) {
            const int j = i / GC_ROWS, node = i - j * GC_ROWS;
            float b = 0.0f, l = 0.0f;
            if (node < N) {
                const int64_t at = (int64_t)(r0 + node) * a.rank + h0 + j * a.groups;
                b = a.beta[at];
                const float dc = a.decay[at];
                l = dc > 0.0f ? fmaxf(logf(dc), -100.0f) : -100.0f;  // a decay that underflowed still wipes the state
            }
            bet[j][node] = b;
            lg[j][node] = l;
        }
        __syncthreads();
        if (warp < heads) {
            // inclusive scan of the (at most 64) log decays: two per lane
            float s0v = lg[warp][lane], s1v = lg[warp][lane + 32];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float u0 = __shfl_up_sync(0xffffffffu, s0v, o), u1 = __shfl_up_sync(0xffffffffu, s1v, o);
                if (lane >= o) { s0v += u0; s1v += u1; }
            }
            const float first = __shfl_sync(0xffffffffu, s0v, 31);
            lg[warp][lane] = s0v;
            lg[warp][lane + 32] = first + s1v;
        }
        __syncthreads();
        // decay ratios and beta folded in; entries above the diagonal inside the diagonal tiles are zero
        for (int j = 0; j < heads; j++) {
            ChunkPair & out = p.pairs[(int64_t)blockIdx.x * a.rank + h0 + j * a.groups];
#pragma unroll
            for (int slot = 0; slot < SLOTS; slot++) {
                const int tile = warp + slot * GC_WARPS, mat = tile >= per_mat;
                if (tile >= 2 * per_mat) continue;
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int rr = g + (e >> 1) * 8, cc = 8 * n + 2 * t + (e & 1);
                        const int r = 16 * tile_r[slot] + rr, c = 16 * tile_c[slot] + cc;
                        const float wgt = c <= r ? expf(lg[j][r] - lg[j][c]) : 0.0f;
                        if (mat) {
                            out.A[r * GC_NP + c] = wgt * acc[slot][n][e];
                        } else {
                            const float v = c < r ? bet[j][r] * wgt * acc[slot][n][e] : 0.0f;
                            if (tile_r[slot] == tile_c[slot]) diag[j][r * 17 + cc] = v;
                            else out.B[r * GC_NP + c] = v;
                        }
                    }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < heads * GC_ROWS; i += GC_THREADS) {
            const int j = i / GC_ROWS, node = i - j * GC_ROWS;
            ChunkPair & out = p.pairs[(int64_t)blockIdx.x * a.rank + h0 + j * a.groups];
            out.beta[node] = bet[j][node];
            out.gam[node] = expf(lg[j][node]);
            out.tail[node] = node < N ? expf(lg[j][N - 1] - lg[j][node]) : 0.0f;
        }
        // half a warp per diagonal block, lane = column s of the inverse T: row r of T is e_r minus the rows before it
        // weighted by row r of B (forward substitution, as inverseLower of recurrent.go:307-331 does for the
        // whole chunk). Rows beyond the chunk have B = 0 and stay rows of the identity.
        if (warp < 2 * heads) {
            const int j = warp >> 1, b0 = ((warp & 1) * 2 + (lane >> 4)) * 16, sc = lane & 15;
            if (b0 < N) {
                float * T = p.pairs[(int64_t)blockIdx.x * a.rank + h0 + j * a.groups].T;
                float tv[16];
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    float v = r == sc ? 1.0f : 0.0f;
                    const float * brow = diag[j] + (b0 + r) * 17;
#pragma unroll
                    for (int u = 0; u < r; u++) v = fmaf(-brow[u], tv[u], v);
                    tv[r] = v;
                    T[(b0 + r) * GC_TP + sc] = v;
                }
            }
        }
    }
}

// (2) grid (S/32 column blocks, rank)
template <int S>
__global__ void __launch_bounds__(GC_THREADS, 1) gdn_chunk_scan_kernel(const ChunkParams p) {
    pdl_entry();
    const GdnArgs & a = p.a;
    const int cb = blockIdx.x, h = blockIdx.y, kh = h % a.groups;
    const int key_dim = a.groups * S, inner = a.rank * S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    constexpr int KP = S + 4, CP = GC_CP, NP = GC_NP;
    extern __shared__ __align__(16) float sm[];
    float * qn = sm;                         // [GC_ROWS][KP]
    float * kbuf = qn + GC_ROWS * KP;        // two of them: this chunk's keys and the next one's
    float * s0 = kbuf + 2 * GC_ROWS * KP;    // [S][CP] this CTA's columns of the state
    float * vv = s0 + S * CP;                // [GC_ROWS][CP] v, later exp(g_C - g_s) d_s
    float * rhs = vv + GC_ROWS * CP;         // [GC_ROWS][CP] beta (v - gam K S_0)
    float * dd = rhs + GC_ROWS * CP;         // [GC_ROWS][CP] D
    ChunkPair & pair = *reinterpret_cast<ChunkPair *>(dd + GC_ROWS * CP);
    const int chunks = (p.rows + GC_ROWS - 1) / GC_ROWS;
    const float * qsrc = a.qn + kh * S, * ksrc = a.khat + kh * S, * vsrc = a.vconv + h * S + cb * GDN_COLS;
    float * state = const_cast<float *>(a.state) + (int64_t)h * S * S + cb * GDN_COLS;
    float * osrc = a.out + h * S + cb * GDN_COLS;

    auto rows_of = [&](int c) { return min(GC_ROWS, p.rows - c * GC_ROWS); };
    auto fetch_qk = [&](int c) {
        const int n = rows_of(c), padded = (n + 15) & ~15;
        chunk_fetch_rows<S>(qn, qsrc + (int64_t)c * GC_ROWS * key_dim, key_dim, n, padded);
        chunk_fetch_rows<S>(kbuf + (c & 1) * GC_ROWS * KP, ksrc + (int64_t)c * GC_ROWS * key_dim, key_dim, n, padded);
        cp_async_commit();
    };
    for (int i = tid; i < S * (GDN_COLS / 4); i += GC_THREADS) {
        const int row = i / (GDN_COLS / 4), c4 = i - row * (GDN_COLS / 4);
        cp_async16(s0 + row * CP + c4 * 4, state + (int64_t)row * S + c4 * 4);
    }
    fetch_qk(0);
    for (int c = 0; c < chunks; c++) {
        const int N = rows_of(c), MT = (N + 15) >> 4, NR = MT * 16, r0 = c * GC_ROWS;
        const float * kn = kbuf + (c & 1) * GC_ROWS * KP;
        {   // v and the matrices of this chunk: needed after the first products
            const float4 * src = reinterpret_cast<const float4 *>(p.pairs + (int64_t)c * a.rank + h);
            for (int i = tid; i < (int)(sizeof(ChunkPair) / 16); i += GC_THREADS) cp_async16(reinterpret_cast<float4 *>(&pair) + i, src + i);
            for (int i = tid; i < NR * (GDN_COLS / 4); i += GC_THREADS) {
                const int node = i / (GDN_COLS / 4), e4 = i - node * (GDN_COLS / 4);
                if (node < N) cp_async16(vv + node * CP + e4 * 4, vsrc + (int64_t)(r0 + node) * inner + e4 * 4);
                else *reinterpret_cast<float4 *>(vv + node * CP + e4 * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            cp_async_commit();
        }
        cp_async_wait<1>();  // q, k (and the state) have landed
        __syncthreads();
        // ---- K S_0 (warps 0-7) and Q S_0 (warps 8-15): a warp per 16 rows x 16 columns; Q S_0 stays in registers ----
        const int nh = warp & 1, mt = (warp >> 1) & 3;
        const bool is_q = warp >= 8;
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        if (mt < MT) {
            const float * arow = (is_q ? qn : kn) + (16 * mt) * KP, * bcol = s0 + 16 * nh;
            warp_mma_3x<2>(acc, S / 8, [&](int r, int k) { return arow[r * KP + k]; }, [&](int k, int col) { return bcol[k * CP + col]; }, g, t);
        }
        cp_async_wait<0>();
        __syncthreads();
        if (c + 1 < chunks) fetch_qk(c + 1);
        // ---- right-hand side beta (v - gam K S_0) ----
        if (!is_q && mt < MT) {
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int r = 16 * mt + g + (e >> 1) * 8, at = r * CP + 16 * nh + 8 * j + 2 * t + (e & 1);
                    rhs[at] = pair.beta[r] * (vv[at] - pair.gam[r] * acc[j][e]);
                }
        }
        __syncthreads();
        // ---- forward substitution over the blocks: D_b = T_b (rhs_b - B[b][earlier] D[earlier]); a warp per 8 columns,
        // which meets no other warp's columns ----
        if (warp < 4) {
            for (int b0 = 0; b0 < N; b0 += 16) {
                float * rh = rhs + b0 * CP + 8 * warp;
                if (b0 > 0) {
                    float sub[1][4] = {{0.f, 0.f, 0.f, 0.f}};
                    const float * arow = pair.B + b0 * NP, * bcol = dd + 8 * warp;
                    warp_mma_3x<1>(sub, b0 / 8, [&](int r, int k) { return arow[r * NP + k]; }, [&](int k, int col) { return bcol[k * CP + col]; }, g, t);
                    float * dst = rh + 2 * t;
                    dst[g * CP] -= sub[0][0];
                    dst[g * CP + 1] -= sub[0][1];
                    dst[(g + 8) * CP] -= sub[0][2];
                    dst[(g + 8) * CP + 1] -= sub[0][3];
                    __syncwarp();
                }
                float d[1][4] = {{0.f, 0.f, 0.f, 0.f}};
                const float * arow = pair.T + b0 * GC_TP;
                warp_mma_3x<1>(d, 2, [&](int r, int k) { return arow[r * GC_TP + k]; }, [&](int k, int col) { return rh[k * CP + col]; }, g, t);
                const int at = b0 * CP + 8 * warp + 2 * t;
                *reinterpret_cast<float2 *>(dd + at + g * CP) = make_float2(d[0][0], d[0][1]);
                *reinterpret_cast<float2 *>(dd + at + (g + 8) * CP) = make_float2(d[0][2], d[0][3]);
                // (v has gone into the right-hand side; its place takes w d)
                const float w0 = pair.tail[b0 + g], w1 = pair.tail[b0 + g + 8];
                *reinterpret_cast<float2 *>(vv + at + g * CP) = make_float2(w0 * d[0][0], w0 * d[0][1]);
                *reinterpret_cast<float2 *>(vv + at + (g + 8) * CP) = make_float2(w1 * d[0][2], w1 * d[0][3]);
                __syncwarp();
            }
        }
        __syncthreads();
        // ---- outputs gam_r (Q S_0)_r + sum_{s <= r} A[r][s] d_s (warps 8-15, which hold Q S_0) and the new state
        // gam_C S_0 + K^T (w d) (warps 0-7: 16 state rows x 32 columns) ----
        if (is_q) {
            if (mt < MT) {
                float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                const float * arow = pair.A + (16 * mt) * NP, * bcol = dd + 16 * nh;
                warp_mma_3x<2>(o, 2 * mt + 2, [&](int r, int k) { return arow[r * NP + k]; }, [&](int k, int col) { return bcol[k * CP + col]; }, g, t);
                const int r = 16 * mt + g;
                const float g0 = pair.gam[r], g1 = pair.gam[r + 8];
                float * dst = osrc + (int64_t)(r0 + r) * inner + 16 * nh + 2 * t;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (r < N) *reinterpret_cast<float2 *>(dst + 8 * j) = make_float2(fmaf(g0, acc[j][0], o[j][0]), fmaf(g0, acc[j][1], o[j][1]));
                    if (r + 8 < N)
                        *reinterpret_cast<float2 *>(dst + (int64_t)8 * inner + 8 * j) = make_float2(fmaf(g1, acc[j][2], o[j][2]), fmaf(g1, acc[j][3], o[j][3]));
                }
            }
        } else if (warp < S / 16) {
            const float gam_c = pair.gam[N - 1];
            float n[4][4];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) n[j][e] = 0.0f;
            const float * acol = kn + 16 * warp;
            warp_mma_3x<4>(n, NR / 8, [&](int r, int k) { return acol[k * KP + r]; }, [&](int k, int col) { return vv[k * CP + col]; }, g, t);
            float * own = s0 + (16 * warp + g) * CP + 2 * t;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float2 * o0 = reinterpret_cast<float2 *>(own + 8 * j), * o1 = reinterpret_cast<float2 *>(own + 8 * CP + 8 * j);
                *o0 = make_float2(fmaf(gam_c, o0->x, n[j][0]), fmaf(gam_c, o0->y, n[j][1]));
                *o1 = make_float2(fmaf(gam_c, o1->x, n[j][2]), fmaf(gam_c, o1->y, n[j][3]));
            }
        }
        __syncthreads();
    }
    pdl_trigger_late();
    for (int i = tid; i < S * (GDN_COLS / 4); i += GC_THREADS) {
        const int row = i / (GDN_COLS / 4), c4 = i - row * (GDN_COLS / 4);
        *reinterpret_cast<float4 *>(state + (int64_t)row * S + c4 * 4) = *reinterpret_cast<const float4 *>(s0 + row * CP + c4 * 4);
    }
}

// (3) gated RMSNorm (recurrent.go:39-50) of every (row, head): a warp each, S / 32 columns per lane, the sums of squares
// in the scan kernel's order. Reads the outputs from a.out and leaves them there and prepared, or, where the out
// projection reads nothing but their fp16 form, only that.
template <int S>
__global__ void __launch_bounds__(256) gdn_gated_norm_kernel(const GdnArgs a, int rows) {
    pdl_entry();
    constexpr int G = S / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, inner = a.rank * S;
    const int64_t item = (int64_t)blockIdx.x * 8 + warp;
    __shared__ __align__(16) float stage[8][S];
    if (item >= (int64_t)rows * a.rank) return;
    const int r = (int)(item / a.rank), h = (int)(item - (int64_t)r * a.rank);
    const int64_t at = (int64_t)r * inner + h * S + lane;
    float o[G], z[G], w[G];
    double sq[G];
#pragma unroll
    for (int i = 0; i < G; i++) {
        o[i] = a.out[at + 32 * i];
        z[i] = a.z[(int64_t)r * a.ldz + h * S + lane + 32 * i];
        w[i] = a.norm[lane + 32 * i];
    }
#pragma unroll
    for (int i = 0; i < G; i++) sq[i] = (double)o[i] * (double)o[i];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1)
#pragma unroll
        for (int i = 0; i < G; i++) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], k);
    double tot = 0;
#pragma unroll
    for (int i = 0; i < G; i++) tot += sq[i];
    const float mean = (float)(tot / (double)S);
    const float scale = (float)(1.0 / sqrt((double)(mean + a.eps)));
    const bool hi_only = a.prep.hi_only();
#pragma unroll
    for (int i = 0; i < G; i++) {
        const float v = o[i] * (scale * w[i]) * silu_ref(z[i]);
        if (hi_only) {
            a.prep.xh[at + 32 * i] = __float2half_rn(v);
        } else {
            a.out[at + 32 * i] = v;
            stage[warp][lane + 32 * i] = v;
        }
    }
    if (hi_only || !a.prep.xh) return;
    __syncwarp();
    if (lane < S / 16) {
        float g16[16];
#pragma unroll
        for (int i = 0; i < 16; i++) g16[i] = stage[warp][lane * 16 + i];
        const int64_t c0 = (int64_t)r * inner + h * S + lane * 16;
        xprep_store16(a.prep.xh + c0, a.prep.xl + c0, a.prep.xs16 + (c0 >> 4), g16);
    }
}

size_t gdn_chunk_scratch_bytes(int rows, int rank) { return (size_t)((rows + GC_ROWS - 1) / GC_ROWS) * rank * sizeof(ChunkPair); }

// One chain of any length whose rows are all committed (a prompt pass of one sequence): the front end for the whole pass
// (conv taps come from the preceding rows and, for the first kernel - 1 rows, from the stored history), then the chunkwise
// scan; the state is rewritten in place (the conv history still moves with launch_gdn_commit(..., conv_only)).
template <int S>
static void launch_gdn_chunks_s(cudaStream_t s, const ChunkParams & p) {
    const GdnArgs & a = p.a;
    constexpr size_t ROW = sizeof(float) * GC_ROWS * (S + 4);
    const size_t pairs_smem = 2 * ROW;
    const size_t scan_smem = 3 * ROW + sizeof(float) * (S + 3 * GC_ROWS) * GC_CP + sizeof(ChunkPair);
    YK_CUDA(cudaFuncSetAttribute(gdn_chunk_pairs_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pairs_smem));
    YK_CUDA(cudaFuncSetAttribute(gdn_chunk_scan_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scan_smem));
    launch_k(gdn_chunk_pairs_kernel<S>, dim3((p.rows + GC_ROWS - 1) / GC_ROWS, a.groups), GC_THREADS, pairs_smem, s, p);
    launch_k(gdn_chunk_scan_kernel<S>, dim3(S / GDN_COLS, a.rank), GC_THREADS, scan_smem, s, p);
    launch_k(gdn_gated_norm_kernel<S>, (int)(((int64_t)p.rows * a.rank + 7) / 8), 256, 0, s, a, p.rows);
    YK_CUDA(cudaGetLastError());
}
int launch_gdn_chunks(cudaStream_t s, const GdnArgs & a, int n_rows, void * scratch) {
    RowMeta rows{};
    rows.batch = 1;
    rows.nodes = n_rows;
    launch_gdn_front(s, a, rows, true);
    const ChunkParams p{a, n_rows, static_cast<ChunkPair *>(scratch)};
    if (a.S == 128) launch_gdn_chunks_s<128>(s, p);
    else launch_gdn_chunks_s<64>(s, p);
    return 4;
}

// ---------------------------------------------------------------------------
// commit

struct CommitParams {
    const GdnLayerCommit * layers;
    int groups, rank, S, kernel, conv_dim;
    int seq_base;  // first sequence of the step within the session's state arrays
    int row_base;  // first row of the step within the layer's per-row logs (sub-chunks of a wide prompt pass)
    int conv_only; // the grid holds only the conv-history blocks (the chunkwise scan has written the state itself)
    RowMeta rows;
    AcceptOut acc;
};

// grid (4 * rank + 8, batch, layers): blocks 0..4*rank-1 update a quarter of one head's state (S/4 rows),
// the last eight rewrite the conv history, an eighth of the channels each.
constexpr int COMMIT_PARTS = 4;
constexpr int COMMIT_CONV_PARTS = 8;
__global__ void __launch_bounds__(256, 4) gdn_commit_kernel(const CommitParams p) {
    pdl_entry();
    const GdnLayerCommit L = p.layers[blockIdx.z];
    const int seq = blockIdx.y, N = p.rows.nodes, S = p.S;
    const int a = p.acc.accepted[seq];
    const int32_t * path = p.acc.path + (int64_t)seq * N;
    auto node_at = [&](int t) { return t == 0 ? 0 : path[t - 1]; };  // t = 0..a
    if (!p.conv_only && (int)blockIdx.x < COMMIT_PARTS * p.rank) {
        // S/4 rows of one head's S x S state, read and written once as float4 however many rows were accepted.
        // A thread owns four columns j and up to four rows i and keeps them in registers. The accepted rows'
        // keys (this part's S/4 of them), d values and decays are brought into shared memory in one round of
        // loads, all rows at once (up to 64 in a prompt sub-chunk: fetching them nine at a time between
        // barriers made that commit a chain of L2 round trips, 57 us per layer).
        constexpr int MAXR = 4;
        const int h = blockIdx.x / COMMIT_PARTS, part = blockIdx.x % COMMIT_PARTS, kh = h % p.groups;
        const int rows_part = S / COMMIT_PARTS, i_base = part * rows_part;
        float * st = L.state + (int64_t)((p.seq_base + seq_of(p.rows, seq)) * p.rank + h) * S * S;
        __shared__ float kh_s[GDN_MAX_NODES][32];
        __shared__ __align__(16) float d_s[GDN_MAX_NODES][128];
        __shared__ float dec_s[GDN_MAX_NODES];
        __shared__ int row_s[GDN_MAX_NODES];
        const int quads = S >> 2;
        const int j4 = threadIdx.x % quads, i0 = threadIdx.x / quads, istep = blockDim.x / quads;
        float4 v[MAXR];
#pragma unroll
        for (int q = 0; q < MAXR; q++) {
            const int i = i0 + q * istep;
            v[q] = i < rows_part ? *reinterpret_cast<const float4 *>(st + (int64_t)(i_base + i) * S + j4 * 4)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const int nt = a + 1;  // <= N <= GDN_MAX_NODES
        for (int t = threadIdx.x; t < nt; t += blockDim.x) {
            const int r = p.row_base + seq * N + node_at(t);
            row_s[t] = r;
            dec_s[t] = L.decay[(int64_t)r * p.rank + h];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < nt * rows_part; idx += blockDim.x) {
            const int t = idx / rows_part, i = idx - t * rows_part;
            kh_s[t][i] = L.khat[(int64_t)row_s[t] * (p.groups * S) + kh * S + i_base + i];
        }
        for (int idx = threadIdx.x; idx < nt * quads; idx += blockDim.x) {
            const int t = idx / quads, c4 = idx - t * quads;
            reinterpret_cast<float4 *>(d_s[t])[c4] =
                *reinterpret_cast<const float4 *>(L.dlog + (int64_t)row_s[t] * (p.rank * S) + h * S + c4 * 4);
        }
        __syncthreads();
        for (int t = 0; t < nt; t++) {
            const float dc = dec_s[t];
            const float4 d = reinterpret_cast<const float4 *>(d_s[t])[j4];
#pragma unroll
            for (int q = 0; q < MAXR; q++) {
                const int i = i0 + q * istep;
                const float k = kh_s[t][i < rows_part ? i : 0];
                v[q].x = state_update(v[q].x, dc, k, d.x);
                v[q].y = state_update(v[q].y, dc, k, d.y);
                v[q].z = state_update(v[q].z, dc, k, d.z);
                v[q].w = state_update(v[q].w, dc, k, d.w);
            }
        }
#pragma unroll
        for (int q = 0; q < MAXR; q++) {
            const int i = i0 + q * istep;
            if (i < rows_part) *reinterpret_cast<float4 *>(st + (int64_t)(i_base + i) * S + j4 * 4) = v[q];
        }
    } else {
        // history after the step = last kernel-1 raw inputs of [old history, accepted rows]: entry t takes the
        // combined index n_new - K1 + t, where the old history occupies [-K1, -1] and the accepted rows
        // [0, n_new - 1]. The (at most kernel-1) source rows are looked up once per CTA; the channels are
        // spread over COMMIT_CONV_PARTS CTAs (one CTA walking all channels with a path look-up per entry was
        // a 45 us chain of dependent loads: most of this kernel's time).
        const int K1 = p.kernel - 1, n_new = a + 1;
        __shared__ int src_row[8];
        if (threadIdx.x < K1) {
            const int src = n_new + (int)threadIdx.x - K1;
            src_row[threadIdx.x] = src >= 0 ? p.row_base + seq * N + node_at(src) : -1;
        }
        __syncthreads();
        const int part = p.conv_only ? (int)blockIdx.x : (int)blockIdx.x - COMMIT_PARTS * p.rank;
        const int per = (p.conv_dim + COMMIT_CONV_PARTS - 1) / COMMIT_CONV_PARTS;
        const int c_end = min(p.conv_dim, (part + 1) * per);
        for (int c = part * per + threadIdx.x; c < c_end; c += blockDim.x) {
            float * hist = L.conv_state + ((int64_t)(p.seq_base + seq_of(p.rows, seq)) * p.conv_dim + c) * K1;
            float nv[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                if (t >= K1) continue;
                const int src = n_new + t - K1;
                nv[t] = src >= 0 ? L.proj[(int64_t)src_row[t] * L.ldp + c] : hist[K1 + src];
            }
#pragma unroll
            for (int t = 0; t < 8; t++)
                if (t < K1) hist[t] = nv[t];
        }
    }
}

void launch_gdn_commit(cudaStream_t s, const GdnLayerCommit * layers_dev, int n_layers, int groups, int rank, int S,
                       int kernel, int conv_dim, int seq_base, const RowMeta & rows, const AcceptOut & acc, int row_base,
                       bool conv_only) {
    if (n_layers == 0) return;
    CommitParams p{layers_dev, groups, rank, S, kernel, conv_dim, seq_base, row_base, conv_only ? 1 : 0, rows, acc};
    dim3 grid(conv_only ? COMMIT_CONV_PARTS : COMMIT_PARTS * rank + COMMIT_CONV_PARTS, rows.batch, n_layers);
    launch_k(gdn_commit_kernel, grid, 256, 0, s, p);
    YK_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// KV commit: accepted row t (t >= 1) of a tree moves from slot pos0 + node to
// its final position pos0 + t. A chain is already in place.

struct KvCommitParams {
    const KvLayerCommit * layers;
    KvPool geom;
    RowMeta rows;
    AcceptOut acc;
};

__global__ void kv_commit_kernel(const KvCommitParams p) {
    pdl_entry();
    const KvLayerCommit L = p.layers[blockIdx.y];
    const int seq = blockIdx.x, N = p.rows.nodes;
    const int a = p.acc.accepted[seq];
    const int sq = seq_of(p.rows, seq);
    const int pos0 = p.rows.pos0[sq];
    const int32_t * path = p.acc.path + (int64_t)seq * N;
    const int words = p.geom.row_bytes / 2;
    for (int t = 1; t <= a; t++) {
        const int node = path[t - 1];
        if (node != t) {
            auto off = [&](int slot) {
                int block = p.geom.tables[(int64_t)sq * p.geom.table_stride + slot / p.geom.block_size];
                return ((int64_t)block * p.geom.block_size + slot % p.geom.block_size) * p.geom.row_bytes;
            };
            const int64_t src = off(pos0 + node), dst = off(pos0 + t);
            const uint16_t * ks = reinterpret_cast<const uint16_t *>(L.k + src);
            const uint16_t * vs = reinterpret_cast<const uint16_t *>(L.v + src);
            uint16_t * kd = reinterpret_cast<uint16_t *>(L.k + dst);
            uint16_t * vd = reinterpret_cast<uint16_t *>(L.v + dst);
            for (int i = threadIdx.x; i < words; i += blockDim.x) {
                kd[i] = ks[i];
                vd[i] = vs[i];
            }
        }
        __syncthreads();
    }
}

void launch_kv_commit(cudaStream_t s, const KvLayerCommit * layers_dev, int n_layers, const KvPool & geom,
                      const RowMeta & rows, const AcceptOut & acc) {
    if (n_layers == 0) return;
    KvCommitParams p{layers_dev, geom, rows, acc};
    dim3 grid(rows.batch, n_layers);
    launch_k(kv_commit_kernel, grid, 256, 0, s, p);
    YK_CUDA(cudaGetLastError());
}

__global__ void advance_positions_kernel(int32_t * pos0, const int32_t * accepted, int batch, const int32_t * seq_map) {
    pdl_entry();
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < batch) pos0[seq_map ? seq_map[b] : b] += accepted[b] + 1;
}

void launch_advance_positions(cudaStream_t s, int32_t * pos0, const AcceptOut & acc, int batch, const int32_t * seq_map) {
    launch_k(advance_positions_kernel, (batch + 127) / 128, 128, 0, s, pos0, acc.accepted, batch, seq_map);
    YK_CUDA(cudaGetLastError());
}

}  // namespace yk
