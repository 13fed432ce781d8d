// Large-M route of the tiled quantized GEMM: tcgen05 tensor cores with the
// accumulator in tensor memory. Included by gemm_tiled.cu (it uses that file's
// record codecs and header decoders).
//
// From 48 rows on (33 on request), re-decoding the packed weights for every 16-row pass of the register-fed
// kernel costs more than the arithmetic. Here two CTAs of a cluster form a pair on one tile of 256 weight rows x up to
// 256 activation rows (cta_group::2, M = 256): each CTA decodes its own 128 weight rows into fp16 (s * q - min, rounded:
// this route does not have the register-fed route's exactness), 64 columns at a time, and fetches half of the
// tile's activation rows (their fp16 hi halves, a tensor-map copy). The even CTA issues the MMAs of both; each CTA reads its own half of D back.
//
// Where the decoded weights lie. Up to 192 activation rows per tile tensor memory has room for two accumulators and four
// stages of weights beside them, and the decode warps store there (tcgen05.st, the A operand of the MMA): the weights then pass
// through shared memory once, packed, instead of three times. Wider tiles keep the stages in shared memory, since their two
// accumulators fill tensor memory (one accumulator beside the weights was no faster: its epilogue runs alone), and so do Q5_K and
// Q8_0 where a pair walks few superblocks (umma_tmem). The operands are
// the same numbers either way, and so are the results.
//
// What bounds it, and why this tile. At M = 128 per CTA a stage of 64 columns keeps the tensor pipe busy for two cycles
// per activation row of the tile. Its activations come from L2, which feeds all SMs 46 bytes per cycle each
// (13 TB/s measured): one CTA alone on 256 activation rows needs 64 bytes per cycle, a pair that shares them 32. The decode
// of a stage (8192 weights per SM) with its barriers and the products do not hide one another: a stage takes 330 cycles and 1.8
// per row (540 and 1.3 through shared memory), a line through measured times that names no cause. Counters at 18432 x 2560 Q4_K,
// 544 rows (three tiles of 192): the tensor pipe is busy 66 % of an SM's active cycles, the issue slots 57 %, the shared-memory
// port 55 % (58 % of its wavefronts are bank conflicts, nearly all of them loads), and the SMs stand idle for 18 % of the launch.
// Tensor memory holds two accumulators at least: the epilogue of a tile runs on warps of its own while the next tile is decoded
// and multiplied.
// Calls on a B200, with the weights in shared memory and in tensor memory: 248320 x 2560 Q6_K 187 -> 154 us at 48 rows (3.4 TB/s
// of weights), 250 -> 222 at 192, 693 -> 590 at 544 (three tiles of 192; 1.2 PFLOP/s); 9216 x 2560 Q4_K at 576 rows
// 38.5 -> 35 us; 9216 x 2560 Q6_K 20.2 -> 17.6 at 48 rows, 21.5 -> 19.0 at 192; 18432 x 2560 Q4_K at 576 rows 50.5 -> 47.
//
// Roles of a CTA's warps: sixteen decode warps (two per 16-row tile), four epilogue warps, one warp that copies packed
// weights (one bulk copy per record, a superblock of all eight tiles per stage, ahead of everything else), one that copies
// activations, one that issues the MMAs (even CTA) or passes on, stage by stage, what the odd CTA's other warps have arrived
// for.
// Every mbarrier wait is bounded. A warp whose wait runs out leaves its loop: it issues no copy and no MMA after that, and
// those it issued before have had the whole of that wait to finish. The others run out of what it owes them and follow; the
// kernel sets the device error word, frees its tensor memory and returns (results are garbage).
#pragma once

namespace yk {

constexpr int UM_ROWS = 128;     // weight rows per CTA; a pair has 256
constexpr int UM_KC = 64;        // columns per stage
constexpr int UM_MAX_N = 256;    // activation rows per tile
constexpr int UM_MAX_STAGES = 6;
constexpr int UM_MAX_ACC = 4;    // accumulators
constexpr int UM_A_COLS = UM_KC / 2;  // tensor-memory columns of a weight stage: 128 lanes (rows) x 64 columns of fp16
constexpr int UM_TMEM_N = 192;   // activation rows per tile up to which the weight stages are in tensor memory
constexpr int UM_MAX_RAW = 4;    // superblocks of packed weights in shared memory
constexpr int UM_TILES = 8;      // 16-row tiles per CTA
constexpr int UM_DW = 16;        // decode warps, two per tile: a half of every record each
constexpr int UM_EW = 4;         // epilogue warps, one per quarter of the tensor-memory lanes
constexpr int UM_WARP_RAW = UM_DW + UM_EW, UM_WARP_X = UM_WARP_RAW + 1, UM_WARP_MMA = UM_WARP_X + 1;
constexpr int UM_THREADS = (UM_WARP_MMA + 1) * 32;
static_assert(UM_TILES * 16 == UM_ROWS && UM_DW == 2 * UM_TILES, "two decode warps per tile");
constexpr uint32_t H2_1024B = 0x64646464u, H2_ONE16 = 0x3C003C00u;

constexpr int UM_A_BYTES = UM_ROWS * 128;      // a weight stage: 128 rows of 64 columns
template <int DT> struct UmmaStage { static constexpr int RAW_BYTES = UM_TILES * Codec<DT>::REC; };

struct UParams {
    DecodeConsts kc;
    const uint8_t * w;
    int N, nsb;           // weight rows, superblocks per row
    int M;                // activation rows
    float * out;
    int64_t ldo;
    int accumulate;
    float * partial;      // [kparts][M][N] when K is split across pairs
    int kparts;
    int halves;           // kparts == 1: the two halves of K are summed apart, in two accumulators
    int n_tile, n_tiles;  // activation rows per tile (a multiple of 32), tiles
    int m_blocks;         // blocks of 256 weight rows
    uint32_t idesc;
    uint32_t stages, raw_stages;  // ring depths
    uint32_t acc_cols, n_acc;     // columns of an accumulator, and how many there are (then the weight stages, if they are there)
    int drop_copies;      // test hook: the even CTA's activations are never copied
};

// Both operands: K-major, 128-byte swizzle: rows of 64 halves (128 bytes), eight rows per 1024-byte atom, as a tensor-map
// copy with CU_TENSOR_MAP_SWIZZLE_128B lays them out. 16 columns further along K = 32 bytes.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}
// where 16-byte piece c (eight columns) of row r of a stage lies in that layout
__device__ __forceinline__ uint32_t sw128(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

__device__ __forceinline__ void tmem_store16(uint32_t dst, const uint32_t (&r)[16]) {  // 16 lanes x 32 columns: four 16 x 16 fp16 A fragments
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(dst),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// ---------------------------------------------------------------------------
// Decode of half a record: 16 rows x 128 columns, two stages of 64, by one warp, into shared memory. fetch() takes the warp's share of a
// record out of shared memory; header() turns the block headers into fp16 scales in the warp's own table; store<c>()
// writes 64 columns (sub-blocks 2c, 2c + 1 of the half) as fp16(s * q - min): lane (g, t) holds rows g and g + 8 and eight
// columns of each sub-block. Rows of odd g take the two sub-blocks in the other order: the lanes of a store then hit
// every bank once in the swizzled layout (in the same order rows g and g + 1 would share theirs).
// Two warps share a tile, a half each: a stage costs a warp about as much in barriers, fences and header work (400 cycles)
// as in arithmetic (380), so that two warps per scheduler leave it idle half the time.

// (v & mask) | magic is fp16 1024 + q (low nibble) or 1024 + 16 q (high nibble); times s plus -1024 s, or times s / 16 plus -64 s,
// gives s * q; then the min is added
__device__ __forceinline__ uint32_t nibble_h2(uint32_t v, uint32_t mask, uint32_t extra, uint32_t s, uint32_t c, uint32_t m) {
    return h2_add(h2_fma(and_or(v, mask, extra), s, c), m);
}

template <int DT> struct HalfRecord;

// Q4_K / Q5_K: table rows of 48 bytes: two pairs of sub-blocks (s_lo, -1024 s_lo, s_hi / 16, -64 s_hi); then rows of four (-min, -min)
template <int DT> struct HalfRecordK4 {
    static constexpr int DS = 48, MN_OFF = 16 * DS, TAB = MN_OFF + 16 * 16;
    uint4 qg, qh, hdr;
    __device__ void fetch_k4(const uint8_t * rec, int lane, int half, int hdr_at) {
        const uint4 * p = reinterpret_cast<const uint4 *>(rec);
        qg = p[half * 32 + lane];
        qh = p[(2 + half) * 32 + lane];
        hdr = p[hdr_at + (lane & 15)];
    }
    // hdr.x = d | dmin << 16, hdr.y/z/w = 12 scale bytes (getScaleMinK4, tensor/quant.go:96-103); lane: row, pair of sub-blocks
    __device__ void header(int lane, int half, uint8_t * tab) const {
        const int r = lane & 15, jl = lane >> 4;
        const uint32_t w0 = hdr.y, w1 = hdr.z, w2 = hdr.w;
        const uint32_t sc4 = half ? ((w2 & 0x0f0f0f0fu) | ((w0 >> 2) & 0x30303030u)) : (w0 & 0x3f3f3f3fu);
        const uint32_t mn4 = half ? (((w2 >> 4) & 0x0f0f0f0fu) | ((w1 >> 2) & 0x30303030u)) : (w1 & 0x3f3f3f3fu);
        const uint32_t sel = jl ? 0x4342u : 0x4140u;  // the pair's two bytes as fp16 1024 + b
        const uint32_t sp = h2_mul(h2_sub(__byte_perm(sc4, H2_1024B, sel), H2_1024), dup_lo(hdr.x));
        const uint32_t mp = h2_mul(h2_sub(__byte_perm(mn4, H2_1024B, sel), H2_1024), dup_hi(hdr.x));
        const uint32_t slo = dup_lo(sp), shi = dup_hi(sp);
        reinterpret_cast<uint4 *>(tab + r * DS)[jl] = make_uint4(slo, h2_mul(slo, H2_NEG1024), h2_mul(shi, H2_INV16), h2_mul(shi, H2_NEG64));
        reinterpret_cast<uint2 *>(tab + MN_OFF + r * 16)[jl] = make_uint2(h2_mul(dup_lo(mp), H2_NEG1), h2_mul(dup_hi(mp), H2_NEG1));
    }
};
template <> struct HalfRecord<YUUKA_DTYPE_Q4_K> : HalfRecordK4<YUUKA_DTYPE_Q4_K> {
    __device__ void fetch(const uint8_t * rec, int lane, int half) { fetch_k4(rec, lane, half, 128); }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint8_t * a_tile) const {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t v[2][2] = {{C ? qg.z : qg.x, C ? qg.w : qg.y}, {C ? qh.z : qh.x, C ? qh.w : qh.y}};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int n = k ^ (g & 1);  // sub-block 2C + n: low or high nibbles
            const uint32_t mask = n ? kc.mf0 : kc.m0f;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint2 s = reinterpret_cast<const uint2 *>(tab + (g + 8 * rr) * DS)[2 * C + n];
                const uint32_t m = reinterpret_cast<const uint32_t *>(tab + MN_OFF + (g + 8 * rr) * 16)[2 * C + n];
                const uint32_t v0 = v[rr][0], v1 = v[rr][1];
                *reinterpret_cast<uint4 *>(a_tile + sw128(g + 8 * rr, 4 * n + t)) =
                    make_uint4(nibble_h2(v0, mask, kc.magic, s.x, s.y, m), nibble_h2(v0 >> 8, mask, kc.magic, s.x, s.y, m),
                               nibble_h2(v1, mask, kc.magic, s.x, s.y, m), nibble_h2(v1 >> 8, mask, kc.magic, s.x, s.y, m));
            }
        }
    }
};
template <> struct HalfRecord<YUUKA_DTYPE_Q5_K> : HalfRecordK4<YUUKA_DTYPE_Q5_K> {
    uint4 hi;  // bit k of byte b: fifth bit of column 8t + b of sub-block k of the half
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        fetch_k4(rec, lane, half, 160);
        hi = reinterpret_cast<const uint4 *>(rec)[128 + lane];
        if (half) hi = make_uint4(hi.x >> 4, hi.y >> 4, hi.z >> 4, hi.w >> 4);
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint8_t * a_tile) const {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t v[2][2] = {{C ? qg.z : qg.x, C ? qg.w : qg.y}, {C ? qh.z : qh.x, C ? qh.w : qh.y}};
        const uint32_t hb[2][2] = {{hi.x, hi.y}, {hi.z, hi.w}};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int n = k ^ (g & 1);  // sub-block 2C + n: low or high nibbles; its bit 2C + n of each byte goes to bit 4 or 8
            const uint32_t mask = n ? kc.mf0 : kc.m0f, hm = n ? kc.h8 : kc.h4;
            const int up = n ? 7 - 2 * C : 4 - 2 * C, down = n ? 1 + 2 * C : 4 + 2 * C;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint2 s = reinterpret_cast<const uint2 *>(tab + (g + 8 * rr) * DS)[2 * C + n];
                const uint32_t m = reinterpret_cast<const uint32_t *>(tab + MN_OFF + (g + 8 * rr) * 16)[2 * C + n];
                uint32_t o[4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    o[2 * h] = nibble_h2(v[rr][h], mask, and_or(hb[rr][h] << up, hm, kc.magic), s.x, s.y, m);
                    o[2 * h + 1] = nibble_h2(v[rr][h] >> 8, mask, and_or(hb[rr][h] >> down, hm, kc.magic), s.x, s.y, m);
                }
                *reinterpret_cast<uint4 *>(a_tile + sw128(g + 8 * rr, 4 * n + t)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
};
// Q6_K: table rows of eight groups of 16 columns (s, -1024 s) or, for high nibbles (the last four), (s / 16, -64 s); then -32 s
template <> struct HalfRecord<YUUKA_DTYPE_Q6_K> {
    static constexpr int DS = 80, MN = 48, MN_OFF = 16 * DS, TAB = MN_OFF + 16 * MN;
    uint4 lg, lh;
    uint2 hg, hh, sc;
    uint32_t d;
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        const uint4 * p = reinterpret_cast<const uint4 *>(rec);
        lg = p[half * 32 + lane];
        lh = p[(2 + half) * 32 + lane];
        hg = reinterpret_cast<const uint2 *>(p + 128 + lane)[half];
        hh = reinterpret_cast<const uint2 *>(p + 160 + lane)[half];
        sc = reinterpret_cast<const uint2 *>(p + 192 + (lane & 15))[half];
        d = reinterpret_cast<const uint16_t *>(rec + 3328)[lane & 15];
    }
    __device__ void header(int lane, int, uint8_t * tab) const {
        const int row = lane & 15, up = lane >> 4;  // groups 4 up .. 4 up + 3; the upper ones sit in high nibbles
        const uint32_t w = (up ? sc.y : sc.x) ^ 0x80808080u, d2 = dup_lo(d);
        const uint32_t f = up ? H2_INV16 : H2_ONE16, c = up ? H2_NEG64 : H2_NEG1024;
        uint2 * scl = reinterpret_cast<uint2 *>(tab + row * DS) + 4 * up;
        uint32_t s[4];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t sp = h2_mul(h2_sub(q ? bytes23_h2(w) : bytes01_h2(w), H2_1152), d2);
            s[2 * q] = dup_lo(sp);
            s[2 * q + 1] = dup_hi(sp);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) scl[q] = make_uint2(h2_mul(s[q], f), h2_mul(s[q], c));
        reinterpret_cast<uint4 *>(tab + MN_OFF + row * MN)[up] =
            make_uint4(h2_mul(s[0], H2_NEG32), h2_mul(s[1], H2_NEG32), h2_mul(s[2], H2_NEG32), h2_mul(s[3], H2_NEG32));
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint8_t * a_tile) const {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t qm = C ? kc.mf0 : kc.m0f, hm = C ? kc.h8 : kc.h4;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int hsel = k ^ (g & 1);  // sub-block 2C + hsel
            const int lsh = 4 - 2 * hsel, rsh = 4 + 2 * hsel;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint4 l4 = rr ? lh : lg;
                const uint2 b2 = rr ? hh : hg, m2 = reinterpret_cast<const uint2 *>(tab + MN_OFF + (g + 8 * rr) * MN)[2 * C + hsel];
                const uint4 s2 = reinterpret_cast<const uint4 *>(tab + (g + 8 * rr) * DS)[2 * C + hsel];
#pragma unroll
                for (int h = 0; h < 2; h++) {  // columns 32 hsel + 16 h + 4t .. + 3 of the stage
                    const uint32_t v0 = h ? (hsel ? l4.w : l4.y) : (hsel ? l4.z : l4.x), b0 = h ? b2.y : b2.x;
                    const uint32_t s = h ? s2.z : s2.x, c = h ? s2.w : s2.y, m = h ? m2.y : m2.x;
                    *reinterpret_cast<uint2 *>(a_tile + sw128(g + 8 * rr, 4 * hsel + 2 * h + (t >> 1)) + (t & 1) * 8) =
                        make_uint2(nibble_h2(v0, qm, and_or(b0 << lsh, hm, kc.magic), s, c, m),
                                   nibble_h2(v0 >> 8, qm, and_or(b0 >> rsh, hm, kc.magic), s, c, m));
                }
            }
        }
    }
};
// Q8_0: table rows of four blocks of 32 columns (d, d)
template <> struct HalfRecord<YUUKA_DTYPE_Q8_0> {
    static constexpr int DS = 16, TAB = 16 * DS;
    uint4 g0, g1, h0, h1;
    uint2 d;
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        const uint4 * p = reinterpret_cast<const uint4 *>(rec);
        g0 = p[(2 * half) * 32 + lane];
        g1 = p[(2 * half + 1) * 32 + lane];
        h0 = p[(4 + 2 * half) * 32 + lane];
        h1 = p[(5 + 2 * half) * 32 + lane];
        d = reinterpret_cast<const uint2 *>(p + 256 + (lane & 15))[half];
    }
    __device__ void header(int lane, int, uint8_t * tab) const {
        const uint32_t v = lane < 16 ? d.x : d.y;
        reinterpret_cast<uint2 *>(tab + (lane & 15) * DS)[lane >> 4] = make_uint2(dup_lo(v), dup_hi(v));
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts &, uint8_t * a_tile) const {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int n = k ^ (g & 1);  // block 2C + n
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint4 q = rr ? (C ? h1 : h0) : (C ? g1 : g0);
                const uint32_t s = reinterpret_cast<const uint32_t *>(tab + (g + 8 * rr) * DS)[2 * C + n];
                const uint32_t v0 = (n ? q.z : q.x) ^ 0x80808080u, v1 = (n ? q.w : q.y) ^ 0x80808080u;
                *reinterpret_cast<uint4 *>(a_tile + sw128(g + 8 * rr, 4 * n + t)) =
                    make_uint4(h2_mul(h2_sub(bytes02_h2(v0), H2_1152), s), h2_mul(h2_sub(bytes13_h2(v0), H2_1152), s),
                               h2_mul(h2_sub(bytes02_h2(v1), H2_1152), s), h2_mul(h2_sub(bytes13_h2(v1), H2_1152), s));
            }
        }
    }
};

// The same for tensor memory: a lane takes from shared memory what its part of the fragments is, and 64 columns go out in one
// store (a quarter of the instructions, and none of the bytes that pass through shared memory twice). The values are the same.
// The words of a packed record that lane (g, t) takes for tensor memory: of a 32-column sub-block columns 4t .. 4t + 3 and 16 + 4t ..
// + 3 (its part of two 16 x 16 fragments). `pieces`: 32 pieces of 16 bytes, one per lane (g, t') of the register-fed kernel, which
// takes columns 8t' .. 8t' + 7 of two sub-blocks as words x y and z w: the columns at 4t are a word of piece t / 2, those at 16 + 4t
// the same word two pieces on. (Lanes g, g + 2, g + 4 and g + 6 of a load meet on one bank: sixteen wavefronts instead of four for
// the 512 bytes. A record order without that would have every other kernel read it otherwise.)
__device__ __forceinline__ uint4 fetch_quads(const uint8_t * pieces, int lane) {
    const uint32_t * w = reinterpret_cast<const uint32_t *>(pieces + (lane >> 2) * 64 + (lane & 2) * 8 + (lane & 1) * 4);
    return make_uint4(w[0], w[8], w[2], w[10]);
}

template <int DT> struct TmemRecord;
template <> struct TmemRecord<YUUKA_DTYPE_Q4_K> : HalfRecordK4<YUUKA_DTYPE_Q4_K> {
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        qg = fetch_quads(rec + half * 512, lane);
        qh = fetch_quads(rec + (2 + half) * 512, lane);
        hdr = reinterpret_cast<const uint4 *>(rec)[128 + (lane & 15)];
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint32_t dst) const {
        const int g = lane >> 2;
        const uint32_t v[2][2] = {{C ? qg.z : qg.x, C ? qg.w : qg.y}, {C ? qh.z : qh.x, C ? qh.w : qh.y}};
        uint32_t r[16];
#pragma unroll
        for (int n = 0; n < 2; n++) {  // sub-block 2C + n: low or high nibbles
            const uint32_t mask = n ? kc.mf0 : kc.m0f;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint2 s = reinterpret_cast<const uint2 *>(tab + (g + 8 * rr) * DS)[2 * C + n];
                const uint32_t m = reinterpret_cast<const uint32_t *>(tab + MN_OFF + (g + 8 * rr) * 16)[2 * C + n];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    r[8 * n + 4 * h + 2 * rr] = nibble_h2(v[rr][h], mask, kc.magic, s.x, s.y, m);
                    r[8 * n + 4 * h + 2 * rr + 1] = nibble_h2(v[rr][h] >> 8, mask, kc.magic, s.x, s.y, m);
                }
            }
        }
        tmem_store16(dst, r);
    }
};
template <> struct TmemRecord<YUUKA_DTYPE_Q5_K> : HalfRecordK4<YUUKA_DTYPE_Q5_K> {
    uint4 hi;  // as in HalfRecord, by quads
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        qg = fetch_quads(rec + half * 512, lane);
        qh = fetch_quads(rec + (2 + half) * 512, lane);
        hdr = reinterpret_cast<const uint4 *>(rec)[160 + (lane & 15)];
        hi = fetch_quads(rec + 2048, lane);
        if (half) hi = make_uint4(hi.x >> 4, hi.y >> 4, hi.z >> 4, hi.w >> 4);
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint32_t dst) const {
        const int g = lane >> 2;
        const uint32_t v[2][2] = {{C ? qg.z : qg.x, C ? qg.w : qg.y}, {C ? qh.z : qh.x, C ? qh.w : qh.y}};
        const uint32_t hb[2][2] = {{hi.x, hi.y}, {hi.z, hi.w}};
        uint32_t r[16];
#pragma unroll
        for (int n = 0; n < 2; n++) {  // sub-block 2C + n: low or high nibbles; its bit 2C + n of each byte goes to bit 4 or 8
            const uint32_t mask = n ? kc.mf0 : kc.m0f, hm = n ? kc.h8 : kc.h4;
            const int up = n ? 7 - 2 * C : 4 - 2 * C, down = n ? 1 + 2 * C : 4 + 2 * C;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint2 s = reinterpret_cast<const uint2 *>(tab + (g + 8 * rr) * DS)[2 * C + n];
                const uint32_t m = reinterpret_cast<const uint32_t *>(tab + MN_OFF + (g + 8 * rr) * 16)[2 * C + n];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    r[8 * n + 4 * h + 2 * rr] = nibble_h2(v[rr][h], mask, and_or(hb[rr][h] << up, hm, kc.magic), s.x, s.y, m);
                    r[8 * n + 4 * h + 2 * rr + 1] = nibble_h2(v[rr][h] >> 8, mask, and_or(hb[rr][h] >> down, hm, kc.magic), s.x, s.y, m);
                }
            }
        }
        tmem_store16(dst, r);
    }
};
template <> struct TmemRecord<YUUKA_DTYPE_Q6_K> : HalfRecord<YUUKA_DTYPE_Q6_K> {  // (its pieces are quads already)
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts & kc, uint32_t dst) const {
        const int g = lane >> 2;
        const uint32_t qm = C ? kc.mf0 : kc.m0f, hm = C ? kc.h8 : kc.h4;
        uint32_t r[16];
#pragma unroll
        for (int hsel = 0; hsel < 2; hsel++) {  // sub-block 2C + hsel
            const int lsh = 4 - 2 * hsel, rsh = 4 + 2 * hsel;
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint4 l4 = rr ? lh : lg;
                const uint2 b2 = rr ? hh : hg, m2 = reinterpret_cast<const uint2 *>(tab + MN_OFF + (g + 8 * rr) * MN)[2 * C + hsel];
                const uint4 s2 = reinterpret_cast<const uint4 *>(tab + (g + 8 * rr) * DS)[2 * C + hsel];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t v0 = h ? (hsel ? l4.w : l4.y) : (hsel ? l4.z : l4.x), b0 = h ? b2.y : b2.x;
                    const uint32_t s = h ? s2.z : s2.x, c = h ? s2.w : s2.y, m = h ? m2.y : m2.x;
                    r[8 * hsel + 4 * h + 2 * rr] = nibble_h2(v0, qm, and_or(b0 << lsh, hm, kc.magic), s, c, m);
                    r[8 * hsel + 4 * h + 2 * rr + 1] = nibble_h2(v0 >> 8, qm, and_or(b0 >> rsh, hm, kc.magic), s, c, m);
                }
            }
        }
        tmem_store16(dst, r);
    }
};
template <> struct TmemRecord<YUUKA_DTYPE_Q8_0> : HalfRecord<YUUKA_DTYPE_Q8_0> {
    __device__ void fetch(const uint8_t * rec, int lane, int half) {
        g0 = fetch_quads(rec + (2 * half) * 512, lane);
        g1 = fetch_quads(rec + (2 * half + 1) * 512, lane);
        h0 = fetch_quads(rec + (4 + 2 * half) * 512, lane);
        h1 = fetch_quads(rec + (5 + 2 * half) * 512, lane);
        d = reinterpret_cast<const uint2 *>(rec + 4096 + (lane & 15) * 16)[half];
    }
    template <int C> __device__ void store(int lane, const uint8_t * tab, const DecodeConsts &, uint32_t dst) const {
        const int g = lane >> 2;
        uint32_t r[16];
#pragma unroll
        for (int n = 0; n < 2; n++) {  // block 2C + n
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const uint4 q = rr ? (C ? h1 : h0) : (C ? g1 : g0);
                const uint32_t s = reinterpret_cast<const uint32_t *>(tab + (g + 8 * rr) * DS)[2 * C + n];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t v = (n ? (h ? q.w : q.z) : (h ? q.y : q.x)) ^ 0x80808080u;
                    r[8 * n + 4 * h + 2 * rr] = h2_mul(h2_sub(bytes02_h2(v), H2_1152), s);
                    r[8 * n + 4 * h + 2 * rr + 1] = h2_mul(h2_sub(bytes13_h2(v), H2_1152), s);
                }
            }
        }
        tmem_store16(dst, r);
    }
};

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return (uint32_t)__cvta_generic_to_shared(p); }
constexpr uint32_t WAIT_LIMIT = 1u << 22, WAIT_LIMIT_TEST = 1u << 8;  // polls of some 4 us each: 17 s; with the test hook 1 ms
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
    uint32_t ok = 0;
    for (uint32_t i = 0; i < limit && !ok; i++) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    }
    return ok != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// From the odd CTA: UM_NOTE bytes into the even CTA's `note`, counted by the barrier at this offset there. The count is a
// release at cluster scope (PTX ISA, st.async: "the complete-tx operation on the mbarrier has .release semantics at the
// .cluster scope"), so whoever waits for it with an acquire at that scope sees what this thread has seen. An arrival would
// order nothing between the CTAs at its default scope, and at cluster scope its release takes some 1500 cycles: with one
// thread passing on the stages 9216 x 2560 took 68 us at 576 rows, with two in turn 45, with four 39, and so 34.6 (34.4 with
// arrivals at CTA scope straight from the decode warps).
constexpr uint32_t UM_NOTE = 4;
__device__ __forceinline__ void note_leader(uint32_t note, uint32_t bar) {
    uint32_t remote_note, remote_bar;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_note) : "r"(note), "r"(0u));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_bar) : "r"(bar), "r"(0u));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(remote_note), "r"(1u), "r"(remote_bar)
                 : "memory");
}
// (Only this wait needs the wider scope. What the odd CTA waits for from the even one are completions of asynchronous
// operations, tcgen05.commit, which the waiter of the barrier sees by the rules of those.)
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, uint32_t limit) {
    uint32_t ok = 0;
    for (uint32_t i = 0; i < limit && !ok; i++) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    }
    return ok != 0;
}
// completion of this thread's MMAs so far -> one arrival on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}

__device__ __forceinline__ void umma_f16_pair_tmem(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        :
        : "r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        :
        : "r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

// 32 accumulator values of one weight row (this lane's) for 32 consecutive activation rows, to out[row][n]:
// MODE 0 stores, 1 adds to what is there, 2 stores a K part past L1. `lim` = rows that exist. One pointer step per
// value: per-value bounds, mode and 64-bit index arithmetic cost more than the stores.
template <int MODE>
__device__ __forceinline__ void umma_store_rows(float * dst, int64_t ld, const uint32_t (&v)[32], int lim) {
#pragma unroll
    for (int i = 0; i < 32; i++) {
        if (lim >= 32 || i < lim) {
            const float val = __uint_as_float(v[i]);
            if (MODE == 2) __stcg(dst, val);
            else if (MODE == 1) *dst += val;
            else *dst = val;
        }
        dst += ld;
    }
}

__device__ __forceinline__ void tmem_load32(uint32_t (&v)[32], uint32_t src) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(src)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Walks the work of a pair: tiles (256 weight rows x n_tile activation rows x a part of K) in steps of the number of
// pairs, activation tiles of the same weights first, so that pairs next to each other read the same weights.
struct UmmaWork {
    int item, step, items;
    __device__ UmmaWork(const UParams & p) {
        item = blockIdx.x >> 1;
        step = gridDim.x >> 1;
        items = p.m_blocks * p.n_tiles * p.kparts;
    }
    __device__ bool valid() const { return item < items; }
    __device__ void next() { item += step; }
    __device__ int n0(const UParams & p) const { return (item % p.n_tiles) * p.n_tile; }
    __device__ int part(const UParams & p) const { return (item / p.n_tiles) % p.kparts; }
    __device__ int block(const UParams & p) const { return item / (p.n_tiles * p.kparts); }
    __device__ int sb_begin(const UParams & p) const { return (int)((long long)p.nsb * part(p) / p.kparts); }
    __device__ int sb_end(const UParams & p) const { return (int)((long long)p.nsb * (part(p) + 1) / p.kparts); }
};
// A position in a ring of `depth` stages: `phase` is the parity a consumer waits for, its inverse a producer's.
struct Ring {
    uint32_t at = 0, phase = 0;
    __device__ void next(uint32_t depth) {
        if (++at == depth) {
            at = 0;
            phase ^= 1u;
        }
    }
};

// TMEM: the decoded weights lie in tensor memory, behind the accumulators, instead of in shared memory.
template <int DT, bool TMEM>
__global__ void __launch_bounds__(UM_THREADS, 1) gemm_umma_kernel(const UParams p, const __grid_constant__ CUtensorMap xmap) {
    using C = Codec<DT>;
    using S = UmmaStage<DT>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the swizzled stages need 1024-byte alignment
    __shared__ __align__(8) uint64_t empty_bar[UM_MAX_STAGES];  // the tensor pipe has read the stage
    __shared__ __align__(8) uint64_t full_bar[UM_MAX_STAGES];   // this CTA's weights and activations are in the stage (even CTA: both CTAs')
    __shared__ __align__(8) uint64_t raw_full[UM_MAX_RAW], raw_empty[UM_MAX_RAW];
    __shared__ __align__(8) uint64_t acc_full[UM_MAX_ACC], acc_empty[UM_MAX_ACC]; // accumulators: finished by the MMAs, read by the epilogue
    __shared__ uint32_t tmem_slot, odd_note[UM_MAX_STAGES];  // (the notes' contents are not read)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform for the compiler too)
    const uint32_t rank = blockIdx.x & 1u;  // clusters are pairs along x
    const uint32_t half_n = (uint32_t)p.n_tile >> 1, b_bytes = half_n * 128u, a_bytes = TMEM ? 0u : (uint32_t)UM_A_BYTES, stage_bytes = a_bytes + b_bytes;
    uint8_t * raw = smem + (size_t)p.stages * stage_bytes;
    uint8_t * tabs = raw + (size_t)p.raw_stages * S::RAW_BYTES;

    if (threadIdx.x == 0) {
        for (int s = 0; s < UM_MAX_STAGES; s++) {
            mbar_init(smem_u32(&empty_bar[s]), 1);
            mbar_init(smem_u32(&full_bar[s]), UM_TILES + 1);
        }
        for (int s = 0; s < UM_MAX_RAW; s++) {
            mbar_init(smem_u32(&raw_full[s]), 1);
            mbar_init(smem_u32(&raw_empty[s]), UM_DW);
        }
        for (int s = 0; s < UM_MAX_ACC; s++) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), UM_EW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == UM_WARP_MMA) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers are set up
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = tmem_slot, smem_base = smem_u32(smem);
    const uint32_t acc_cols = p.acc_cols, n_acc = p.n_acc, a_base = taddr + n_acc * acc_cols;
    const int n_tiles16 = (p.N + 15) >> 4;
    const size_t rec_row = (size_t)p.nsb * C::REC;
    const uint32_t limit = p.drop_copies ? WAIT_LIMIT_TEST : WAIT_LIMIT;
    bool expired = false;
    // (by whole warps, whose lanes agree on the outcome)
    auto wait = [&](const uint64_t & bar, uint32_t parity) {
        expired = __any_sync(0xffffffffu, !mbar_wait(smem_u32(&bar), parity, limit));
        return !expired;
    };

    pdl_trigger();
    // (the copy and issue warps walk their loops whole, so that addresses and descriptors stay in uniform registers; one
    // lane issues: a loop of that lane alone spent 85 cycles on each MMA)
    if (warp == UM_WARP_RAW) {
        // ---------------- packed weights: they do not depend on the previous kernel ----------------
        Ring ring;
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            const int rt = min((wk.block(p) * 2 + (int)rank) * UM_TILES + (lane & (UM_TILES - 1)), n_tiles16 - 1), sb1 = wk.sb_end(p);
            const uint8_t * src = p.w + rt * rec_row;
            for (int sb = wk.sb_begin(p); sb < sb1; sb++) {
                if (!wait(raw_empty[ring.at], ring.phase ^ 1u)) break;
                const uint32_t bar = smem_u32(&raw_full[ring.at]);
                if (lane == 0) mbar_expect(bar, S::RAW_BYTES);
                __syncwarp();
                if (lane < UM_TILES)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     smem_u32(raw + (size_t)ring.at * S::RAW_BYTES) + (uint32_t)(lane * C::REC)),
                                 "l"(src + (size_t)sb * C::REC), "r"((uint32_t)C::REC), "r"(bar)
                                 : "memory");
                ring.next(p.raw_stages);
            }
        }
    } else if (warp == UM_WARP_X) {
        // ---------------- activations: this CTA's half of the tile's rows ----------------
        pdl_wait();
        Ring ring;
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            const int row = wk.n0(p) + (int)(rank * half_n), sb1 = wk.sb_end(p);
            for (int col = wk.sb_begin(p) * 256; col < sb1 * 256; col += UM_KC) {
                if (!wait(empty_bar[ring.at], ring.phase ^ 1u)) break;
                const uint32_t bar = smem_u32(&full_bar[ring.at]);
                if (lane == 0 && !(p.drop_copies && rank == 0)) {
                    mbar_expect(bar, b_bytes + (rank == 0 ? UM_NOTE : 0u));
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                        :
                        : "r"(smem_base + ring.at * stage_bytes + a_bytes), "l"(&xmap), "r"(col), "r"(row), "r"(bar)
                        : "memory");
                }
                __syncwarp();
                ring.next(p.stages);
            }
        }
    } else if (warp == UM_WARP_MMA && rank == 0) {
        // ---------------- MMAs of the pair ----------------
        Ring ring, acc;
        const uint64_t da0 = umma_desc_sw128(smem_base), db0 = umma_desc_sw128(smem_base + a_bytes);
        const uint32_t step = stage_bytes >> 4;
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            if (!wait(acc_empty[acc.at], acc.phase ^ 1u)) break;
            uint32_t d = taddr + acc.at * acc_cols, keep = 0;
            const int chunks = (wk.sb_end(p) - wk.sb_begin(p)) * 4, second = p.halves ? (p.nsb >> 1) * 4 : chunks;
            for (int c = 0; c < chunks; c++) {
                if (c == second) {  // the other half of K goes to an accumulator of its own
                    if (elect_one()) umma_commit_pair(smem_u32(&acc_full[acc.at]));
                    __syncwarp();
                    acc.next(n_acc);
                    if (!wait(acc_empty[acc.at], acc.phase ^ 1u)) break;
                    d = taddr + acc.at * acc_cols;
                    keep = 0;
                }
                expired = __any_sync(0xffffffffu, !mbar_wait_cluster(smem_u32(&full_bar[ring.at]), ring.phase, limit));
                if (expired) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = da0 + (uint64_t)(ring.at * step), db = db0 + (uint64_t)(ring.at * step);
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < UM_KC / 16; j++) {
                        if constexpr (TMEM) umma_f16_pair_tmem(d, a_base + ring.at * UM_A_COLS + (uint32_t)(j * 8), db + (uint64_t)(j * 2), p.idesc, j > 0 ? 1u : keep);
                        else umma_f16_pair(d, da + (uint64_t)(j * 2), db + (uint64_t)(j * 2), p.idesc, j > 0 ? 1u : keep);
                    }
                    umma_commit_pair(smem_u32(&empty_bar[ring.at]));
                }
                __syncwarp();
                keep = 1;
                ring.next(p.stages);
            }
            if (expired) break;
            if (elect_one()) umma_commit_pair(smem_u32(&acc_full[acc.at]));
            __syncwarp();
            acc.next(n_acc);
        }
    } else if (warp == UM_WARP_MMA) {
        // ---------------- odd CTA: its part of a stage is there (and, at the start of an accumulator, its epilogue has
        // read what the accumulator held) -> the even CTA's barrier ----------------
        Ring ring, acc;
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            const int chunks = (wk.sb_end(p) - wk.sb_begin(p)) * 4, second = p.halves ? (p.nsb >> 1) * 4 : chunks;
            for (int c = 0; c < chunks; c++) {
                if (c == 0 || c == second) {
                    if (!wait(acc_empty[acc.at], acc.phase ^ 1u)) break;
                    acc.next(n_acc);
                }
                if (!wait(full_bar[ring.at], ring.phase)) break;
                if constexpr (TMEM) {  // the decode warps' stores come before the note
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                }
                if (lane == 0) note_leader(smem_u32(&odd_note[ring.at]), smem_u32(&full_bar[ring.at]));
                __syncwarp();
                ring.next(p.stages);
            }
        }
    } else if (warp < UM_DW) {
        // ---------------- decode ----------------
        // Stages 2 half, 2 half + 1 of every superblock. (In tensor memory a warp reaches the 32 lanes of its number mod 4: two tiles.)
        const int tile = TMEM ? 2 * (warp & 3) + ((warp >> 2) & 1) : warp >> 1, half = TMEM ? warp >> 3 : warp & 1;
        const uint32_t lanes = (uint32_t)(tile * 16) << 16;
        uint8_t * tab = tabs + warp * HalfRecord<DT>::TAB;
        const DecodeConsts kc = p.kc;
        Ring ring, rr;
        if (half) {
            ring.next(p.stages);
            ring.next(p.stages);
        }
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            for (int n = wk.sb_end(p) - wk.sb_begin(p); n > 0; n--) {
                std::conditional_t<TMEM, TmemRecord<DT>, HalfRecord<DT>> r;
                if (!wait(raw_full[rr.at], rr.phase)) break;
                r.fetch(raw + (size_t)rr.at * S::RAW_BYTES + tile * C::REC, lane, half);
                r.header(lane, half, tab);
                __syncwarp();  // the table is complete, and every lane has its part of the record
                if (lane == 0) mbar_arrive(smem_u32(&raw_empty[rr.at]));
                rr.next(p.raw_stages);
                auto chunk = [&](auto c) {
                    if (expired || !wait(empty_bar[ring.at], ring.phase ^ 1u)) return;
                    if constexpr (TMEM) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        r.template store<decltype(c)::value>(lane, tab, kc, a_base + ring.at * UM_A_COLS + lanes);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    } else {
                        r.template store<decltype(c)::value>(lane, tab, kc, smem + (size_t)ring.at * stage_bytes + tile * 16 * 128);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&full_bar[ring.at]));
                    ring.next(p.stages);
                };
                chunk(std::integral_constant<int, 0>());
                chunk(std::integral_constant<int, 1>());
                if (expired) break;
                ring.next(p.stages);
                ring.next(p.stages);
            }
        }
    } else {
        // ---------------- epilogue: tensor-memory lane = weight row, column = activation row ----------------
        pdl_wait();
        const int quad = warp & 3;
        Ring acc;
        for (UmmaWork wk(p); wk.valid() && !expired; wk.next()) {
            const uint32_t first = acc.at;
            if (!wait(acc_full[first], acc.phase)) break;
            if (p.halves) {
                acc.next(n_acc);
                if (!wait(acc_full[acc.at], acc.phase)) break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int n = (wk.block(p) * 2 + (int)rank) * UM_ROWS + quad * 32 + lane, m0 = wk.n0(p);
            const bool split = p.kparts > 1;
            float * base = split ? p.partial + (size_t)wk.part(p) * p.M * p.N : p.out;
            const int64_t ld = split ? p.N : p.ldo;
            for (int c0 = 0; c0 < p.n_tile && m0 + c0 < p.M; c0 += 32) {
                uint32_t v[32];
                const uint32_t from = taddr + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
                tmem_load32(v, from + first * acc_cols);
                if (p.halves) {
                    uint32_t v2[32];
                    tmem_load32(v2, from + acc.at * acc_cols);
#pragma unroll
                    for (int e = 0; e < 32; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(v2[e]));
                }
                if (n < p.N) {
                    float * dst = base + (int64_t)(m0 + c0) * ld + n;
                    const int lim = min(p.M - m0, p.n_tile) - c0;
                    if (split) umma_store_rows<2>(dst, ld, v, lim);
                    else if (p.accumulate) umma_store_rows<1>(dst, ld, v, lim);
                    else umma_store_rows<0>(dst, ld, v, lim);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&acc_empty[first]));
                if (p.halves) mbar_arrive(smem_u32(&acc_empty[acc.at]));
            }
            acc.next(n_acc);
        }
    }
    if (expired) atomicExch(&g_gemm_wait_expired, 3);
    // every MMA has completed (the epilogue has waited for the last one of each accumulator); nothing of this CTA is touched by
    // the other one after the barrier
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    if (warp == UM_WARP_MMA)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512u) : "memory");
}

// Sum of the K parts of a split tensor-memory GEMM, in part order: out[tok][n] (+)= sum over parts of
// partial[part][tok][n], by the whole machine (the last CTA of a block doing it alone took longer than the decode the
// split saves). V = 4 where rows allow 16-byte accesses.
template <int V>
__global__ void __launch_bounds__(256) umma_reduce_kernel(float * __restrict__ out, int64_t ldo, const float * __restrict__ partial,
                                                          int parts, int M, int N, int accumulate) {
    pdl_entry();
    const int nv = N / V;
    const int64_t total = (int64_t)M * nv;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int tok = (int)(i / nv), n = (int)(i - (int64_t)tok * nv) * V;
        float * dst = out + (int64_t)tok * ldo + n;
        float sum[V];
#pragma unroll
        for (int e = 0; e < V; e++) sum[e] = 0.0f;
        for (int part = 0; part < parts; part++) {
            const float * src = partial + ((size_t)part * M + tok) * N + n;
            if constexpr (V == 4) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(src));
                sum[0] += v.x;
                sum[1] += v.y;
                sum[2] += v.z;
                sum[3] += v.w;
            } else {
                sum[0] += __ldcg(src);
            }
        }
#pragma unroll
        for (int e = 0; e < V; e++) dst[e] = accumulate ? dst[e] + sum[e] : sum[e];
    }
}

}  // namespace yk
