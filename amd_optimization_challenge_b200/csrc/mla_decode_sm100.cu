// Stage-1 MLA decode on the 5th-generation tensor cores (tcgen05) with TMEM accumulators, for every pair of
// cache format (e4m3, MXFP4, hybrid) and query format (e4m3, bf16).
//
// Swap-AB formulation, so that the 128-row MMA dimension is filled by KV tokens (QK) and output dims (PV) and the
// small dimension (16, 32 or 64 query rows) is the MMA N:
//     S^T[tok x NQ]   = K[tok x 576] . Q^T           A = K tile (K-major, 128B swizzle), B = Q
//     O^T[512 x OB]  += V^T[512 x tok] . P^T         A = the same tile read MN-major (V = first 512 dims of K),
//                                                    B = P written by the softmax warps, 4 M-blocks of 128 dims
// Both run as kind::f8f6f4 on e4m3 operands with fp32 accumulation in TMEM.
//   * P is split into two e4m3 terms (~8 significant bits): for 16 / 32 rows P = hi + lo/16 as the two halves of the
//     MMA's 2N columns, for 64 rows hi and lo (unscaled) are two k-steps into the same columns (side by side, O alone
//     would fill the 512 TMEM columns); how far below the maximum the eight bits reach: Cfg::P_SCALE_LOG2.
//   * A bf16 Q is split the same way: Q = (hi + lo/16) / s, s a power of two per group of N rows; the QK MMA then has
//     2N columns and the softmax adds the two halves.  (No tensor-core kind mixes bf16 with fp8 / fp4 operands.)
//   * MXFP4 / hybrid cache rows become e4m3 operand bytes in "feed" warps: all blocks of a 16-token unit share one
//     exponent frame, byte value = e2m1 * 2^(scale - E_unit + 6) with E_unit the largest E8M0 byte of the unit, exact in
//     e4m3 for blocks up to 14 binades below the largest.  The softmax thread of a token applies 2^(E_unit - 133) to its
//     scores and 2^(E_unit - E_run) to its probabilities, E_run being the frame O is held in (O is rescaled in TMEM when
//     a later tile has a larger frame, like the softmax re-centering).
//   * hybrid cache: the 64 rope dims are e4m3 with a per-tensor scale that is not a power of two, so their QK k-steps
//     accumulate into TMEM columns of their own and the softmax adds a_lat * S_lat + a_rope * S_rope.
//
// The CTA walks its span of tiles as one continuous stream, also across the boundary between two sequences: the roles
// run their own loops over the tiles and meet only through mbarriers.
//
// Roles: SW softmax warps (one or two warpgroups; they also load and convert the Q rows of each sequence and write O)
//        FW feed warps: fill the operand stages (TMA row gathers / boxes for an e4m3 cache, conversion of fetched units else)
//        1 QK warp, 1 PV warp (the whole warp runs the loop, one elected lane issues), for a block-scaled cache 2 fetch warps
//        (the PV warp, or the first fetch warp, searches the CTA's span before that)
// What bounds it, and microseconds a call before (a kernel per family, maximum of Q and merge as launches of their own, one
// issuing warp) and now: e4m3 256 x 8192 the HBM rate (264 -> 210), 128 heads over an e4m3 cache the chain load -> QK -> softmax -> PV
// of two stages (236 -> 80), MXFP4 64 x 8192 the same chain with the conversion in it (96 -> 65), MXFP4 8 x 131072 with two
// queries and hybrid 128 heads that chain and shared memory, conversion and MMA operands alike (214 -> 147, 640 -> 390), e4m3 4 x 1024 latencies
// (23.5 -> 10.0 to 10.6).  Long calls vary by 8 % from GPU to GPU.
// Synchronisation is mbarrier based; every such wait is bounded and on expiry sets a status word.  The two waits for other CTAs
// are shorter, and who gives up goes on without them and sets no status: see MlaParams::meet_cycles.
//
// Role in the reference: the split-KV stage-1 kernels (mixed-mla/submission.py:122-250,
// mixed-mla/versions/hip_mxfp4_v5/submission.py:214-656) and their block decode (mixed-mla/triton_mla_mxfp4.py:20-67).
#include <cuda.h>
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "sm100_ptx.cuh"

namespace b200mla {
namespace sm100 {

constexpr int NS_MAX = 3;                 // operand stages
constexpr int UNIT_TOK = 16;              // tokens per unit of the feed warps
constexpr int RAW_MAX = 10;               // landing buffers of a block-scaled cache
constexpr int SMEM_LIMIT = 232448;        // opt-in shared memory per CTA
constexpr int E_BIAS = 127 + 6;           // operand bytes of a block-scaled unit are in units of 2^(E_unit - E_BIAS)

// Outcome of the CTAs' meeting for one of them: bits, all clear where every CTA came in time.  MEET_LEFT: it has left before the last
// came.  MEET_LATE: others had left before it came.  MEET_NO_TABLE: MlaParams::seq_ctas is not there yet.
enum { MEET_LEFT = 1, MEET_LATE = 2, MEET_NO_TABLE = 4 };
constexpr int NO_BIT_CYCLES = 20000;      // 10 us, what the CTAs of an ordinary call are apart: as long a CTA only counts as come
enum { MASK_ARRIVED = 0, MASK_LATE_ARRIVED = 1, MASK_LATE_LEFT = 2 };      // see Misc::mask

struct Misc {
    uint64_t kv_full[NS_MAX], kv_empty[NS_MAX][4], s_full[2], s_empty[2], p_full[NS_MAX], p_empty[NS_MAX], q_full, o_free;
    uint64_t raw_full[RAW_MAX], raw_empty[RAW_MAX];
    int raw_slot[RAW_MAX][UNIT_TOK];      // cache rows of the unit in each landing buffer
    uint32_t tmem_base;
    int abort_flag;
    int meet;                             // outcome of the CTAs' meeting (MEET_*)
    int q_share;                          // share of Q that this CTA looks at for another one, -1: all have been looked at
    int span[4];                          // first sequence, its first global tile, first and end tile of this CTA
    unsigned int q_red[8];                // cross-warp maximum of a split Q
    long long q_off[4];                   // element offset of each 16-row chunk of this row group inside a sequence's Q
    __align__(16) int tile_exp[NS_MAX][8];    // exponent frame of each unit of the tile in each stage
    __align__(16) float nm[2][2][32];     // P_SCALE_LOG2 - reference maximum per query row, 0 before the first tile: [warpgroup][double buffer][row]
    __align__(16) float shift[2][32];     // what nm moves by at a tile
    __align__(16) float fac[2][32];       // per-row factors published to a warpgroup
    __align__(16) float red[2][4][32];    // cross-warp column reductions
    // The CTAs that had come when this one left; those that had come, and those that had left, when it came.  In memory that the
    // fetch warps are done with by then.
    __device__ __forceinline__ int (&mask(int which))[UNIT_TOK] { return raw_slot[which]; }
};
static_assert(SYNC_MASK_WORDS <= UNIT_TOK, "Misc::mask");

template <int N_, int KVFMT, int QFMT>
struct Cfg {
    static constexpr int N = N_;
    static constexpr bool QSPLIT = QFMT == Q_BF16, XF = KVFMT != KV_E4M3, ROPE_SEP = KVFMT == KV_HYBRID;
    static constexpr int NQ = N * (QSPLIT ? 2 : 1);               // Q rows in shared memory = columns of one S accumulator
    static constexpr int SC = NQ * (ROPE_SEP ? 2 : 1);            // S columns per buffer
    static constexpr int SMG = N == 16 ? 1 : 2;                   // softmax warpgroups (warps w and w + 4 reach the same TMEM lanes)
    static constexpr int NC = N / SMG;                            // query rows per softmax thread
    // Tokens per tile and operand stages.  128 x 2: every row of the 128-row MMAs is a token, which matters where shared
    // memory bandwidth sets the pace (an MMA reads its whole A operand whatever the rows hold).  96 x 3 for an e4m3 cache
    // and few rows, which HBM paces: more bytes in flight, finer schedule; rows 96..127 of a QK operand are then whatever
    // follows the panel in shared memory, and their scores are never read.
    static constexpr int TILE = (!XF && N < 64) ? 96 : 128, NS = TILE == 96 ? 3 : 2;
    static constexpr int UNITS = TILE / UNIT_TOK;                 // units of 16 tokens
    static constexpr int PANEL_BYTES = TILE * 128;                // dims 128j..128j+127: 128-byte rows, 128B swizzle
    static constexpr int ROPE_PANEL_BYTES = TILE * 64;            // dims 512..575: 64-byte rows, 64B swizzle
    static constexpr int STAGE_BYTES = 4 * PANEL_BYTES + ROPE_PANEL_BYTES;
    static constexpr bool MERGED = N == 64;
    static constexpr int OB = MERGED ? N : 2 * N;                 // TMEM columns of one O block
    // A probability p (relative to the reference maximum) is stored as 2^P_SCALE_LOG2 p; a score more than RECENTER log2 units above
    // the reference maximum moves it.  2^(P_SCALE_LOG2 + RECENTER) must stay below 448.  The smallest step of the stored pair is
    // 2^-13 with lo / 16 in columns of its own, 2^-9 where lo shares hi's columns (MERGED): there the larger factor keeps the same
    // 2^-17 below the reference maximum, at the price of moving it at most tiles (48 ragged sequences of 128 heads: 81 us; 85 when
    // O was rescaled before the probabilities were computed, all of it, and the scores read three times; less with 2^4, but like
    // keys 12 binades down come out 28 % wrong).  Block-scaled caches at 64 rows keep 2^4, i.e. 2^-13.
    static constexpr bool DEEP = MERGED && !XF;
    static constexpr float P_SCALE_LOG2 = DEEP ? 8.0f : 4.0f, RECENTER = DEEP ? 0.75f : 4.0f;
    static constexpr int P_CHUNK_BYTES = TILE * 16;               // 16 columns x TILE tokens
    static constexpr int P_BUF_BYTES = (2 * N / 16) * P_CHUNK_BYTES;
    static constexpr int P_BUFS = XF && N > 16 ? 1 : NS;          // single where the landing buffers need the room
    static constexpr int Q_PANEL_BYTES = NQ * 128;
    static constexpr int Q_BYTES = NQ * QK_DIM;                   // four 128B-swizzled panels and one 64B-swizzled
    // Landing buffer of one unit: 16 code rows (see raw_chunk), then 32 bytes around each E8M0 row.
    static constexpr int CODE_BYTES = KVFMT == KV_MXFP4 ? 288 : 256;
    static constexpr int RAW_BYTES = XF ? UNIT_TOK * (CODE_BYTES + 32) : 0;
    static constexpr int OFF_Q = NS * STAGE_BYTES;
    static constexpr int OFF_P = OFF_Q + Q_BYTES;
    static constexpr int OFF_RAW = OFF_P + P_BUFS * P_BUF_BYTES;
    // Softmax and feed warps: 16 warps in all at most, because registers are handed out per scheduler - 128 a thread up to
    // four warps each, 96 with a fifth (the 64-row kernels then spilled 1.2 KB a thread).
    // An e4m3 cache has at most as many feed warps as a tile has units: with ten for six units the copies of the second tile went
    // out among those of the first, which landed later for it (32 x 4096: 27.0 us, 26.2 with six).
    static constexpr int SW = 4 * SMG, NAUX = XF ? 3 : 1, FW_ROOM = 15 - NAUX - SW, FW_MAX = !XF && FW_ROOM > UNITS ? UNITS : FW_ROOM;
    static constexpr int RAW_FIT = XF ? (SMEM_LIMIT - OFF_RAW - (int)sizeof(Misc)) / (XF ? RAW_BYTES : 1) : FW_MAX;
    // Even numbers of landing buffers and of feed warps, no more warps than buffers.  A barrier's phase parity tells only
    // neighbouring rounds of a buffer apart, so nobody may wait for a round while the one before the previous is open:
    //   fetch   unit u is fetched by auxiliary warp u % 2, which then fetches every round of buffer u % NBUF, in order
    //   feed    a warp that waits for unit u has had unit u - FW, fetched by the same auxiliary warp after (or as) u - NBUF
    static constexpr int NBUF = XF ? (RAW_FIT < RAW_MAX ? RAW_FIT : RAW_MAX) & ~1 : 0;
    static constexpr int FW = !XF ? FW_MAX : (NBUF < FW_MAX ? NBUF : FW_MAX) & ~1;
    static_assert(!XF || (NBUF % 2 == 0 && FW % 2 == 0 && FW >= 2 && FW <= NBUF && UNITS % 2 == 0), "landing buffer rounds");
    static constexpr int QK_WARP = SW + FW, PV_WARP = QK_WARP + 1, AUX_WARP = XF ? PV_WARP + 1 : PV_WARP;
    static constexpr int THREADS = 32 * (SW + FW + 1 + NAUX);
    static constexpr int OFF_MISC = OFF_RAW + NBUF * RAW_BYTES;
    static constexpr int SMEM = OFF_MISC + (int)sizeof(Misc);
    static constexpr int TMEM_O = 2 * SC;
    static constexpr int TMEM_NEED = 2 * SC + 4 * OB;
    static constexpr int TMEM_COLS = TMEM_NEED <= 128 ? 128 : (TMEM_NEED <= 256 ? 256 : 512);
    static_assert(TILE % 32 == 0 && TILE <= 128 && UNITS <= 8 && PANEL_BYTES % 1024 == 0 && ROPE_PANEL_BYTES % 512 == 0, "operand layout");
    static_assert(TMEM_NEED <= 512, "TMEM columns");
    static_assert(SMEM <= SMEM_LIMIT && OFF_MISC % 16 == 0 && (!XF || NBUF >= 4), "shared memory");
};

// e4m3 cache: row gathers (boxes of one row) and boxes of 16 rows of the latent and rope panels
struct Maps { CUtensorMap lat, rope, lat_box, rope_box; };

// Byte offset of 16-byte column c of row t (0..15) in a landing buffer.  The feed warps read four columns of rows t and
// t + 1 (t even) at once, which must not share banks: rows of 288 bytes are placed so that the two are half a bank cycle
// apart, rows of 256 have the columns of odd rows exchanged in groups of four.
template <int ROW>
__device__ __forceinline__ constexpr int raw_chunk(int t, int c) {
    return ROW == 288 ? ((t & ~3) | ((t & 1) << 1) | ((t >> 1) & 1)) * 288 + c * 16 : t * 256 + ((c ^ ((t & 1) << 2)) * 16);
}

// 2^e as a float; 0 below the normal range
__device__ __forceinline__ float pow2i(int e) { return e < -126 ? 0.0f : __int_as_float((min(e, 127) + 127) << 23); }

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// 32 e2m1 codes (one uint4, even element in the low nibble) -> 32 e4m3 bytes, value = code * 2^k, k <= 6.
// Magnitudes: a byte permute through the 8-entry table of this block's k.  For k >= -5 every non-zero entry is a
// normal e4m3 number, i.e. the k = 0 bytes plus 8k; below that (ANY_K) the table comes from the rounding conversion
// (entries that e4m3 cannot hold exactly are rounded or flushed).  Signs: a byte permute in sign-replication
// mode turns nibble bit 3 (of the code word and of the word shifted by 4) into 0xff / 0x00 bytes.
// The two forms are separate because a choice inside keeps the compiler from interleaving blocks: nine blocks took one
// warp 1310 cycles with it, 811 without.
template <bool ANY_K>
__device__ __forceinline__ void dequant_block(const uint4& v, int k, uint4& lo, uint4& hi) {
    uint32_t t0 = 0x3C383000u + (uint32_t)(k * 0x08080800);      // 0, .5, 1, 1.5
    uint32_t t1 = 0x4C484440u + (uint32_t)(k * 0x08080808);      // 2, 3, 4, 6
    if (ANY_K && k < -5) {
        const float sc = pow2i(max(k, -40));
        t0 = pack_e4m3x4(0.0f, 0.5f * sc, sc, 1.5f * sc);
        t1 = pack_e4m3x4(2.0f * sc, 3.0f * sc, 4.0f * sc, 6.0f * sc);
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t m = w[i] & 0x77777777u, w4 = w[i] << 4;
        o[2 * i] = prmt(t0, t1, m) | (prmt(w4, w[i], 0xD9C8u) & 0x80808080u);
        o[2 * i + 1] = prmt(t0, t1, m >> 16) | (prmt(w4, w[i], 0xFBEAu) & 0x80808080u);
    }
    lo = make_uint4(o[0], o[1], o[2], o[3]);
    hi = make_uint4(o[4], o[5], o[6], o[7]);
}

// ----------------------------------------------------------------------------------------------
// Span search.  One warp finds this CTA's part of the schedule straight from kv_indptr (no table in shared memory, so
// any batch fits): lane l sums the tiles of the sequences [l*per, (l+1)*per), a warp scan gives their prefix, and each
// end of the span is located in one lane's range and then inside it, 32 sequences at a time.
// ----------------------------------------------------------------------------------------------
template <int TILE>
__device__ __forceinline__ int tiles_of_len(int len) { return len > 0 ? (len + TILE - 1) / TILE : 0; }

template <int TILE>
__device__ __forceinline__ int seq_tiles(const int* ip, int b, int end) {
    return b < end ? tiles_of_len<TILE>(load_global(ip + b + 1) - load_global(ip + b)) : 0;
}
__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// The table of the merge, by the lanes of a warp: the CTAs of this lane's sequences [s0, s1), the first of which begins at tile t.
template <int TILE>
__device__ __forceinline__ void write_seq_ctas(const MlaParams& p, const Sched& sc, int s0, int s1, int t) {
    for (int b = s0; b < s1; ++b) {
        const int n = seq_tiles<TILE>(p.kv_indptr, b, s1);
        p.seq_ctas[b] = seq_span(b, t, t + n, sc);
        t += n;
    }
    __syncwarp();
}

// This lane's sequences [s0, s1), and the tiles up to and with them.
template <int TILE>
__device__ __forceinline__ int lane_tiles(const MlaParams& p, int lane, int& s0, int& s1, int& mine) {
    const int per = (p.batch + 31) >> 5;
    s0 = min(lane * per, p.batch); s1 = min(s0 + per, p.batch);
    mine = 0;
    for (int b = s0; b < s1; ++b) mine += seq_tiles<TILE>(p.kv_indptr, b, s1);
    return warp_scan(mine, lane);
}

template <int TILE>
__device__ __forceinline__ void find_span(const MlaParams& p, int w, int G, int lane, int (&span)[4], bool write_table) {
    const int batch = p.batch, per = (batch + 31) >> 5;
    int s0, s1, mine;
    const int incl = lane_tiles<TILE>(p, lane, s0, s1, mine);
    const int tt = __shfl_sync(0xffffffffu, incl, 31);
    const Sched sc = make_sched(tt, batch, G, p.seq_units);
    int t_first = 0, t_end = 0, seq = 0, seq_t0 = 0;
#pragma unroll 1
    for (int e = 1; e >= 0; --e) {                                // the end first, so that seq / seq_t0 end up describing the start
        const int u = unit_begin(w + e, sc);
        int t = tt;
        if (u < sc.units) {
            const int l = __ffs(__ballot_sync(0xffffffffu, incl + sc.k * s1 > u)) - 1;
            int before = __shfl_sync(0xffffffffu, incl - mine, l), b0 = min(l * per, batch);      // tiles before sequence b0
            const int bend = min(b0 + per, batch);
            for (; per > 1 && b0 < bend; b0 += 32) {
                const int n = seq_tiles<TILE>(p.kv_indptr, b0 + lane, bend), sum = before + warp_scan(n, lane);
                const unsigned int hit = __ballot_sync(0xffffffffu, b0 + lane < bend && sum + sc.k * (b0 + lane + 1) > u);
                if (hit) {
                    const int h = __ffs(hit) - 1;
                    before = __shfl_sync(0xffffffffu, sum - n, h);
                    b0 += h;
                    break;
                }
                before = __shfl_sync(0xffffffffu, sum, 31);
            }
            seq = b0;
            seq_t0 = before;
            t = max(seq_t0, u - sc.k * (b0 + 1));
        }
        if (e) t_end = t; else t_first = t;
    }
    span[0] = seq; span[1] = seq_t0; span[2] = t_first; span[3] = t_end;
    if (write_table) {
        write_seq_ctas<TILE>(p, sc, s0, s1, incl - mine);
        if (lane == 0 && p.fused) red_release(p.status + SYNC_TABLE, 1);      // cumulative: __syncwarp orders the lanes' stores before it
    }
}

// largest magnitude of eight bf16 values, as its bit pattern (they order like their bit patterns)
__device__ __forceinline__ unsigned int bf16x8_amax_bits(const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    unsigned int m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) m = max(m, max(w[k] & 0x7fffu, (w[k] >> 16) & 0x7fffu));
    return m;
}
// Maximum of Q that the CTAs find together, as a bit pattern.
__device__ __forceinline__ unsigned int amax_bits(const int* status) { return *reinterpret_cast<const volatile unsigned int*>(status + SYNC_AMAX); }
// One thread: a share of Q that is not marked in SYNC_AMAX_DONE, another one for each CTA as far as there are that many; -1 if there is
// none, and then the other CTAs need not look either.
__device__ __forceinline__ int open_share(int* status, int n_cta, int cta) {
    auto open = [&](int i) {
        const unsigned int all = n_cta - 32 * i >= 32 ? ~0u : (1u << (n_cta - 32 * i)) - 1u;
        return ~(unsigned int)load_acquire(status + SYNC_AMAX_DONE + i) & all;
    };
    for (;;) {
        int n = 0;
#pragma unroll 1
        for (int i = 0; 32 * i < n_cta; ++i) n += __popc(open(i));
        if (n == 0) break;
        int k = cta % n;
#pragma unroll 1
        for (int i = 0; 32 * i < n_cta; ++i) {
            unsigned int o = open(i);
            const int here = __popc(o);
            if (k < here) {
                for (; k > 0; --k) o &= o - 1;
                return 32 * i + __ffs(o) - 1;
            }
            k -= here;
        }                                                         // marked in between, at least one each time: look again
    }
    atomicOr(status + SYNC_AMAX_COUNT, 0x8000);
    return -1;
}
// The softmax warps (SW of them, the first of the CTA) look at share c of a dense bf16 Q of `rows` rows: its maximum goes to SYNC_AMAX,
// then its bit to SYNC_AMAX_DONE.  Twice does no harm.
template <int SW>
__device__ __forceinline__ void look_at_share(const uint4* q8, int rows, int* status, unsigned int n_cta, unsigned int c, unsigned int* q_red) {
    constexpr int ST = 32 * SW, BATCH = 8;                        // loads in flight per thread
    const unsigned long long n8 = (unsigned long long)rows * (QK_DIM / 8), end = n8 * (c + 1) / n_cta;
    unsigned int m = 0;
#pragma unroll 1
    for (unsigned long long i = n8 * c / n_cta + threadIdx.x; i < end; i += BATCH * ST) {
        uint4 v[BATCH];
#pragma unroll
        for (int k = 0; k < BATCH; ++k) v[k] = i + k * ST < end ? __ldcg(q8 + i + k * ST) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < BATCH; ++k) m = max(m, bf16x8_amax_bits(v[k]));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) q_red[threadIdx.x >> 5] = m;
    named_bar_sync(3, ST);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < SW; ++k) m = max(m, q_red[k]);
        atomicMax(reinterpret_cast<unsigned int*>(status + SYNC_AMAX), m);
        fence_acq_rel();
        atomicOr(status + SYNC_AMAX_DONE + (c >> 5), 1 << (c & 31));
    }
}
// Not all CTAs run yet: those that do look at the shares of the others, each at one that is open, until none is.  The maximum is in
// q_red[0] then.  (When each looked at all of Q: 128 sequences of 128 heads, hybrid cache, limit 0, 1580 us a call; 362 so, 347 where all wait.)
// Not inlined: registers of calls that never come here.
template <int SW>
__device__ __noinline__ void look_at_open_shares(const uint4* q8, int rows, int* status, int n_cta, int cta, unsigned int* q_red, int* q_share) {
    for (;;) {
        named_bar_sync(3, 32 * SW);                               // q_red has been read
        if (threadIdx.x == 0) {
            const int share = open_share(status, n_cta, cta);
            *q_share = share;
            if (share < 0) q_red[0] = amax_bits(status);
        }
        named_bar_sync(3, 32 * SW);
        if (*q_share < 0) break;
        look_at_share<SW>(q8, rows, status, n_cta, *q_share, q_red);
    }
}

// Meeting of the CTAs (end of the kernel).  One thread: the CTAs that have come, every one that had when this began among them, and
// their partials are visible.  A CTA sets its bit NO_BIT_CYCLES after being counted; the wait is bounded like mbar_wait.
__device__ __forceinline__ void who_came(int* status, int n_cta, int (&mask)[UNIT_TOK], volatile int* abort_flag) {
    const long long t0 = clock64();
    for (;;) {
        int bits = 0;
#pragma unroll 1
        for (int i = 0; i < SYNC_MASK_WORDS; ++i) {
            const int word = load_acquire(status + SYNC_ARRIVED + i);
            mask[i] = word;
            bits += __popc(word);
        }
        const int count = load_acquire(status + SYNC_ARRIVE) & 0xffff;
        if (bits == count) return;
        if (count >= n_cta) break;
        if (*abort_flag || clock64() - t0 > WAIT_LIMIT_CYCLES) { *abort_flag = 1; break; }
    }
    for (int i = 0; i < SYNC_MASK_WORDS; ++i) mask[i] = -1;
}
// Whether the CTAs [lo, hi] are all in the mask (true if there are none).
__device__ __forceinline__ bool in_mask(const int (&mask)[UNIT_TOK], int lo, int hi) {
    for (int i = lo >> 5; i <= hi >> 5 && lo <= hi; ++i) {
        const unsigned int want = (i == lo >> 5 ? ~0u << (lo & 31) : ~0u) & (i == hi >> 5 ? ~0u >> (31 - (hi & 31)) : ~0u);
        if (want & ~(unsigned int)mask[i]) return false;
    }
    return true;
}
// The first sequence from b0 on that CTA w holds together with others, and its CTAs; p.batch if there is none.
__device__ __forceinline__ int next_shared(const MlaParams& p, int b0, int w, int lane, int2& ctas) {
    for (; b0 < p.batch; b0 += 32) {
        const int2 c = b0 + lane < p.batch ? __ldcg(p.seq_ctas + b0 + lane) : make_int2(0, -1);
        const unsigned int hit = __ballot_sync(0xffffffffu, c.x < c.y && c.x <= w && w <= c.y);
        if (hit) {
            const int l = __ffs(hit) - 1;
            ctas = make_int2(__shfl_sync(0xffffffffu, c.x, l), __shfl_sync(0xffffffffu, c.y, l));
            return b0 + l;
        }
        if (__ballot_sync(0xffffffffu, c.x > w)) break;
    }
    return p.batch;
}

// One item of the merge: row r of sequence b (sh = 0), a half (1) or a quarter of it (2), which `item` tells.
__device__ __forceinline__ void merge_item(const MlaParams& p, int b, int r, int w0, int w1, int item, int sh, int lane) {
    if (sh == 2) merge_row<1, 12>(p, b, r, w0, w1, (item & 3) * 128 + lane * 4);
    else if (sh == 1) merge_row<2, 6>(p, b, r, w0, w1, (item & 1) * 256 + lane * 4);
    else merge_row<4, 4>(p, b, r, w0, w1, lane * 4);
}
// Not all CTAs have come in NO_BIT_CYCLES, or some had left when this one came (`seen`: SYNC_ARRIVE before it was counted).  One thread; returns
// the outcome of the meeting.  This and merge_late are not inlined: inside the kernel they cost the calls that never reach them
// registers (4-byte spills; e4m3 32 x 4096 24.15 us, 23.9 so).
__device__ __noinline__ int meet_late(Misc& ms, int* status, int n_cta, int cta, int seen, bool all, int cycles) {
    int* arrive = status + SYNC_ARRIVE;
    const int bit = 1 << (cta & 31);
    int meet = 0;
    or_release(status + SYNC_ARRIVED + (cta >> 5), bit);
    if (seen >> 16) {
        meet = MEET_LATE;
        who_came(status, n_cta, ms.mask(MASK_LATE_ARRIVED), &ms.abort_flag);
        for (int i = 0; i < SYNC_MASK_WORDS; ++i) ms.mask(MASK_LATE_LEFT)[i] = load_acquire(status + SYNC_LEFT + i);
    }
    if (!all) all = count_reached(arrive, n_cta, cycles);
    if (!all) {
        atomicOr(status + SYNC_LEFT + (cta >> 5), bit);
        all = (add_acq_rel(arrive, 1 << 16) & 0xffff) == n_cta;
    }
    if (!all) {
        meet |= MEET_LEFT;
        who_came(status, n_cta, ms.mask(MASK_ARRIVED), &ms.abort_flag);
        atomicAdd(status + ST_LEAVES, 1);
    }
    if (meet && load_acquire(status + SYNC_TABLE) == 0) meet |= MEET_NO_TABLE;
    return meet;
}
// The merge by a CTA that has left before the last came, or come after others had left.  All its threads; N rows per CTA.
template <int TILE, int N>
__device__ __noinline__ void merge_late(const MlaParams& p, Misc& ms, int first_item, int sh) {
    const int meet = ms.meet, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int w = blockIdx.x, y0 = blockIdx.y, G = gridDim.x, n_cta = G * gridDim.y;
    if (meet & MEET_NO_TABLE) {                                   // the first CTA has not begun: the same table, by this one
        if (warp == 0) {
            int s0, s1, mine;
            const int incl = lane_tiles<TILE>(p, lane, s0, s1, mine);
            write_seq_ctas<TILE>(p, make_sched(__shfl_sync(0xffffffffu, incl, 31), p.batch, G, p.seq_units), s0, s1, incl - mine);
        }
        __syncthreads();
    }
    int item = first_item, end = p.batch * p.rows << sh, heir_of = -1;       // >= 0: rows that others have left of this sequence
    for (;;) {
        for (; item < end; item += heir_of < 0 ? n_cta * warps : warps) {
            const int b = (item >> sh) / p.rows, r = (item >> sh) - b * p.rows, y = r / N;
            const int2 ctas = __ldcg(p.seq_ctas + b);
            if (ctas.x != ctas.y && (heir_of >= 0 ? in_mask(ms.mask(MASK_LATE_LEFT), item % n_cta, item % n_cta)
                                                  : !(meet & MEET_LEFT) || in_mask(ms.mask(MASK_ARRIVED), y * G + ctas.x, y * G + ctas.y)))
                merge_item(p, b, r, ctas.x, ctas.y, item, sh, lane);
        }
        if (!(meet & MEET_LATE)) break;
        int2 ctas;                                                // the next sequence that this CTA shares with others
        if (heir_of < 0) heir_of = ms.span[0] - 1;
        do heir_of = next_shared(p, heir_of + 1, w, lane, ctas);
        while (heir_of < p.batch && !in_mask(ms.mask(MASK_LATE_ARRIVED), y0 * G + ctas.x, y0 * G + ctas.y));
        if (heir_of >= p.batch) break;
        end = (heir_of * p.rows + (y0 + 1) * N) << sh;
        item = ((heir_of * p.rows + y0 * N) << sh) + warp;
    }
}

// Position of one role inside the CTA's span: the sequence of the current tile and its geometry.
template <int TILE>
struct Walk {
    int b, t0, t1, base, len, pair;
    __device__ __forceinline__ void start(const int* span) { b = span[0] - 1; t0 = 0; t1 = span[1]; base = len = 0; pair = -1; }
    // Make it describe the sequence that owns global tile t (t only grows between calls); true when that is a new one.
    __device__ __forceinline__ bool seek(const MlaParams& p, int t) {
        if (t < t1) return false;
        do {
            ++b;
            base = load_global(p.kv_indptr + b);
            len = max(load_global(p.kv_indptr + b + 1) - base, 0);
            t0 = t1;
            t1 = t0 + tiles_of_len<TILE>(len);
        } while (t1 <= t);
        ++pair;
        return true;
    }
};

// Column reductions over the 32 lanes of a warp by recursive halving: every step exchanges half of the columns that are
// left, so NC columns cost NC - 1 shuffles (+ 1 for 16) instead of 5 NC.  Lane l ends with column l (NC = 32) or l / 2 (NC = 16).
template <int NC, bool IS_MAX>
__device__ __forceinline__ float fold_columns(const float (&x)[NC], int lane) {
    float v[NC / 2];
#pragma unroll
    for (int h = NC / 2, m = 16; h >= 1; h >>= 1, m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float a = h == NC / 2 ? x[i] : v[i], b = h == NC / 2 ? x[i + h] : v[i + h];
            const float got = __shfl_xor_sync(0xffffffffu, up ? a : b, m), keep = up ? b : a;
            v[i] = IS_MAX ? fmaxf(keep, got) : keep + got;
        }
    }
    if (NC == 16) {
        const float got = __shfl_xor_sync(0xffffffffu, v[0], 1);
        v[0] = IS_MAX ? fmaxf(v[0], got) : v[0] + got;
    }
    return v[0];
}

__device__ __forceinline__ f32x2 bf16x2_to_f32x2(uint32_t w) { return pk2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
// eight bf16 values -> the eight e4m3 codes of q_cast_e4m3x8 (mla_common.cuh) in half the instructions: s2 = -scale and
// r2 = RN(1 / scale), twice.  For values below general_from(r), which those of a tensor are of its own scale; a -0 may come out
// as +0 (no product or sum of the decode tells them apart).
__device__ __forceinline__ uint2 q_quant_e4m3x8(const uint4& v, f32x2 s2, f32x2 r2) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const f32x2 x = bf16x2_to_f32x2(w[k]), t = mul2(x, r2), y = fma2(fma2(t, s2, x), r2, t);
        float y0, y1;
        unpk2(y, y0, y1);
        uint32_t h;                                               // the reference divides bf16 tensors: the quotient is a bf16 value
        asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(h) : "f"(y0), "f"(y1));
        unpk2(bf16x2_to_f32x2(h), y0, y1);
        uint16_t c;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(c) : "f"(y0), "f"(y1));
        q[k] = c;
    }
    return make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
}
// eight bf16 values x -> hi = e4m3(x s), lo = e4m3((x s - hi) * 16)
__device__ __forceinline__ void q_split_e4m3x8(const uint4& v, float s, uint2& hi, uint2& lo) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const f32x2 s2 = pk2(s, s), neg = pk2(-1.0f, -1.0f), c16 = pk2(16.0f, 16.0f);
    uint32_t h[2], l[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const f32x2 a = mul2(bf16x2_to_f32x2(w[2 * k]), s2), b = mul2(bf16x2_to_f32x2(w[2 * k + 1]), s2);
        float f0, f1, f2, f3;
        unpk2(a, f0, f1); unpk2(b, f2, f3);
        h[k] = pack_e4m3x4(f0, f1, f2, f3);
        const float2 h01 = unpack_e4m3x2((uint16_t)(h[k] & 0xffffu)), h23 = unpack_e4m3x2((uint16_t)(h[k] >> 16));
        unpk2(mul2(fma2(pk2(h01.x, h01.y), neg, a), c16), f0, f1);
        unpk2(mul2(fma2(pk2(h23.x, h23.y), neg, b), c16), f2, f3);
        l[k] = pack_e4m3x4(f0, f1, f2, f3);
    }
    hi = make_uint2(h[0], h[1]);
    lo = make_uint2(l[0], l[1]);
}

// byte offset of 16-byte column c of row r inside an operand (four panels of 128-byte rows, PANEL bytes each, then 64-byte rows)
template <int PANEL>
__device__ __forceinline__ uint32_t operand_offset(int r, int c) {
    return c < 32 ? (uint32_t)((c >> 3) * PANEL + r * 128 + (((c & 7) ^ (r & 7)) << 4))
                  : (uint32_t)(4 * PANEL + r * 64 + (((c - 32) ^ ((r >> 1) & 3)) << 4));
}

template <int N, int KVFMT, int QFMT>
__global__ void __launch_bounds__(Cfg<N, KVFMT, QFMT>::THREADS, 1)
mla_decode_sm100_kernel(const __grid_constant__ MlaParams p, const __grid_constant__ Maps maps, const bool use_tma) {
    using C = Cfg<N, KVFMT, QFMT>;
    constexpr int NQ = C::NQ, NC = C::NC, SW = C::SW, FW = C::FW, TILE = C::TILE, NS = C::NS, UNITS = C::UNITS;
    constexpr int PANEL_BYTES = C::PANEL_BYTES, STAGE_BYTES = C::STAGE_BYTES, P_BUFS = C::P_BUFS;
    extern __shared__ __align__(1024) unsigned char smem[];
    Misc& ms = *reinterpret_cast<Misc*>(smem + C::OFF_MISC);
    const uint32_t smem_base = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int w = blockIdx.x, G = p.num_ctas;
    const int row0 = blockIdx.y * N;
    const bool paged = p.kv_indices != nullptr;

    // Q quantised by this launch: its CTAs find the largest magnitude together, each in its share of Q
    const bool own_amax = !C::QSPLIT && p.q_cast && p.q_amax_parts == nullptr;

    // Nothing of this touches memory that the kernel before may still write: it runs while that one drains.  TMEM is taken later:
    // a kernel before it that lets its dependents start early may not have its own columns yet, and would wait for this CTA, which waits for it.
    if (tid == 32 * SW) {
        // a stage is full after one arrival per unit (copy loop, and the rope rows of a hybrid cache: also one per lane)
        for (int i = 0; i < NS; ++i) {
            mbar_init(&ms.kv_full[i], C::XF ? UNITS * (C::ROPE_SEP ? 33 : 1) : (use_tma ? UNITS : 32 * UNITS));
            for (int q = 0; q < TILE / 32; ++q) mbar_init(&ms.kv_empty[i][q], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ms.s_full[i], 1); mbar_init(&ms.s_empty[i], SW);
        }
        for (int i = 0; i < P_BUFS; ++i) { mbar_init(&ms.p_full[i], SW); mbar_init(&ms.p_empty[i], 1); }
        for (int i = 0; i < C::NBUF; ++i) { mbar_init(&ms.raw_full[i], 33); mbar_init(&ms.raw_empty[i], 1); }
        mbar_init(&ms.q_full, SW);
        mbar_init(&ms.o_free, SW);
        ms.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (warp == SW + 1) {
        ms.nm[0][0][lane] = ms.nm[1][0][lane] = 0.0f;
        if (lane == 0 && use_tma) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.lat) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.rope) : "memory");
        }
    }
    __syncwarp();
    pdl_wait();
    if (warp == C::AUX_WARP) {
        int span[4];
        find_span<TILE>(p, w, G, lane, span, w == 0 && blockIdx.y == 0);
        if (lane < 4) ms.span[lane] = lane == 0 ? span[0] : (lane == 1 ? span[1] : (lane == 2 ? span[2] : span[3]));
        if (lane < N / 16) {
            const int r = row0 + 16 * lane, j = r / p.heads;
            ms.q_off[lane] = (long long)j * p.q_row_stride + (long long)(r - j * p.heads) * p.q_head_stride;
        }
    } else if (warp > SW + 1 && warp <= SW + 3 && paged && p.total_kv_hint > 0 && p.total_kv_hint < (1LL << 31)) {
        // The page ids this CTA will walk lie near w/G of the table: pull that neighbourhood into L2 while the span is
        // being searched, so that the first dependent page-table read is not a cold DRAM access.
        const unsigned int n_ids = (unsigned int)p.total_kv_hint / (unsigned int)p.page_size, per = n_ids / (unsigned int)G;
        const unsigned int lo = (w * per > 256u ? w * per - 256u : 0u) & ~31u, hi = min((w + 1) * per + 256u, n_ids);
        for (unsigned int i = lo + (tid - 32 * (SW + 2)) * 32; i < hi; i += 64 * 32) prefetch_l2(p.kv_indices + i);
    } else if (warp < SW && own_amax) {
        look_at_share<SW>(reinterpret_cast<const uint4*>(p.q), p.batch * p.rows, p.status, gridDim.x * gridDim.y, blockIdx.y * gridDim.x + blockIdx.x, ms.q_red);
        if (tid == 0) atomicAdd(p.status + SYNC_AMAX_COUNT, 1);   // behind the fence of look_at_share
    }
    if (warp == C::QK_WARP) {
        tmem_alloc(&ms.tmem_base, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ms.tmem_base;
    const int t_begin = ms.span[2], t_end = ms.span[3];
    const int n_total = t_end - t_begin;                          // tiles of this CTA; tile index g = 0..n_total-1
    volatile int* abort_flag = &ms.abort_flag;

    if (n_total > 0) {
        if (warp < SW) {
            // =========================== softmax / correction / epilogue, Q rows ===========================
            // warpgroup sg owns the query rows (S / O columns) [col0, col0 + NC); thread = token `tok` = TMEM lane.  A tile has
            // 96 tokens: the fourth warp of a group only takes part in the votes, the rescaling and the epilogue.
            constexpr int ST = 32 * SW;                           // softmax threads
            const int sg = C::SMG == 1 ? 0 : warp >> 2, wv = warp & 3, tok = tid & 127, col0 = sg * NC, bar_id = 1 + sg;
            const bool active = wv < TILE / 32;
            const uint32_t lane_base = (uint32_t)(wv * 32) << 16;
            const float kv_tensor_scale = KVFMT != KV_MXFP4 ? __ldcg(p.kv_scale) : 1.0f;
            float q_scale = 1.0f;
            bool q_scale_due = own_amax;
            if constexpr (!C::QSPLIT) {
                if (p.q_cast && !own_amax) {                      // every warp reduces the partial maxima itself
                    unsigned int m = 0;
#pragma unroll
                    for (int i = 0; i < Q_AMAX_PARTS / 32; ++i) m = max(m, __ldcg(p.q_amax_parts + lane + 32 * i));
                    q_scale = q_scale_from_amax_bits(__reduce_max_sync(0xffffffffu, m));
                } else if (!p.q_cast) {
                    q_scale = __ldcg(p.q_scale);
                }
            }

            // Q rows of sequence b -> swizzled K-major panels.  Called when every S of the previous sequence has been read
            // by this thread's warpgroup, i.e. its QK MMAs have completed: the buffer is free without a barrier.
            auto load_q = [&](int b) {
                unsigned char* q_smem = smem + C::OFF_Q;
                int t0 = tid;
                asm volatile("" : "+r"(t0));                      // keeps the index arithmetic here: hoisted out of the tile loop it spilled
                if (C::QSPLIT || p.q_cast) {
                    // eight threads per row, thread = every eighth of the row's 72 eight-element vectors: source and destination
                    // of the nine are constants away from each other (the swizzle depends on the row and the parity of u only)
                    constexpr int ROUND = ST / 8;                 // rows at once
                    static_assert(N % ROUND == 0 && (!C::QSPLIT || N == ROUND), "a split group is held in registers");
                    const __nv_bfloat16* q0 = reinterpret_cast<const __nv_bfloat16*>(p.q) + (long long)b * p.q_len * p.q_row_stride;
                    const int cl = t0 & 7;
#pragma unroll 1
                    for (int r = t0 >> 3; r < N; r += ROUND) {
                        const uint4* src = reinterpret_cast<const uint4*>(q0 + ms.q_off[r >> 4] + (long long)(r & 15) * p.q_head_stride) + cl;
                        uint4 raw[9];
#pragma unroll
                        for (int u = 0; u < 9; ++u) raw[u] = __ldcg(src + 8 * u);
                        unsigned char* even = q_smem + r * 128 + (((cl >> 1) ^ (r & 7)) << 4) + (cl & 1) * 8;
                        unsigned char* odd = q_smem + r * 128 + (((cl >> 1) ^ 4 ^ (r & 7)) << 4) + (cl & 1) * 8;
                        unsigned char* rope = q_smem + 4 * C::Q_PANEL_BYTES + r * 64 + (((cl >> 1) ^ ((r >> 1) & 3)) << 4) + (cl & 1) * 8;
                        auto dst = [&](int u) { return reinterpret_cast<uint2*>(u == 8 ? rope : ((u & 1) ? odd : even) + (u >> 1) * C::Q_PANEL_BYTES); };
                        if constexpr (C::QSPLIT) {
                            // s = the power of two that puts the group's largest magnitude in [128, 256); zero group: s = 1
                            unsigned int m = 0;
#pragma unroll
                            for (int u = 0; u < 9; ++u) m = max(m, bf16x8_amax_bits(raw[u]));
                            m = __reduce_max_sync(0xffffffffu, m);
                            if (lane == 0) ms.q_red[warp] = m;
                            named_bar_sync(3, ST);
#pragma unroll
                            for (int k = 0; k < SW; ++k) m = max(m, ms.q_red[k]);
                            named_bar_sync(3, ST);                // q_red may be rewritten by the next sequence
                            int e = (int)(m >> 7) - 127;
                            e = m > 0 ? max(-100, min(e, 100)) : 7;
                            const float s = __int_as_float((7 - e + 127) << 23);
                            q_scale = __int_as_float((e - 7 + 127) << 23);
#pragma unroll
                            for (int u = 0; u < 9; ++u) {
                                uint2 hi, lo;
                                q_split_e4m3x8(raw[u], s, hi, lo);
                                *dst(u) = hi;
                                dst(u)[u == 8 ? N * 8 : N * 16] = lo;     // the lo rows follow the hi rows in every panel
                            }
                        } else {
                            if (q_scale_due) {                    // first use of the scale all CTAs contribute to: by now it is there
                                const int n_cta = (int)(gridDim.x * gridDim.y);
                                if (tid == 0)
                                    ms.q_red[0] = count_reached(p.status + SYNC_AMAX_COUNT, n_cta, p.meet_cycles) ? amax_bits(p.status) : 0xffffffffu;
                                named_bar_sync(3, ST);
                                unsigned int m = ms.q_red[0];
                                if (__builtin_expect(m == 0xffffffffu, 0)) {
                                    look_at_open_shares<SW>(reinterpret_cast<const uint4*>(p.q), p.batch * p.rows, p.status, n_cta,
                                                            (int)(blockIdx.y * gridDim.x + blockIdx.x), ms.q_red, &ms.q_share);
                                    m = ms.q_red[0];
#pragma unroll
                                    for (int u = 0; u < 9; ++u) raw[u] = __ldcg(src + 8 * u);     // again: not kept over the loop
                                }
                                q_scale = q_scale_from_amax_bits(m);
                                q_scale_due = false;
                            }
                            // an infinite scale (infinite Q) gives zeros and NaNs as the division would
                            const float rs = __frcp_rn(q_scale), sn = q_scale <= 3.0e38f ? -q_scale : 0.0f;
                            const f32x2 r2 = pk2(rs, rs), s2 = pk2(sn, sn);
                            bool special = false;
                            if (!own_amax) {                      // the caller's maxima: there may be values far beyond them
                                unsigned int m = 0;
#pragma unroll
                                for (int u = 0; u < 9; ++u) m = max(m, bf16x8_amax_bits(raw[u]));
                                special = m >= general_from(rs);
                            }
                            if (special) {
#pragma unroll 1
                                for (int u = 0; u < 9; ++u) *dst(u) = q_cast_e4m3x8(__ldcg(src + 8 * u), q_scale);
                            } else {
#pragma unroll
                                for (int u = 0; u < 9; ++u) *dst(u) = q_quant_e4m3x8(raw[u], s2, r2);
                            }
                        }
                    }
                } else {
                    const uint8_t* q0 = reinterpret_cast<const uint8_t*>(p.q) + (long long)b * p.q_len * p.q_row_stride;
                    const int cl = t0 & 3;                        // the same with four threads per row and 16-byte vectors
#pragma unroll 1
                    for (int r = t0 >> 2; r < N; r += ST / 4) {
                        const uint4* src = reinterpret_cast<const uint4*>(q0 + ms.q_off[r >> 4] + (long long)(r & 15) * p.q_head_stride) + cl;
                        uint4 raw[9];
#pragma unroll
                        for (int u = 0; u < 9; ++u) raw[u] = __ldcg(src + 4 * u);
#pragma unroll
                        for (int u = 0; u < 9; ++u)
                            *reinterpret_cast<uint4*>(q_smem + (u < 8 ? (u >> 1) * C::Q_PANEL_BYTES + r * 128 + ((((u & 1) << 2 | cl) ^ (r & 7)) << 4)
                                                                      : 4 * C::Q_PANEL_BYTES + r * 64 + ((cl ^ ((r >> 1) & 3)) << 4))) = raw[u];
                    }
                }
                fence_proxy_async();                              // the MMA reads Q through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&ms.q_full);
            };

            Walk<TILE> wk;
            wk.start(ms.span);
            float qk_base = 0.0f;          // sm_scale * log2(e) * (scale of this sequence's Q bytes)
            int e_run = 0;                 // exponent frame of O (block-scaled caches)
            int nm_cur = 0;
            f32x2 l_acc[NC / 2];           // this thread's share of the denominators
            // token position pos is visible to the rows of 16-column chunk q iff pos < lim[q]
            // (heads is a multiple of 16, so the query index j is constant inside a chunk)
            int lim[NC / 16], lim_min = 0;
            bool first = true;             // the tile starts a new (CTA, sequence) pair
            int b_prev = 0;
            bool whole_prev = false;
            for (int g = 0; g <= n_total; ++g) {
                const int sb = g & 1, st = g % NS;
                if (first) {
                    float lw = 0.0f;
                    if (g > 0) {
                        float l[NC];
#pragma unroll
                        for (int c = 0; c < NC; c += 2) unpk2(l_acc[c / 2], l[c], l[c + 1]);
                        lw = fold_columns<NC, false>(l, lane);
                        b_prev = wk.b;
                        whole_prev = (t_begin <= wk.t0) && (wk.t1 <= t_end);
                    }
                    // the next sequence's Q goes out before O of the previous one is read: its first QK overlaps that epilogue
                    if (g < n_total) { wk.seek(p, t_begin + g); load_q(wk.b); }
                    if (g > 0) {
                        // ---- epilogue of the (CTA, sequence) pair that ended with tile g-1: wait for its last PV, normalise, write out
                        if (NC == 32 || !(lane & 1)) ms.red[sg][wv][NC == 32 ? lane : lane >> 1] = lw;
                        named_bar_sync(bar_id, 128);
                        const bool whole = whole_prev;
                        const float out_scale = C::XF ? pow2i(e_run - E_BIAS) : kv_tensor_scale;
                        const long long orow0 = (whole ? (long long)b_prev * p.rows : (long long)(w + b_prev) * p.rows) + row0 + col0;
                        if (tok < NC) {                               // one thread per query row
                            const float sum = (ms.red[sg][0][tok] + ms.red[sg][1][tok]) + (ms.red[sg][2][tok] + ms.red[sg][3][tok]);
                            ms.fac[sg][tok] = sum > 0.0f ? __fdividef(out_scale, sum) : 0.0f;
                            const float lse = sum > 0.0f ? (log2f(sum) - ms.nm[sg][nm_cur][tok]) * LN2 : -INFINITY;
                            ms.nm[sg][nm_cur][tok] = 0.0f;
                            if (!whole) p.part_lse[orow0 + tok] = lse;
                            else if (p.out_lse) p.out_lse[orow0 + tok] = lse;
                        }
                        named_bar_sync(bar_id, 128);
                        mbar_wait(&ms.p_empty[(g - 1) % P_BUFS], (g - 1) / P_BUFS, abort_flag);
                        tc_fence_after();
                        // one output element per (row, dim): this thread owns dims tok, 128 + tok, ... of its warpgroup's rows
                        float* dst_f32 = whole ? p.out_o_f32 : p.part_o;
                        __nv_bfloat16* dst_bf16 = whole ? p.out : nullptr;
                        if (dst_f32) dst_f32 += orow0 * V_DIM + tok;
                        if (dst_bf16) dst_bf16 += orow0 * V_DIM + tok;
#pragma unroll 1
                        for (int jb = 0; jb < 4 * (NC / 16); ++jb) {                 // once per sequence: code size before speed
                            const int c0 = (jb % (NC / 16)) * 16, blk = jb / (NC / 16);
                            float o[16], olo[16];
                            tmem_ld16(tmem + lane_base + C::TMEM_O + blk * C::OB + col0 + c0, o);
                            if (!C::MERGED) tmem_ld16(tmem + lane_base + C::TMEM_O + blk * C::OB + N + col0 + c0, olo);
                            tmem_wait_ld();
                            const long long off = (long long)c0 * V_DIM + blk * 128;
#pragma unroll
                            for (int c = 0; c < 16; ++c) o[c] = (C::MERGED ? o[c] : fmaf(olo[c], 0.0625f, o[c])) * ms.fac[sg][c0 + c];
                            if (dst_bf16) {
#pragma unroll
                                for (int c = 0; c < 16; ++c) dst_bf16[off + c * V_DIM] = __float2bfloat16_rn(o[c]);
                            }
                            if (dst_f32) {
#pragma unroll
                                for (int c = 0; c < 16; ++c) dst_f32[off + c * V_DIM] = o[c];
                            }
                        }
                        // O has been read: the next sequence's first PV may overwrite it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&ms.o_free);
                    }
                    if (g == n_total) break;
#pragma unroll
                    for (int c = 0; c < NC / 2; ++c) l_acc[c] = 0ull;
                    lim_min = 0x7fffffff;
                    const int pos_off = p.kv_pos_offset ? __ldcg(p.kv_pos_offset + wk.b) : 0;
                    const int tot_len = p.kv_total_len ? __ldcg(p.kv_total_len + wk.b) : wk.len;
#pragma unroll
                    for (int q = 0; q < NC / 16; ++q) {
                        const int j = (row0 + col0 + 16 * q) / p.heads;
                        lim[q] = min(wk.len, p.causal ? tot_len - p.q_len + j + 1 - pos_off : 0x7fffffff);
                        lim_min = min(lim_min, lim[q]);
                    }
                    qk_base = p.sm_scale * LOG2E * q_scale;
                }
                const int pos_first = (t_begin + g - wk.t0) * TILE;
                // P(g) may overwrite its buffer once the PV that read it last has completed.  With as many buffers as stages that is the PV that
                // gives back the stage of this tile, which S waits for as well: looked at here it costs nothing, 130 cycles of the chain
                // behind S otherwise.
                const int pb = g % P_BUFS;
                if (P_BUFS == NS) mbar_wait(&ms.p_empty[pb], g / P_BUFS - 1, abort_flag);
                mbar_wait(&ms.s_full[sb], g / 2, abort_flag);
                tc_fence_after();
                // exponent frames: e_unit of this thread's token, e_tile = the largest of the tile's units
                int e_unit = 0, e_tile = 0;
                if (C::XF) {
                    const int4 ea = *reinterpret_cast<const int4*>(&ms.tile_exp[st][0]), eb = *reinterpret_cast<const int4*>(&ms.tile_exp[st][4]);
                    static_assert(!C::XF || UNITS == 8, "two vectors of frames");
                    e_tile = max(max(max(ea.x, ea.y), max(ea.z, ea.w)), max(max(eb.x, eb.y), max(eb.z, eb.w)));
                    e_unit = active ? ms.tile_exp[st][tok / UNIT_TOK] : 0;
                }
                const float a_lat = C::XF ? qk_base * pow2i(e_unit - E_BIAS) : qk_base * kv_tensor_scale;
                const float a_rope = qk_base * kv_tensor_scale;
                const uint32_t s_addr = tmem + lane_base + sb * C::SC + col0;
                float x[NC];
                // x = score in log2 units + nm: the exponent of the stored probability
                auto load_scores = [&](const float* nm) {
                    const f32x2 al = pk2(a_lat, a_lat), ar = pk2(a_rope, a_rope), c16 = pk2(0.0625f, 0.0625f);
#pragma unroll
                    for (int c0 = 0; c0 < NC; c0 += 16) {
                        float v[16], vl[16], r[16], rl[16];
                        tmem_ld16(s_addr + c0, v);
                        if (C::QSPLIT) tmem_ld16(s_addr + N + c0, vl);
                        if (C::ROPE_SEP) {
                            tmem_ld16(s_addr + NQ + c0, r);
                            if (C::QSPLIT) tmem_ld16(s_addr + NQ + N + c0, rl);
                        }
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 16; c += 4) {
                            const float4 n4 = *reinterpret_cast<const float4*>(nm + c0 + c);
#pragma unroll
                            for (int h = 0; h < 4; h += 2) {
                                f32x2 lat = pk2(v[c + h], v[c + h + 1]);
                                if (C::QSPLIT) lat = fma2(pk2(vl[c + h], vl[c + h + 1]), c16, lat);
                                f32x2 y = h ? pk2(n4.z, n4.w) : pk2(n4.x, n4.y);
                                if (C::ROPE_SEP) {
                                    f32x2 rope = pk2(r[c + h], r[c + h + 1]);
                                    if (C::QSPLIT) rope = fma2(pk2(rl[c + h], rl[c + h + 1]), c16, rope);
                                    y = fma2(rope, ar, y);
                                }
                                unpk2(fma2(lat, al, y), x[c0 + c + h], x[c0 + c + h + 1]);
                            }
                        }
                    }
                };
                const int pos = pos_first + tok;
                const bool masked_tile = pos_first + TILE > lim_min;                 // uniform
                auto mask_scores = [&]() {
                    if (masked_tile) {
#pragma unroll
                        for (int c = 0; c < NC; ++c) if (pos >= lim[c / 16]) x[c] = -INFINITY;
                    }
                };
                // x = scores relative to the reference maxima (to zero at a sequence's first tile, see nm); from here on the
                // tile lives in registers.  Where a maximum moves, x is shifted, so it is rounded twice, the first time relative to the old
                // maximum: half an ulp of FAR at most.  Beyond FAR the scores are read once more, absolutely (without that the LSE was off by
                // 3e-5 for a maximum that moves by 2^15 and by 2e-3 for 2^21; 1e-6 so).
                constexpr float FAR = 256.0f;
                if (active) {
                    load_scores(ms.nm[sg][nm_cur]);
                    mask_scores();
                }
                bool recenter = first;
                if (!first) {
                    float xm = -INFINITY;
                    if (active) {
                        xm = x[0];
#pragma unroll
                        for (int c = 1; c < NC - 1; c += 2) xm = max3(xm, x[c], x[c + 1]);
                        xm = fmaxf(xm, x[NC - 1]);
                    }
                    recenter = named_bar_or(bar_id, 128, xm > C::P_SCALE_LOG2 + C::RECENTER);
                }
                // a larger exponent frame than the one O is held in: O moves to the new frame
                float o_frame = 1.0f;
                if (C::XF) {
                    if (first) e_run = e_tile;
                    if (e_tile > e_run) { o_frame = pow2i(e_run - e_tile); e_run = e_tile; }
                }
                unsigned int moved = 0;                           // rows of O to rescale
                if (recenter) {
                    // the tile's maximum of query row tok, in its thread
                    auto row_max = [&]() {
                        const float top = active ? fold_columns<NC, true>(x, lane) : -INFINITY;
                        if (NC == 32 || !(lane & 1)) ms.red[sg][wv][NC == 32 ? lane : lane >> 1] = top;
                        named_bar_sync(bar_id, 128);
                        return tok < NC ? fmaxf(fmaxf(ms.red[sg][0][tok], ms.red[sg][1][tok]), fmaxf(ms.red[sg][2][tok], ms.red[sg][3][tok])) : -INFINITY;
                    };
                    // x is relative to P_SCALE_LOG2 - base; the row's reference maximum goes from P_SCALE_LOG2 - old to P_SCALE_LOG2 - next
                    auto move_row = [&](float base, float old, float next) {
                        ms.nm[sg][nm_cur ^ 1][tok] = next;
                        ms.shift[sg][tok] = next - base;
                        ms.fac[sg][tok] = ex2(next - old);
                    };
                    float mx = row_max();
                    if (tok < NC) {                               // one thread per query row
                        const float old = ms.nm[sg][nm_cur][tok];
                        move_row(old, old, mx > (first ? -INFINITY : C::P_SCALE_LOG2) ? old + (C::P_SCALE_LOG2 - mx) : old);
                    }
                    if (__builtin_expect(named_bar_or(bar_id, 128, !first && tok < NC && mx > FAR), 0)) {
                        if (tok < NC) ms.shift[sg][tok] = 0.0f;
                        named_bar_sync(bar_id, 128);
                        if (active) {
                            load_scores(ms.shift[sg]);
                            mask_scores();
                        }
                        mx = row_max();
                        if (tok < NC) {
                            const float old = ms.nm[sg][nm_cur][tok];
                            move_row(0.0f, old, fminf(old, C::P_SCALE_LOG2 - mx));
                        }
                        named_bar_sync(bar_id, 128);
                    }
                    nm_cur ^= 1;
#pragma unroll
                    for (int c = 0; c < NC; c += 4) {
                        const float4 d4 = *reinterpret_cast<const float4*>(&ms.shift[sg][c]);
                        x[c] += d4.x; x[c + 1] += d4.y; x[c + 2] += d4.z; x[c + 3] += d4.w;
                    }
                    if (!first) {
                        moved = __ballot_sync(0xffffffffu, lane < NC && ms.fac[sg][lane & (NC - 1)] != 1.0f);
#pragma unroll
                        for (int c = 0; c < NC / 2; c += 2) {
                            const float4 f4 = *reinterpret_cast<const float4*>(&ms.fac[sg][2 * c]);
                            l_acc[c] = mul2(l_acc[c], pk2(f4.x, f4.y)); l_acc[c + 1] = mul2(l_acc[c + 1], pk2(f4.z, f4.w));
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ms.s_empty[sb]);
                uint32_t hi[NC / 4], lo[NC / 4];
                if (active) {
                    // stored probability = p * 2^P_SCALE_LOG2 * 2^(e_unit - e_run): this token's V bytes are in the frame e_unit, O in e_run
                    const float p_frame = C::XF ? pow2i(e_unit - e_run) : 1.0f;
                    const f32x2 pf = pk2(p_frame, p_frame), neg = pk2(-1.0f, -1.0f);
                    // MERGED: the lo term shares O's columns with the hi term, so it carries no factor of its own
                    const f32x2 gain = pk2(16.0f, 16.0f);
#pragma unroll
                    for (int q4 = 0; q4 < NC / 4; ++q4) {
                        const int c = q4 * 4;
                        f32x2 p01 = pk2(ex2(x[c]), ex2(x[c + 1])), p23 = pk2(ex2(x[c + 2]), ex2(x[c + 3]));   // ex2(-inf) = 0 for masked keys
                        l_acc[c / 2] = add2(l_acc[c / 2], p01);
                        l_acc[c / 2 + 1] = add2(l_acc[c / 2 + 1], p23);
                        if (C::XF) { p01 = mul2(p01, pf); p23 = mul2(p23, pf); }
                        float p0, p1, p2, p3;
                        unpk2(p01, p0, p1); unpk2(p23, p2, p3);
                        hi[q4] = pack_e4m3x4(p0, p1, p2, p3);
                        const float2 h01 = unpack_e4m3x2((uint16_t)(hi[q4] & 0xffffu)), h23 = unpack_e4m3x2((uint16_t)(hi[q4] >> 16));
                        p01 = fma2(pk2(h01.x, h01.y), neg, p01); p23 = fma2(pk2(h23.x, h23.y), neg, p23);       // exact residuals
                        if (!C::MERGED) { p01 = mul2(p01, gain); p23 = mul2(p23, gain); }
                        unpk2(p01, p0, p1); unpk2(p23, p2, p3);
                        lo[q4] = pack_e4m3x4(p0, p1, p2, p3);
                    }
                }
                if (P_BUFS < NS) mbar_wait(&ms.p_empty[pb], g / P_BUFS - 1, abort_flag);
                if (active) {
                    uint8_t* pbuf = smem + C::OFF_P + pb * C::P_BUF_BYTES + (col0 / 16) * C::P_CHUNK_BYTES + tok * 16;
#pragma unroll
                    for (int q = 0; q < NC / 16; ++q) {
                        *reinterpret_cast<uint4*>(pbuf + q * C::P_CHUNK_BYTES) = make_uint4(hi[4 * q], hi[4 * q + 1], hi[4 * q + 2], hi[4 * q + 3]);
                        *reinterpret_cast<uint4*>(pbuf + (N / 16 + q) * C::P_CHUNK_BYTES) = make_uint4(lo[4 * q], lo[4 * q + 1], lo[4 * q + 2], lo[4 * q + 3]);
                    }
                    fence_proxy_async();
                }
                if (moved || (o_frame != 1.0f && !first)) {
                    // O holds the sequence's earlier tiles once PV(g-1) has completed; nothing else touches it until P(g) is published.
                    // This is the last thing before that, with P already stored: the tensor pipe waits only for the rescaling itself.
                    // Eight rows of the four blocks at a time, where one of them moved.
                    mbar_wait(&ms.p_empty[(g - 1) % P_BUFS], (g - 1) / P_BUFS, abort_flag);
                    tc_fence_after();
#pragma unroll 1
                    for (int i = 0; i < (C::MERGED ? 1 : 2) * (NC / 8); ++i) {                 // eight rows and, side by side, hi / lo half
                        const int r = i % (NC / 8) * 8;
                        if (o_frame == 1.0f && !(moved >> r & 0xffu)) continue;
                        const uint32_t addr = tmem + lane_base + C::TMEM_O + i / (NC / 8) * N + col0 + r;
                        float o[4][8];
#pragma unroll
                        for (int blk = 0; blk < 4; ++blk) tmem_ld8(addr + blk * C::OB, o[blk]);
                        float f[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) f[c] = recenter ? ms.fac[sg][r + c] * o_frame : o_frame;
                        tmem_wait_ld();
#pragma unroll
                        for (int blk = 0; blk < 4; ++blk) {
#pragma unroll
                            for (int c = 0; c < 8; ++c) o[blk][c] *= f[c];
                            tmem_st8(addr + blk * C::OB, o[blk]);
                        }
                    }
                    tmem_wait_st();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ms.p_full[pb]);

                first = t_begin + g + 1 == min(t_end, wk.t1);
            }
        } else if (warp < SW + FW) {
            // =========================== feed ===========================
            // The CTA's tiles are a stream of 16-token units; feed warp xw owns units xw, xw + FW, ...  Page ids are looked up ahead
            // of their use and not touched until they become an address (a compare at the load would wait for it).  Rows past
            // the end of the sequence name its last row instead (real cache bytes, finite; their probabilities are zero).
            const int ft = tid - 32 * SW, xw = ft >> 5;
            const int J = (n_total * UNITS - xw + FW - 1) / FW;       // units of this warp
            auto advance = [&](int& g, int& k) {                      // unit index += FW
                k += FW % UNITS; g += FW / UNITS;
                if (k >= UNITS) { k -= UNITS; ++g; }
            };
            int g = xw / UNITS, k = xw % UNITS;                       // unit at hand
            if constexpr (!C::XF) {
                // e4m3 cache: the rows' five panels (four 128-byte-wide, one 64-byte) go straight into the operand stage with the
                // swizzle of its layout, four rows per gather or sixteen per box, completion in bytes on the stage's mbarrier.
                // Copy-engine instructions are issued by one elected lane with warp-uniform operands: from a divergent lane each
                // costs a loop of some 150 cycles around it, which set the pace of this role.
                // evict_first: the streaming megabytes must not push the code, Q and the page table out of L2.
                Walk<TILE> wk;
                wk.start(ms.span);
                int page_base = 0;
                bool bad = false;
                int id = 0, off = 0, inside = 0;                      // page id and offset in it of row (lane & 15) of the unit fetched last;
                                                                      // inside: all of its 16 rows lie in the sequence
                const int id_mul = paged ? p.page_size : 1;
                const unsigned int id_max = paged ? p.last_page : p.last_slot;
                // sixteen neighbouring positions are sixteen neighbouring rows of the planes: one box instead of four gathers
                const bool boxes = use_tma && (!paged || p.page_size % UNIT_TOK == 0);
                int g2 = g, k2 = k;                                   // unit whose page ids are fetched next
                auto fetch_id = [&]() {
                    if (wk.seek(p, t_begin + g2)) page_base = p.kv_page_indptr ? load_global(p.kv_page_indptr + wk.b) : wk.base;
                    const int pos0 = (t_begin + g2 - wk.t0) * TILE + k2 * UNIT_TOK, pos = min(pos0 + (lane & 15), wk.len - 1);
                    inside = pos0 + UNIT_TOK <= wk.len;
                    id = paged ? load_global(p.kv_indices + page_base + page_of(p, pos)) : wk.base + pos;
                    off = paged ? off_in_page(p, pos) : 0;
                    advance(g2, k2);
                };
                const uint64_t pol = l2_evict_first_policy();
                if (J > 0) fetch_id();
#pragma unroll 1
                for (int j = 0; j < J; ++j) {
                    const int st = g % NS;
                    bad |= (unsigned int)id > id_max;
                    const unsigned int slot = clamp_slot(p, id * id_mul + off);
                    const bool box = boxes && inside;
                    if (j + 1 < J) fetch_id();
                    mbar_wait(&ms.kv_empty[st][k * UNIT_TOK / 32], g / NS - 1, abort_flag);
                    const uint32_t lat = smem_base + st * STAGE_BYTES + k * (UNIT_TOK * 128), rope = smem_base + st * STAGE_BYTES + 4 * PANEL_BYTES + k * (UNIT_TOK * 64);
                    if (use_tma) {
                        mbar_arrive_expect_tx_elect(&ms.kv_full[st], UNIT_TOK * QK_DIM);
                        if (box) {
                            tma_rows_box_elect<PANEL_BYTES>(lat, rope, &maps.lat_box, &maps.rope_box, (int)__shfl_sync(0xffffffffu, slot, 0), &ms.kv_full[st], pol);
                        } else {
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                int r[4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) r[i] = (int)__shfl_sync(0xffffffffu, slot, 4 * q + i);
                                tma_rows_gather4_elect<PANEL_BYTES>(lat + q * 512, rope + q * 256, &maps.lat, &maps.rope, r[0], r[1], r[2], r[3], &ms.kv_full[st], pol);
                            }
                        }
                    } else {                                          // no tensor maps (driver entry point missing): 16-byte copies
                        for (int i = lane; i < UNIT_TOK * 36; i += 32) {
                            const int t = i / 36, c = i - t * 36;
                            cp_async16(smem_base + st * STAGE_BYTES + operand_offset<PANEL_BYTES>(k * UNIT_TOK + t, c),
                                       p.kv_codes + (long long)__shfl_sync(0xffffffffu, slot, t) * p.kv_codes_stride + c * 16, 16u);
                        }
                        cp_async_mbar_arrive_noinc(&ms.kv_full[st]);
                    }
                    advance(g, k);
                }
                cp_async_wait_all();
                if (bad) report_status(p.status, ST_BAD_PAGE);
            } else {
                // Block-scaled cache: convert.  The auxiliary warps bring the units into the landing buffers, in rounds; a landed unit
                // moves into registers, its buffer goes back at once, and the e4m3 operand bytes go to the stage.
                // Lane = (32-code block hb of the row, row parity rp): every eight-lane phase of the 16-byte stores into the
                // swizzled tile hits all banks; the two rope blocks of an MXFP4 row are one more, (row, block).
                constexpr int NB = KVFMT == KV_MXFP4 ? 9 : 8;         // blocks per lane
                const int hb = (lane & 3) | ((lane >> 3) << 2), rp = (lane >> 2) & 1;
                const unsigned int scale_stride = (unsigned int)p.kv_bs_stride, bs_lo = (unsigned int)reinterpret_cast<uintptr_t>(p.kv_bs);
                // store offsets: block hb of row r = rp + 2i sits at row * 128 + ((2 (hb & 3)) ^ (r & 7)) * 16 of panel hb / 4
                const uint32_t st_row = smem_base + (uint32_t)((hb >> 2) * PANEL_BYTES + rp * 128), st_x = (uint32_t)(((2 * (hb & 3)) ^ rp) << 4);
                const uint32_t st_rope = smem_base + 4u * PANEL_BYTES + (uint32_t)((lane >> 1) * 64 + (((2 * (lane & 1)) ^ ((lane >> 2) & 3)) << 4));
                int u = xw;
#pragma unroll 1
                for (int j = 0; j < J; ++j, u += FW) {
                    const int st = g % NS, n = u % C::NBUF;
                    const unsigned char* raw = smem + C::OFF_RAW + n * C::RAW_BYTES;
                    mbar_wait(&ms.raw_full[n], u / C::NBUF, abort_flag);
                    const unsigned int row_slot = clamp_slot(p, ms.raw_slot[n][lane >> 1]);
                    const int so = (int)((bs_lo + row_slot * scale_stride) & 15u);    // the E8M0 row starts so bytes into its 32
                    uint4 v[NB];
                    uint32_t sc[NB], e = 0, e_min = 255;
#pragma unroll
                    for (int i = 0; i < NB; ++i) {
                        const int r = i < 8 ? rp + 2 * i : lane >> 1, blk = i < 8 ? hb : 16 + (lane & 1);
                        sc[i] = raw[UNIT_TOK * C::CODE_BYTES + r * 32 + __shfl_sync(0xffffffffu, so, 2 * r) + blk];
                        v[i] = *reinterpret_cast<const uint4*>(raw + raw_chunk<C::CODE_BYTES>(r, blk));
                        e = max(e, sc[i]);
                        e_min = min(e_min, sc[i]);
                    }
                    const int e_unit = (int)__reduce_max_sync(0xffffffffu, e);
                    const bool narrow = __all_sync(0xffffffffu, (int)e_min >= e_unit - 11);     // every block's k is -5 or more
#pragma unroll
                    for (int i = 0; i < NB; ++i) asm volatile("" : "+r"(v[i].x), "+r"(v[i].y), "+r"(v[i].z), "+r"(v[i].w));
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ms.raw_empty[n]);     // every lane has read the buffer
                    mbar_wait(&ms.kv_empty[st][k * UNIT_TOK / 32], g / NS - 1, abort_flag);
                    if (lane == 0) ms.tile_exp[st][k] = e_unit;
                    if (C::ROPE_SEP) {                                // rope bytes are e4m3 already: straight into the rope panel
                        const uint8_t* src = p.kv_rope + (unsigned long long)row_slot * (unsigned int)p.kv_rope_stride + (lane & 1) * 32;
                        const uint32_t panel = smem_base + st * STAGE_BYTES;
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            cp_async16(panel + operand_offset<PANEL_BYTES>(k * UNIT_TOK + (lane >> 1), 32 + (lane & 1) * 2 + c), src + c * 16, 16u);
                        cp_async_mbar_arrive_noinc(&ms.kv_full[st]);
                    }
                    const uint32_t dst = st_row + st * STAGE_BYTES + k * (UNIT_TOK * 128), dst_rope = st_rope + st * STAGE_BYTES + k * (UNIT_TOK * 64);
                    auto store_block = [&](int i, const uint4& lo, const uint4& hi) {
                        const uint32_t xo = st_x ^ ((i & 3) << 5);
                        st_shared_v4(i < 8 ? dst + 256 * i + xo : dst_rope, lo);
                        st_shared_v4(i < 8 ? dst + 256 * i + (xo ^ 16) : dst_rope ^ 16, hi);
                    };
                    uint4 lo, hi;
                    if (narrow) {
#pragma unroll
                        for (int i = 0; i < NB; ++i) { dequant_block<false>(v[i], (int)sc[i] - e_unit + 6, lo, hi); store_block(i, lo, hi); }
                    } else {
#pragma unroll
                        for (int i = 0; i < NB; ++i) { dequant_block<true>(v[i], (int)sc[i] - e_unit + 6, lo, hi); store_block(i, lo, hi); }
                    }
                    fence_proxy_async();                              // the MMA reads the tile through the async proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ms.kv_full[st]);      // one arrival per unit
                    advance(g, k);
                }
                cp_async_wait_all();
            }
        } else if (warp == C::QK_WARP) {
            // =========================== issue of S^T = K . Q^T (whole warp, one elected lane per instruction) ===========================
            // Scores and output have a warp each, so that either MMA goes out when its own operands are there.  One warp for both
            // polled all barriers with a vote per round: 660 cycles from P to its MMAs, and QK of a tile that had landed meanwhile
            // waited for both (2100 cycles; MXFP4, 32 rows).
            constexpr uint32_t IDESC_QK = make_idesc(128, NQ, false, false);
            // descriptor bases; per-MMA descriptors differ only in the start address
            const uint64_t d_qk_a = make_desc(smem_base, 16, 1024, SWIZZLE_128B);                              // + stage
            const uint64_t d_qk_a_rope = make_desc(smem_base + 4 * PANEL_BYTES, 16, 512, SWIZZLE_64B);         // + stage
            const uint64_t d_qk_b = make_desc(smem_base + C::OFF_Q, 16, 1024, SWIZZLE_128B);
            const uint64_t d_qk_b_rope = make_desc(smem_base + C::OFF_Q + 4 * C::Q_PANEL_BYTES, 16, 512, SWIZZLE_64B);
            Walk<TILE> wk;
            wk.start(ms.span);
            // A hybrid cache keeps the scores of its rope dims in columns of their own.  The panel loop is not unrolled: the issue
            // code stays a few hundred bytes, which is what the first pass through it pays for.
#pragma unroll 1
            for (int g = 0; g < n_total; ++g) {
                const int st = g % NS, sb = g & 1;
                const bool q_first = wk.seek(p, t_begin + g);
                mbar_wait(&ms.s_empty[sb], g / 2 - 1, abort_flag);
                if (q_first) mbar_wait(&ms.q_full, wk.pair, abort_flag);
                mbar_wait(&ms.kv_full[st], g / NS, abort_flag);
                __syncwarp();
                fence_proxy_async();       // cp.async (copy loop) wrote through the generic proxy; the MMA reads through the async proxy
                tc_fence_after();
                const uint32_t d_lat = tmem + sb * C::SC, d_rope = d_lat + (C::ROPE_SEP ? NQ : 0);
#pragma unroll 1
                for (int j = 0; j < 4; ++j)
                    umma_f8_x4_elect<0, 32, 32>(d_lat, desc_advance(d_qk_a, st * STAGE_BYTES + j * PANEL_BYTES), desc_advance(d_qk_b, j * C::Q_PANEL_BYTES),
                                                IDESC_QK, j, 1u);
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    umma_f8_elect(d_rope, desc_advance(d_qk_a_rope, st * STAGE_BYTES + k * 32), desc_advance(d_qk_b_rope, k * 32),
                                  IDESC_QK, (!C::ROPE_SEP || k > 0) ? 1u : 0u);
                umma_commit_elect(&ms.s_full[sb]);
            }
        } else if (warp == C::PV_WARP) {
            // =========================== issue of O^T += V^T P^T, four blocks of 128 dims (whole warp as above) ===========================
            constexpr uint32_t IDESC_PV = make_idesc(128, C::OB, true, true);
            const uint64_t d_pv_a = make_desc(smem_base, PANEL_BYTES, 1024, SWIZZLE_128B);                     // + stage
            const uint64_t d_pv_b = make_desc(smem_base + C::OFF_P, 128, C::P_CHUNK_BYTES, SWIZZLE_NONE);      // + buffer
            Walk<TILE> wk;
            wk.start(ms.span);
#pragma unroll 1
            for (int g = 0; g < n_total; ++g) {
                const int st = g % NS, pb = g % P_BUFS;
                const bool first = wk.seek(p, t_begin + g);
                // the first PV of a sequence overwrites O: the previous sequence's epilogue must have read it
                if (first && wk.pair > 0) mbar_wait(&ms.o_free, wk.pair - 1, abort_flag);
                mbar_wait(&ms.p_full[pb], g / P_BUFS, abort_flag);
                __syncwarp();
                tc_fence_after();
                const uint64_t a0 = desc_advance(d_pv_a, st * STAGE_BYTES);
                const uint64_t b0 = desc_advance(d_pv_b, pb * C::P_BUF_BYTES);
#pragma unroll 1
                for (int kk = 0; kk < TILE / 32; ++kk) {
#pragma unroll
                    for (int half = 0; half < (C::MERGED ? 2 : 1); ++half) {
                        const uint32_t acc = !first || kk > 0 || half > 0;
                        umma_f8_x4_elect<C::OB, PANEL_BYTES, 0>(tmem + C::TMEM_O, desc_advance(a0, kk * 32 * 128),
                                                                desc_advance(b0, kk * 32 * 16 + half * (N / 16) * C::P_CHUNK_BYTES), IDESC_PV, acc, acc);
                    }
                    umma_commit_elect(&ms.kv_empty[st][kk]);          // these 32 tokens' part of the stage may be refilled
                }
                umma_commit_elect(&ms.p_empty[pb]);
            }
        } else if constexpr (C::XF) {
            // =========================== auxiliary warps of a block-scaled cache: fetch ===========================
            // Two warps bring the units, every other one each, into the landing buffers by 16-byte cp.async, eight lanes on 128
            // consecutive bytes of a row, plus one copy of the aligned 16-byte words around each E8M0 row.  (Row gathers by the copy
            // engine were slower, 75.8 us against 69.4 for 64 x 8192 MXFP4; loads straight into registers much slower: with nearly
            // all of the L1 configured as shared memory there are not enough lines left for loads in flight.)
            constexpr int HALF = UNITS / 2, NB2 = 2 * (KVFMT == KV_MXFP4 ? 9 : 8);
            const int aw = warp - C::AUX_WARP, t = lane >> 1;
            Walk<TILE> wk;
            wk.start(ms.span);
            int page_base = 0;
            bool bad = false;
            static_assert(HALF == 4, "a tile's units of one warp are two rows a lane");
            const int id_mul = paged ? p.page_size : 1;
            const unsigned int id_max = paged ? p.last_page : p.last_slot;
            const unsigned int code_stride = (unsigned int)p.kv_codes_stride, scale_stride = (unsigned int)p.kv_bs_stride;
            // Page ids of a tile's four units of this warp, lane = (unit parity, token): fetched a tile ahead and not touched before
            // the tile's turn (a move of a register that a load is still to fill waits for it: with a ring of ids shifted per unit
            // this loop spent 600 of its 1300 cycles there).
            int id[2], off[2];
            auto look_up = [&](int g) {
                if (wk.seek(p, t_begin + g)) page_base = p.kv_page_indptr ? load_global(p.kv_page_indptr + wk.b) : wk.base;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int pos = min((t_begin + g - wk.t0) * TILE + ((4 * i + ((lane >> 4) << 1)) + aw) * UNIT_TOK + (lane & 15), wk.len - 1);
                    id[i] = paged ? load_global(p.kv_indices + page_base + page_of(p, pos)) : wk.base + pos;
                    off[i] = paged ? off_in_page(p, pos) : 0;
                }
            };
            look_up(0);
            const uint32_t dst8 = smem_base + C::OFF_RAW + raw_chunk<C::CODE_BYTES>(lane >> 3, lane & 7);
            const uint32_t dst2 = smem_base + C::OFF_RAW + raw_chunk<C::CODE_BYTES>(t, 0) + 256 + (lane & 1) * 16;
            const uint32_t dst_bs = smem_base + C::OFF_RAW + UNIT_TOK * C::CODE_BYTES + lane * 16;
            const uint8_t* codes8 = p.kv_codes + (lane & 7) * 16;
            int n = aw, round = 0;                                    // landing buffer and its round
#pragma unroll 1
            for (int g = 0; g < n_total; ++g) {
                unsigned int rows[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    bad |= (unsigned int)id[i] > id_max;
                    rows[i] = clamp_slot(p, id[i] * id_mul + off[i]);
                }
                if (g + 1 < n_total) look_up(g + 1);
#pragma unroll 1
                for (int k = 0; k < HALF; ++k) {
                    const unsigned int row = __shfl_sync(0xffffffffu, k & 2 ? rows[1] : rows[0], ((k & 1) << 4) | t);
                    const uint8_t* src[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) src[q] = codes8 + (unsigned long long)__shfl_sync(0xffffffffu, row, 8 * q + 2 * (lane >> 3)) * code_stride;
                    const uintptr_t sb = reinterpret_cast<uintptr_t>(p.kv_bs) + (unsigned long long)row * scale_stride;
                    const bool need = (lane & 1) == 0 || (int)(sb & 15) + NB2 > 16;                 // the second word only where the row reaches into it
                    const uint32_t buf = n * C::RAW_BYTES;
                    mbar_wait(&ms.raw_empty[n], round - 1, abort_flag);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        cp_async16(dst8 + buf + q * 4 * C::CODE_BYTES, src[q], 16u);
                        cp_async16(dst8 + buf + q * 4 * C::CODE_BYTES + 128, src[q] + 128, 16u);
                    }
                    if (C::CODE_BYTES == 288)
                        cp_async16(dst2 + buf, p.kv_codes + (unsigned long long)row * code_stride + 256 + (lane & 1) * 16, 16u);
                    cp_async16(dst_bs + buf, reinterpret_cast<const void*>((sb & ~(uintptr_t)15) + (need ? (lane & 1) * 16 : 0)), 16u);
                    cp_async_mbar_arrive_noinc(&ms.raw_full[n]);
                    if ((lane & 1) == 0) ms.raw_slot[n][t] = (int)row;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ms.raw_full[n]);
                    n += 2;
                    if (n >= C::NBUF) { n -= C::NBUF; ++round; }
                }
            }
            cp_async_wait_all();
            if (bad) report_status(p.status, ST_BAD_PAGE);
        }
    }

    // Merge of the partials by the same launch: the CTAs meet, then the query rows are dealt out to all warps - whole rows,
    // halves or quarters, so that every warp has one item at most where there are few.  (A second kernel cost 5 us and more per
    // call: launch, drain, cold code.)  The first items go to the warps that are done before the epilogue: they look up
    // what theirs consists of while the softmax warps still write (a load, about 1 k cycles behind the meeting otherwise), so a
    // row is cut up only as far as there are such warps (MXFP4 32 x 1024: 15.15 us with quarters that softmax warps share, 14.7 with
    // halves), and the loads of all its partials are in flight together where registers allow: one more round over them costs
    // 0.5 to 1.3 us (halves, four at a time -> six: MXFP4 32 x 1024 14.7 -> 14.1, e4m3 32 x 4096 24.05 -> 23.65; twenty
    // quarters: spills, 32.9 us for a rank of eight instead of 31.2).
    // The launch is not cooperative (see MlaParams::meet_cycles): a CTA that has waited meet_cycles for the others goes.  It says so (its
    // bit in SYNC_LEFT, then one in the upper half of SYNC_ARRIVE), looks who has come, and merges those rows of its share whose
    // partials are all there.  A row that it has to leave behind lacks a CTA that comes later; that one learns from SYNC_ARRIVE that
    // others had left, and the last CTA of a sequence to come merges what those have left of it.  So what falls on a late CTA is rows of the
    // one or two sequences that it shares with others, in its row group: 64 rows of 74 partials at most, 10 MB and 270 us for one CTA (one
    // sequence of 131072 tokens, 128 heads, one SM held by another stream: 450 us, 64 without that).
    // When all of it fell on the last CTA of the call, 50 us of waiting in vain became several hundred of merging by one CTA (us a call: 500
    // sequences of 3 tokens, 500 of 700 and 20 of 100000 mixed, 128 heads over an e4m3 cache, 1447, 865 so and 937 if every CTA waits for
    // all; 3000 of 5 and 30 of 300000, MXFP4, 2315, 1127 and 1162; 48 sequences of 128 heads with a limit of 0, 753 and 90, where 78 is
    // without anyone leaving).
    // Two that write a row (a CTA that learns only as it goes that all have come merges its share after all) write the same values.
    // Who has come is read from SYNC_ARRIVED, whose bits are set after the count: a look that shows as many bits as the count
    // read after it shows every CTA that had come by then.
    constexpr int WARPS = C::THREADS / 32;
    const int n_cta = (int)(gridDim.x * gridDim.y), cta = (int)(blockIdx.y * gridDim.x + blockIdx.x);
    const int rows_all = p.batch * p.rows, n_warps = n_cta * WARPS;
    const int n_early = n_cta * (WARPS - SW), sh = rows_all * 4 <= n_early ? 2 : (rows_all * 2 <= n_early ? 1 : 0);
    const int first_item = (warp >= SW ? warp - SW : warp + WARPS - SW) * n_cta;      // of CTA 0
    int b = 0, w0 = 0, w1 = -1, item = first_item + cta;
    bool work = false, looked_up = false;
    auto look_up = [&]() {
        if ((item >> sh) >= rows_all) return;
        b = (item >> sh) / p.rows;
        const int2 ctas = __ldcg(p.seq_ctas + b);
        w0 = ctas.x; w1 = ctas.y;
        work = w0 != w1;                                          // one CTA has finished the sequence; none: zeros
    };
    if (p.fused && warp >= SW) {
        looked_up = __shfl_sync(0xffffffffu, lane == 0 && load_acquire(p.status + SYNC_TABLE) > 0, 0);
        __syncwarp();                                             // lane 0 has acquired for all: a shuffle orders no memory accesses
        if (looked_up) look_up();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == C::QK_WARP) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
    if (p.fused) {
        int exited = 0;
        if (tid == 0) {                                           // after the __syncthreads: covers the stores of the whole CTA
            const int seen = add_acq_rel(p.status + SYNC_ARRIVE, 1);
            bool all = (seen & 0xffff) == n_cta - 1;
            if (!all && !(seen >> 16)) all = count_reached(p.status + SYNC_ARRIVE, n_cta, min(p.meet_cycles, NO_BIT_CYCLES));
            ms.meet = __builtin_expect(all && !(seen >> 16), 1) ? 0 : meet_late(ms, p.status, n_cta, cta, seen, all, p.meet_cycles);
        }
        __syncthreads();
        if (tid == 0) exited = atomicAdd(p.status + SYNC_EXIT, 1);        // looked at after the merge
        if (__builtin_expect(ms.meet == 0, 1)) {
            if (!looked_up) look_up();
            for (; (item >> sh) < rows_all; item += n_warps, look_up())
                if (work) merge_item(p, b, (item >> sh) - b * p.rows, w0, w1, item, sh, lane);
        } else {
            merge_late<TILE, N>(p, ms, item, sh);
        }
        if (tid == 0 && exited == n_cta - 1) {                    // the last one past the meeting: nobody looks at these any more
            p.status[SYNC_AMAX] = 0; p.status[SYNC_AMAX_COUNT] = 0; p.status[SYNC_TABLE] = 0; p.status[SYNC_ARRIVE] = 0; p.status[SYNC_EXIT] = 0;
            for (int i = 0; i < SYNC_MASK_WORDS; i += 4) {
                *reinterpret_cast<int4*>(p.status + SYNC_AMAX_DONE + i) = make_int4(0, 0, 0, 0);
                *reinterpret_cast<int4*>(p.status + SYNC_ARRIVED + i) = make_int4(0, 0, 0, 0);
                *reinterpret_cast<int4*>(p.status + SYNC_LEFT + i) = make_int4(0, 0, 0, 0);
            }
        }
    }
    if (tid == 0 && ms.abort_flag) report_status(p.status, ST_TIMEOUT);
}

}  // namespace sm100

namespace {

// Tensor map over a plane [rows x 576 bytes] with a box of `box_bytes` x `box_rows`; false if the driver entry point is
// missing or refuses the arguments (the kernel then copies with cp.async).
bool make_map(CUtensorMap* map, const void* base, long long rows, long long stride, int box_bytes, int box_rows, CUtensorMapSwizzle swizzle) {
    typedef CUresult (*encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const encode_fn encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) fn = nullptr;
        return (encode_fn)fn;
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)QK_DIM, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)stride};
    const cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The maps of an e4m3 cache plane: they depend on its address, row count and stride only, so the last few are kept per host
// thread (a serving loop that decodes from the same cache does not pay the driver calls, ~1.5 us each, on every call).
// This GPU's own plane only; no multi-CTA delivery of any kind.
const sm100::Maps* cache_maps(const MlaParams& p) {
    struct Entry { const void* codes; long long rows, stride; bool ok; sm100::Maps maps; };
    static thread_local Entry cache[8] = {};
    static thread_local int next = 0;
    if (((uintptr_t)p.kv_codes & 15) || p.kv_codes_stride % 16 || p.kv_codes_stride < QK_DIM || p.num_slots <= 0 || p.num_slots >= (1LL << 31)) return nullptr;
    for (Entry& m : cache)
        if (m.codes == p.kv_codes && m.rows == p.num_slots && m.stride == p.kv_codes_stride) return m.ok ? &m.maps : nullptr;
    Entry& m = cache[next];
    next = (next + 1) % 8;
    m.codes = p.kv_codes; m.rows = p.num_slots; m.stride = p.kv_codes_stride;
    memset(&m.maps, 0, sizeof(m.maps));
    m.ok = make_map(&m.maps.lat, m.codes, m.rows, m.stride, 128, 1, CU_TENSOR_MAP_SWIZZLE_128B) &&
           make_map(&m.maps.rope, m.codes, m.rows, m.stride, 64, 1, CU_TENSOR_MAP_SWIZZLE_64B) &&
           make_map(&m.maps.lat_box, m.codes, m.rows, m.stride, 128, sm100::UNIT_TOK, CU_TENSOR_MAP_SWIZZLE_128B) &&
           make_map(&m.maps.rope_box, m.codes, m.rows, m.stride, 64, sm100::UNIT_TOK, CU_TENSOR_MAP_SWIZZLE_64B);
    return m.ok ? &m.maps : nullptr;
}

template <int N, int KVFMT, int QFMT>
cudaError_t launch_cfg(const MlaParams& p, cudaStream_t stream) {
    using C = sm100::Cfg<N, KVFMT, QFMT>;
    auto kernel = sm100::mla_decode_sm100_kernel<N, KVFMT, QFMT>;
    static std::atomic<unsigned long long> sized{0};                  // bit d: the attribute is set on device d
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev > 63 || !(sized.load(std::memory_order_relaxed) >> dev & 1)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return e;
        if (dev <= 63) sized.fetch_or(1ULL << dev, std::memory_order_relaxed);
    }
    static const sm100::Maps no_maps = {};
    const sm100::Maps* maps = nullptr;
    const char* off = getenv("B200_MLA_DISABLE_TMA");                 // testing aid: "1" keeps every tile on the copy loop
    if (KVFMT == KV_E4M3 && !(off && off[0] == '1')) maps = cache_maps(p);
    return launch_pdl(kernel, dim3(p.num_ctas, p.rows / N), C::THREADS, C::SMEM, stream, p, maps ? *maps : no_maps, maps != nullptr);
}

template <int KVFMT>
cudaError_t dispatch(const MlaParams& p, cudaStream_t stream) {
    if (p.q_format == Q_BF16)
        return p.rows_per_cta == 32 ? launch_cfg<32, KVFMT, Q_BF16>(p, stream) : launch_cfg<16, KVFMT, Q_BF16>(p, stream);
    if (p.rows_per_cta == 64) return launch_cfg<64, KVFMT, Q_E4M3>(p, stream);
    return p.rows_per_cta == 32 ? launch_cfg<32, KVFMT, Q_E4M3>(p, stream) : launch_cfg<16, KVFMT, Q_E4M3>(p, stream);
}

}  // namespace

// Set-up units per sequence: about how many tiles a sequence boundary costs a CTA.  Two tiles of an e4m3 cache or of the
// 64-row kernels; one of a block-scaled cache below that, whose tiles take longer.  With one instead of two: 32 x 1024 MXFP4
// 18.4 -> 16.4 us, a rank of eight 34.8 -> 32.8; but e4m3 32 x 4096 26.9 -> 28.0, hybrid at 64 rows 391 -> 395.
int sm100_seq_units(const MlaParams& p) { return p.kv_format != KV_E4M3 && p.rows_per_cta < 64 ? 1 : 2; }

// Tokens per schedule tile, given p.rows_per_cta (Cfg::TILE).
int sm100_tile_tokens(const MlaParams& p) { return p.kv_format == KV_E4M3 && p.rows_per_cta < 64 ? 96 : 128; }

// The widest row group that divides the rows: a tile is fetched (and converted) once per group.  A bf16 Q doubles the
// QK columns and the shared memory of Q, so it stops at 32.
int sm100_rows_per_cta(const MlaParams& p) {
    if (p.rows % 64 == 0 && p.q_format == Q_E4M3) return 64;
    return p.rows % 32 == 0 ? 32 : 16;
}

// Block-scaled caches: the E8M0 rows must start on an even address.  Strides are multiplied as 32-bit numbers.
bool sm100_supported(const MlaParams& p) {
    if (p.kv_codes_stride >= (1LL << 31) || p.kv_bs_stride >= (1LL << 31) || p.kv_rope_stride >= (1LL << 31)) return false;
    return p.rows % 16 == 0 && (p.kv_format == KV_E4M3 || ((reinterpret_cast<uintptr_t>(p.kv_bs) | (uintptr_t)p.kv_bs_stride) & 1u) == 0);
}

cudaError_t launch_sm100(const MlaParams& p, cudaStream_t stream) {
    if (p.kv_format == KV_E4M3) return dispatch<KV_E4M3>(p, stream);
    return p.kv_format == KV_MXFP4 ? dispatch<KV_MXFP4>(p, stream) : dispatch<KV_HYBRID>(p, stream);
}

}  // namespace b200mla
