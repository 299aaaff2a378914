// Shared device-side definitions for the MLA decode kernels: kernel parameter block, the
// KV-span schedule that every CTA derives from kv_indptr, the merge of partials, and the
// byte-format decoders (e4m3fn, e2m1 + E8M0).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200mla {

constexpr int QK_DIM = 576;
constexpr int V_DIM = 512;
constexpr int ROPE_DIM = 64;
constexpr int MAX_BATCH = 8192;        // the warp-level kernel's tile-prefix table lives in shared memory

constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

enum { Q_BF16 = 0, Q_E4M3 = 1 };
constexpr int Q_AMAX_PARTS = 256;      // partial maxima handed over by the amax kernel when Q is cast on load
enum { KV_E4M3 = 0, KV_MXFP4 = 1, KV_HYBRID = 2 };
// Bits of the sticky status word at the head of the workspace (B200_MLA_STATUS_* in b200_mla.h).
enum { ST_OK = 0, ST_TIMEOUT = 1, ST_BAD_PAGE = 2 };

// Launch of a kernel all of whose threads call pdl_wait(): its blocks are placed while the kernel before it in the stream
// drains, which leaves 1 us between the two instead of 3 us.  pdl_wait returns when that kernel is complete and its writes
// are visible.  Before it a block may set up its own shared memory and nothing else: no global memory is read or written, and nothing
// taken that the kernel before could wait for (TMEM columns).  All but the decode kernel call it first of all.  What that kernel may have written is read with __ldcg or
// load_global: __ldg is for data that nobody writes while the kernel runs, and its blocks run already.
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, unsigned int threads, unsigned int smem, cudaStream_t stream, const Args&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename T>
__device__ __forceinline__ T load_global(const T* p) { return *p; }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Words of the 256-byte workspace header behind the status word.  ST_FORWARD: address (two words) of a second status word that
// receives the same bits, 0 if there is none.  ST_LEAVES: how many CTAs have left a meeting before all had come, in all launches
// so far (for tests and measurements).  SYNC_TABLE: MlaParams::seq_ctas has been written.  SYNC_*: for launches whose CTAs work together; they are zero between launches: the last
// CTA to exit resets them.  SYNC_AMAX_DONE, SYNC_ARRIVED, SYNC_LEFT: SYNC_MASK_WORDS words each, one bit per CTA.
enum { ST_FORWARD = 2, ST_LEAVES = 4, SYNC_AMAX = 16, SYNC_AMAX_COUNT = 17, SYNC_TABLE = 18, SYNC_AMAX_DONE = 20, SYNC_ARRIVE = 32, SYNC_ARRIVED = 36, SYNC_EXIT = 48,
       SYNC_LEFT = 52, SYNC_MASK_WORDS = 8 };
constexpr int MAX_FUSED_CTAS = 32 * SYNC_MASK_WORDS;

struct MlaParams {
    int batch, heads, q_len, rows;      // rows = q_len * heads (query rows per sequence)
    int q_format, kv_format, causal, page_size;
    float sm_scale;
    int num_ctas;                       // G: stage-1 CTAs along x (KV spans)
    int tile_tokens;                    // tokens per schedule tile (kernel specific)
    int seq_units;                      // set-up units per sequence of the schedule (kernel specific)
    int rows_per_cta;                   // query rows handled by one CTA (grid.y = rows / rows_per_cta)

    const void* q; long long q_row_stride, q_head_stride; const float* q_scale;
    const uint8_t* kv_codes; long long kv_codes_stride;
    const uint8_t* kv_bs; long long kv_bs_stride;
    const uint8_t* kv_rope; long long kv_rope_stride;
    const float* kv_scale; long long num_slots;
    unsigned int last_slot;             // min(num_slots, 2^31) - 1: the row an out-of-range page id is redirected to
    unsigned int last_page;             // last_slot / page_size: the last page id that names a row of the planes
    int page_shift;                     // log2(page_size), -1 if it is no power of two
    long long total_kv_hint;            // > 0: the host's bound on kv_indptr[batch]; kv_indices holds at least that many tokens' ids
    const int* kv_indptr; const int* kv_indices; const int* kv_page_indptr;
    const int* kv_pos_offset; const int* kv_total_len;

    __nv_bfloat16* out; float* out_o_f32; float* out_lse;
    float* part_o;                      // [G + batch - 1][rows][512] normalised partial O
    float* part_lse;                    // [G + batch - 1][rows]      natural-log LSE
    int2* seq_ctas;                     // [batch] first and last CTA (along x) that hold tiles of the sequence; (0, -1): none
                                        // (worked out once, by the first CTA; when each item of the merge did it from the tiles
                                        // before its sequence, three loads and two divisions: MXFP4 32 x 1024 14.05 us, 13.7 so)
    int* status;                        // sticky status word (bits ST_*), first word of the workspace
    int q_cast;                         // q is bf16 and is quantised to e4m3 (per-tensor, reference rule) as it is loaded;
    const unsigned int* q_amax_parts;   //   its scale comes from these Q_AMAX_PARTS partial maxima (bf16 bit patterns),
                                        //   or, nullptr, from the maximum the CTAs of the launch find together (SYNC_AMAX)
    int fused;                          // the CTAs of the launch also merge the partials, where they meet
    // How long a CTA waits for the others of its launch, twice: for the maximum of Q and before the merge.  They are all resident at
    // once unless something else holds SMs, but nothing depends on it: when the time is up, the CTA looks at shares of Q that
    // nobody has looked at yet, and merges what it can of its share of the rows; the rest goes to the CTAs that are late, each of which can be left with rows of
    // the sequences it holds and no others.  So the launch need not be cooperative, and it can overlap with the
    // end of the kernel before it (launch_pdl): 0.8 us between two kernels instead of 2.1, and no rounding up to ticks of 1 or 2 us,
    // which is how other launches of a stream start (e4m3 4 x 1024 12.3 -> 10.0 us a call, 32 x 4096 26.3 -> 23.9).
    int meet_cycles;
};

// ---------------------------------------------------------------------------------------------
// Schedule.  Sequence b owns tiles [P[b], P[b+1]) with ceil(len_b / tile_tokens) tiles.  The work is
// measured in units: one per tile plus K = p.seq_units per sequence (its Q load, first-tile re-centering
// and epilogues cost a CTA as much as one tile or two), so sequence b owns
// units [P[b] + K*b, P[b+1] + K*(b+1)) (K = 0 where tiles are few, see Sched), the first K being set-up units.  CTA w of G
// owns the units [w*TU/G, (w+1)*TU/G), TU = P[batch] + K*batch, i.e. the tiles those units stand
// for.  A (CTA, sequence) pair that does not cover the whole sequence writes a partial into slot
// w + b, which is unique because both coordinates are monotone along the chain of pairs.
// ---------------------------------------------------------------------------------------------
// Where there are no more tiles than CTAs, CTA w takes tile w: no set-up units (nothing is there to balance, and with them
// some CTAs would hold two tiles while others hold none) and only as many CTAs as tiles.
struct Sched {
    int k, units, G;                    // set-up units per sequence, all units, CTAs that hold any (each at least one unit)
};
__device__ __forceinline__ Sched make_sched(int total_tiles, int batch, int num_ctas, int seq_units) {
    return total_tiles <= num_ctas ? Sched{0, total_tiles, total_tiles} : Sched{seq_units, total_tiles + seq_units * batch, num_ctas};
}
// Unit at which CTA w's span begins (the end of all units for w >= G).  The 64-bit division is only taken where the product
// needs it (this runs in every CTA right after launch).
__device__ __forceinline__ int unit_begin(int w, const Sched& c) {
    if (w >= c.G) return c.units;
    return __umulhi((unsigned)w, (unsigned)c.units) == 0 ? (int)(((unsigned)w * (unsigned)c.units) / (unsigned)c.G) : (int)(((long long)w * c.units) / c.G);
}
// First tile of CTA w's span (w >= G gives the total number of tiles).
__device__ __forceinline__ int span_begin(const int* prefix, int batch, int w, int num_ctas, int seq_units) {
    const Sched c = make_sched(prefix[batch], batch, num_ctas, seq_units);
    const int u = unit_begin(w, c);
    if (u >= c.units) return prefix[batch];
    int lo = 0, hi = batch - 1;                               // the sequence that owns unit u: the first b with P[b+1] + k*(b+1) > u
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid + 1] + c.k * (mid + 1) > u) hi = mid; else lo = mid + 1;
    }
    return max(prefix[lo], u - c.k * (lo + 1));
}
// CTA whose span contains tile t of sequence b (unit t + k*(b+1)).
__device__ __forceinline__ int cta_of_tile(int t, int b, const Sched& c) {
    if (c.k == 0) return t;                                   // a tile per CTA
    const long long u = (long long)(t + c.k * (b + 1) + 1) * c.G + c.units - 1;
    return (u >> 32 ? (int)(u / c.units) : (int)((unsigned)u / (unsigned)c.units)) - 1;
}

// CTAs that hold tiles of sequence b, whose tiles are [t0, t1).
__device__ __forceinline__ int2 seq_span(int b, int t0, int t1, const Sched& c) {
    return t1 > t0 ? make_int2(cta_of_tile(t0, b, c), cta_of_tile(t1 - 1, b, c)) : make_int2(0, -1);
}

// ---------------------------------------------------------------------------------------------
// LSE merge of the partials of one query row, which the CTAs [w0, w1] hold (none for an empty sequence: zeros / -inf; nothing is to
// be done where there is one): this thread's V vectors of four output elements at d, d + 128, ... of row r.  Streaming, U partials
// per step so that their loads are in flight together; the loads bypass L1, which may hold lines from before another CTA wrote them.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void store_bf16x4(__nv_bfloat16* dst, float4 v) {
    __align__(8) __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(o);
}


template <int V, int U>
__device__ __forceinline__ void merge_row(const MlaParams& p, int b, int r, int w0, int w1, int d) {
    const long long orow = (long long)b * p.rows + r;
    float M = -INFINITY, den = 0.f;
    float4 acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int wb = w0; wb <= w1; wb += U) {
        float l[U];
        float4 x[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int w = wb + u;
            const bool ok = w <= w1;
            const long long slot = (long long)(w + b) * p.rows + r;
            l[u] = ok ? __ldcg(p.part_lse + slot) : -INFINITY;
#pragma unroll
            for (int v = 0; v < V; ++v)
                x[u][v] = ok ? __ldcg(reinterpret_cast<const float4*>(p.part_o + slot * V_DIM + d + 128 * v)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float m_new = M;
#pragma unroll
        for (int u = 0; u < U; ++u) m_new = fmaxf(m_new, l[u]);
        if (m_new > -INFINITY) {
            const float f = M > -INFINITY ? expf(M - m_new) : 0.f;
            den *= f;
#pragma unroll
            for (int v = 0; v < V; ++v) { acc[v].x *= f; acc[v].y *= f; acc[v].z *= f; acc[v].w *= f; }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float wt = expf(l[u] - m_new);              // 0 for an empty partial (-inf)
                den += wt;
#pragma unroll
                for (int v = 0; v < V; ++v) { acc[v].x += wt * x[u][v].x; acc[v].y += wt * x[u][v].y; acc[v].z += wt * x[u][v].z; acc[v].w += wt * x[u][v].w; }
            }
            M = m_new;
        }
    }
    const float inv = den > 0.f ? 1.0f / den : 1.0f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        acc[v].x *= inv; acc[v].y *= inv; acc[v].z *= inv; acc[v].w *= inv;
        if (p.out) store_bf16x4(p.out + orow * V_DIM + d + 128 * v, acc[v]);
        if (p.out_o_f32) *reinterpret_cast<float4*>(p.out_o_f32 + orow * V_DIM + d + 128 * v) = acc[v];
    }
    if (p.out_lse && d == 0) p.out_lse[orow] = den > 0.f ? M + logf(den) : -INFINITY;
}

// Fills prefix[0..batch] (shared memory) with the exclusive prefix of tiles per sequence.
// All threads of the block must call it; ends with a __syncthreads().
__device__ inline void build_tile_prefix(const int* __restrict__ kv_indptr, int batch, int tile_tokens,
                                         int* prefix) {
    for (int b = threadIdx.x; b < batch; b += blockDim.x) {
        int len = kv_indptr[b + 1] - kv_indptr[b];
        prefix[b + 1] = len > 0 ? (len + tile_tokens - 1) / tile_tokens : 0;
    }
    if (threadIdx.x == 0) prefix[0] = 0;
    __syncthreads();
    if (threadIdx.x < 32) {
        int carry = 0;
        for (int base = 1; base <= batch; base += 32) {
            int i = base + threadIdx.x;
            int v = i <= batch ? prefix[i] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int n = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += n;
            }
            v += carry;
            if (i <= batch) prefix[i] = v;
            carry = __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
}

// First sequence b with prefix[b+1] > t (sequence containing global tile t).
__device__ __forceinline__ int seq_of_tile(const int* prefix, int batch, int t) {
    int lo = 0, hi = batch - 1;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (prefix[mid + 1] > t) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// Cache slot of the token at position `pos` of sequence b, as the page table gives it (unchecked).
__device__ __forceinline__ long long slot_of(const MlaParams& p, int b, int seq_base, int page_base, int pos) {
    if (p.kv_indices == nullptr) return (long long)seq_base + pos;
    if (p.page_size == 1) return (long long)p.kv_indices[page_base + pos];
    int pg = pos / p.page_size;
    return (long long)p.kv_indices[page_base + pg] * p.page_size + (pos - pg * p.page_size);
}
// The same in pieces, for kernels that load a page id ahead of its use: entry of the sequence's part of the table that
// covers position `pos`, and the position's offset inside that page.
__device__ __forceinline__ int page_of(const MlaParams& p, int pos) { return p.page_shift >= 0 ? pos >> p.page_shift : pos / p.page_size; }
__device__ __forceinline__ int off_in_page(const MlaParams& p, int pos) { return p.page_shift >= 0 ? pos & (p.page_size - 1) : pos % p.page_size; }
// Row of the cache planes that is actually read for slot `s`: s itself inside [0, num_slots), else a row inside
// (negative values, the "no row" marker -1 included, map to the last row).  Nothing outside the planes is ever read;
// a key whose id needed the clamp reads as some other row, which is reported as ST_BAD_PAGE (by the tcgen05 kernels where the id
// becomes an address, by the warp-level kernel in check_span_pages).  The
// clamp is applied where a slot is turned into an address, not where it is loaded: the kernels load page ids one or
// two steps ahead of their use, and touching the value early would wait for that load (measured: 10-25 % of a call).
__device__ __forceinline__ unsigned int clamp_slot(const MlaParams& p, int s) { return min((unsigned int)s, p.last_slot); }

__device__ __forceinline__ void report_status(int* status, int bits) {
    atomicOr(status, bits);
    int* forward = *reinterpret_cast<int* const*>(status + ST_FORWARD);
    if (forward) atomicOr(forward, bits);
}

// Page ids of the tiles [t_begin, t_end) a stage-1 CTA owns: sets ST_BAD_PAGE if one of them names a page outside
// the cache planes (or, without a page table, if a token range reaches beyond them).  Called by `nthreads` threads
// (tid = 0 .. nthreads - 1) that have nothing else to do at the time; `tile` = tokens per tile.  Inlined: a call would
// make every thread of the kernel reserve a stack frame in local memory (measured: 19 MB of extra DRAM traffic per launch).
__device__ __forceinline__ void check_span_pages(const MlaParams& p, const int* prefix, int t_begin, int t_end, int tile,
                                              int tid, int nthreads) {
    bool bad = false;
    int b = seq_of_tile(prefix, p.batch, t_begin);
    for (int t = t_begin; t < t_end;) {
        while (prefix[b + 1] <= t) ++b;
        const int t1 = min(t_end, prefix[b + 1]);
        const int seq_base = p.kv_indptr[b], len = max(p.kv_indptr[b + 1] - seq_base, 0);
        const int pos0 = (t - prefix[b]) * tile, pos1 = min((t1 - prefix[b]) * tile, len);
        if (p.kv_indices != nullptr) {
            const int page_base = p.kv_page_indptr ? p.kv_page_indptr[b] : seq_base;
            const int e0 = pos0 / p.page_size, e1 = (pos1 + p.page_size - 1) / p.page_size;
            for (int e = e0 + tid; e < e1; e += nthreads) {
                const long long id = p.kv_indices[page_base + e];
                bad |= id < 0 || id * p.page_size >= p.num_slots;
            }
        } else if (tid == 0) {
            bad |= seq_base < 0 || (long long)seq_base + pos1 > p.num_slots;
        }
        t = t1;
    }
    if (bad) report_status(p.status, ST_BAD_PAGE);
}

// ---------------------------------------------------------------------------------------------
// Per-tensor e4m3 quantisation of Q, arithmetic order of the reference's quantize_fp8
// (competitor_submissions/mi355x_reference/reference.py:65-80): every intermediate is a bf16 value.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float q_scale_from_amax_bits(unsigned int bits) {
    float amax = __bfloat162float(__ushort_as_bfloat16((unsigned short)bits));
    amax = __bfloat162float(__float2bfloat16_rn(fmaxf(amax, 1e-12f)));
    return __bfloat162float(__float2bfloat16_rn(amax / 448.0f));
}
// x / scale rounded to bf16, as a float: the reference divides two bf16 tensors, i.e. an IEEE fp32 division whose
// result is rounded to bf16.  Evaluated without a division: t = x * r with r = RN(1 / scale), one exact residual
// and one correction (Markstein) give the correctly rounded fp32 quotient; checked exhaustively on the CPU against
// x / scale for every finite bf16 x and every positive normal bf16 scale (identical after the bf16 rounding and the
// clamp to +-448).  The sign is taken from x, so that -0 stays -0.
__device__ __forceinline__ float q_quotient_bf16(float x, float scale, float rscale) {
    const float t = x * rscale;
    float y = fmaf(fmaf(-t, scale, x), rscale, t);
    if (!(fabsf(t) <= 3.0e38f)) y = t;                                        // infinite / NaN input
    y = copysignf(fabsf(y), x);
    return __bfloat162float(__float2bfloat16_rn(y));
}
// Magnitude bits (exponent field f) of a bf16 x below which |x r| < 2^127 and finite: |x| < 2^(f - 126), |r| < 2^(e - 126), e the
// exponent field of r = RN(1 / scale).  Such quotients need no special cases.
__device__ __forceinline__ unsigned int general_from(float r) {
    const int e = (int)((__float_as_uint(r) >> 23) & 0xffu);
    return e == 255 ? 0u : (unsigned int)min(380 - e, 255) << 7;
}
// eight bf16 values (one 16-byte vector) -> eight e4m3 bytes
__device__ __forceinline__ uint2 q_cast_e4m3x8(const uint4& v, float scale) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};             // by value: the vector stays in registers
    const float r = __frcp_rn(scale);
    uint32_t o[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t word = w[2 * h + (k >> 1)];
            const float x = __uint_as_float((k & 1) ? (word & 0xffff0000u) : (word << 16));   // bf16 -> fp32
            y[k] = q_quotient_bf16(x, scale, r);
        }
        // the conversion saturates to +-448, which is the reference's clamp
        uint16_t lo16, hi16;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(lo16) : "f"(y[0]), "f"(y[1]));
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(hi16) : "f"(y[2]), "f"(y[3]));
        o[h] = (uint32_t)lo16 | ((uint32_t)hi16 << 16);
    }
    return make_uint2(o[0], o[1]);
}
// Scale of the e4m3 Q codes, the same value in every thread of the block.  All threads call it (it
// synchronises the block when the scale has to be reduced from the partial maxima); `word` is one
// 32-bit word of shared memory.
// block_q_amax_begin issues this thread's loads of the partial maxima (call it early, the result is
// only needed by block_q_scale); without a cast it returns 0 and touches nothing.
__device__ __forceinline__ unsigned int block_q_amax_begin(const unsigned int* amax_parts, int q_cast) {
    unsigned int m = 0;
    if (q_cast)
        for (int i = threadIdx.x; i < Q_AMAX_PARTS; i += blockDim.x) m = max(m, __ldg(amax_parts + i));
    return m;
}
__device__ inline float block_q_scale(unsigned int m, const float* q_scale, int q_cast, unsigned int* word) {
    if (!q_cast) return q_scale ? __ldg(q_scale) : 1.0f;
    if (threadIdx.x == 0) *word = 0u;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(word, m);
    __syncthreads();
    return q_scale_from_amax_bits(*word);
}

// ---------------------------------------------------------------------------------------------
// byte formats
// ---------------------------------------------------------------------------------------------

// two e4m3fn bytes (low 16 bits) -> two halves (exact)
__device__ __forceinline__ __half2 e4m3x2_to_half2(uint16_t v) {
    __half2_raw r = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)v, __NV_E4M3);
    return *reinterpret_cast<__half2*>(&r);
}

__device__ __forceinline__ float e4m3_to_float(uint8_t v) {
    __half_raw r = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)v, __NV_E4M3);
    return __half2float(*reinterpret_cast<__half*>(&r));
}

// E8M0 byte -> float 2^(b-127).  Byte 0 gives 2^-127 (a denormal), 255 is NaN in the format.
__device__ __forceinline__ float e8m0_to_float(uint8_t b) {
    if (b == 255) return __int_as_float(0x7fc00000);
    return b == 0 ? __int_as_float(0x00400000) : __int_as_float((int)b << 23);
}

// e2m1 code (4 bits, bit3 = sign) -> float
__device__ __forceinline__ float e2m1_to_float(uint32_t c) {
    // magnitudes 0, .5, 1, 1.5, 2, 3, 4, 6
    uint32_t mag = c & 7u;
    float v = mag < 2u ? 0.5f * (float)mag
                       : __int_as_float((int)(((mag >> 1) + 126u) << 23) | (int)((mag & 1u) << 22));
    return (c & 8u) ? -v : v;
}

}  // namespace b200mla
