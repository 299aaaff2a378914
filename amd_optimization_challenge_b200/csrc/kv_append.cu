// KV-cache append: bf16 latent rows [n, 576] -> rows of an FP8, MXFP4 or hybrid cache at given slots.
//
// The inverse of what the decode kernels read, with the arithmetic of the reference's quantisers so that a
// cache filled on the device holds the same bytes as one quantised by the reference on the host:
//   * e4m3 codes: x / scale rounded to bf16, clamped to +-448, cast (quantize_fp8,
//     competitor_submissions/mi355x_reference/reference.py:65-80).  The per-tensor scale is an input here:
//     rows appended later cannot change the scale of rows already in the cache.
//   * MXFP4: per block of 32 elements the E8M0 exponent floor(log2(amax rounded up at mantissa 1.75)) - 2 and
//     e2m1 codes rounded to nearest even (aiter's dynamic_mxfp4_quant as restated in
//     mxfp4-mm/submission_v3_self_contained.py:19-72; reference.py:88-113), two codes per byte, even element
//     in the low nibble.
//   * hybrid: dims 0..511 as MXFP4 (16 blocks), dims 512..575 as e4m3 with the per-tensor rope scale.
// One thread quantises eight elements, or sixteen of an e4m3 row (16 bytes a load; 16 or 4 a store), so that neighbouring lanes
// read and write neighbouring bytes; the four lanes of a 32-element block share its exponent by two shuffles.  HBM bound from
// some ten thousand rows on, launch and load latency below.
#include "mla_common.cuh"
#include "sm100_ptx.cuh"

namespace b200mla {

namespace {

using namespace sm100;

struct AppendParams {
    const __nv_bfloat16* src; long long n; long long src_stride;   // elements between rows
    const int* slots; long long base_slot; long long num_slots;
    uint8_t* codes; long long codes_stride;
    uint8_t* bs; long long bs_stride;
    uint8_t* rope; long long rope_stride;
    const float* scale;
    int* bad;                                                       // set to 1 if a slot is outside [0, num_slots)
    int write_status;                                               // the last block looks the slots over and writes *bad, 0 or 1
};

constexpr int THREADS = 288;
constexpr int resident(bool ahead) { return ahead ? 4 : 7; }        // blocks on an SM
constexpr int vectors(int kv_format) { return kv_format == KV_E4M3 ? 2 : 1; }                   // of eight elements per thread
constexpr int block_rows(int kv_format) { return THREADS * 8 * vectors(kv_format) / QK_DIM; }   // rows a block covers at a time

__device__ __forceinline__ f32x2 widen(uint32_t w) { return pk2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// Eight bf16 values -> their e4m3 codes, the codes of q_cast_e4m3x8 (mla_common.cuh) for every input: two values per
// instruction, and vectors that may need its special cases (infinite or NaN quotients) are left to it: those with a value whose
// magnitude bits reach `general` (general_from).  r = RN(1 / scale).
__device__ __forceinline__ uint2 cast_e4m3x8(const uint4& v, float scale, float r, unsigned int general) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const f32x2 s2 = pk2(-scale, -scale), r2 = pk2(r, r);
    uint32_t c[4], m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        m = __vmaxu2(m, w[k] & 0x7fff7fffu);
        const f32x2 x = widen(w[k]), t = mul2(x, r2);
        float y0, y1;
        unpk2(fma2(fma2(t, s2, x), r2, t), y0, y1);
        uint32_t h;
        asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(h) : "f"(y0), "f"(y1));
        h = (h & 0x7fff7fffu) | (w[k] & 0x80008000u);                         // -0 stays -0
        unpk2(widen(h), y0, y1);
        uint16_t q;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(q) : "f"(y0), "f"(y1));
        c[k] = q;
    }
    if (max(m & 0xffffu, m >> 16) >= general) return q_cast_e4m3x8(v, scale);
    return make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
}
// Eight bf16 values of a 32-element block whose other values are in the lanes of the same aligned group of four -> eight
// e2m1 codes and the block's E8M0 byte.  All 32 lanes call it.
__device__ __forceinline__ uint32_t quant_mxfp4x8(const uint4& v, uint8_t& scale_byte) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float x[8], amax = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) unpk2(widen(w[k]), x[2 * k], x[2 * k + 1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) asm("max.NaN.f32 %0, %0, %1;" : "+f"(amax) : "f"(fabsf(x[i])));
    const bool nan = amax != amax;
    if (nan) {                                                    // NaNs do not count towards the exponent
        amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    // next power of two when the mantissa is >= 1.75, then two binades of headroom for the largest code (6 = 1.5 * 4)
    const unsigned int bits = ((unsigned int)__float_as_int(amax) + 0x200000u) & 0xFF800000u;
    const int e_field = (int)(bits >> 23);
    int e = e_field == 0 ? -127 : e_field - 127 - 2;
    e = max(-127, min(e, 127));
    scale_byte = (uint8_t)(e + 127);
    // 2^-e, also where it is a subnormal (e = 127)
    const float inv = e <= 126 ? __int_as_float((127 - e) << 23) : __int_as_float(0x00400000);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= inv;
    uint32_t codes;                                               // to nearest even, saturating at 6; the even element in the low nibble
    asm("{ .reg .b8 t0, t1, t2, t3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n\t"
        "mov.b32 %0, {t0, t1, t2, t3}; }"
        : "=r"(codes) : "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]));
    if (nan) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (x[i] != x[i]) codes = (codes & ~(0xfu << (4 * i))) | (0x4u << (4 * i));   // a NaN is stored as 2
    }
    return codes;
}

// Instructions bound it next to HBM, so a thread keeps pointers and advances them, and an e4m3 thread has two vectors: 500000
// rows into an e4m3 cache (864 MB moved) 158 us with listed slots and 146 without, 205 and 176 with one vector and 64-bit
// products per row (all with seven blocks).  A block's first loads are issued before anything that waits for the scale.  Seven resident blocks of
// 32 registers a thread, one step in flight each; with AHEAD four, whose next rows are on their way while a step is converted and
// stored (see launch_format): that takes 51 registers, and 56 are given out.
template <int KVFMT, bool LISTED, bool AHEAD>
__global__ void __launch_bounds__(THREADS, resident(AHEAD)) kv_append_kernel(const AppendParams p) {
    pdl_wait();
    constexpr int VEC = vectors(KVFMT), CHUNKS = QK_DIM / 8 / VEC, STEP = block_rows(KVFMT);
    const int lead = p.write_status;
    const unsigned int top = (unsigned int)min(p.num_slots, 1ll << 31);               // a negative slot is above it
    if ((int)blockIdx.x < lead) {
        // Slots are looked over once more by one block: *bad has to be 0 where all are good, and nobody zeroes it before.
        // Single ones up to a 16-byte boundary and after the last, four at a time between: a list that is a slice of a longer one
        // starts anywhere (500000 rows, e4m3: 167 us one word at a time, 158 so).
        bool any = false;
        if (LISTED) {
            const int tid = (int)threadIdx.x, head = (int)min((long long)((0u - (unsigned int)(uintptr_t)p.slots) >> 2 & 3u), p.n);
            const long long n4 = (p.n - head) >> 2, tail = head + 4 * n4;
            const int4* s4 = reinterpret_cast<const int4*>(p.slots + head);
            if (tid < head) any = (unsigned int)__ldcg(p.slots + tid) >= top;
            if (tail + tid < p.n) any |= (unsigned int)__ldcg(p.slots + tail + tid) >= top;
#pragma unroll 8
            for (long long i = tid; i < n4; i += THREADS) {
                const int4 s = __ldcg(s4 + i);
                any |= max(max((unsigned int)s.x, (unsigned int)s.y), max((unsigned int)s.z, (unsigned int)s.w)) >= top;
            }
        }
        any = __syncthreads_or(any);
        if (threadIdx.x == 0) *p.bad = any ? 1 : 0;
        return;
    }
    const int sub = (int)threadIdx.x / CHUNKS, chunk = (int)threadIdx.x - sub * CHUNKS;
    const long long hop = (long long)((int)gridDim.x - lead) * STEP, row0 = (long long)((int)blockIdx.x - lead) * STEP;
    const uint4* src = reinterpret_cast<const uint4*>(p.src + (row0 + sub) * p.src_stride) + chunk * VEC;
    const long long src_hop = hop * p.src_stride / 8;
    const int* list = p.slots + row0 + sub;
    long long to = p.base_slot + row0 + sub;                                          // row of the cache, where no slots are listed
    long long left = p.n - row0;                                                      // rows from the block's first one on
    uint4 v[VEC], next[VEC];
    unsigned int slot, next_slot;
    auto fetch = [&](uint4 (&v)[VEC], unsigned int& slot) {
        slot = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < VEC; ++k) v[k] = make_uint4(0u, 0u, 0u, 0u);
        if (sub < left) {
            if (LISTED) slot = (unsigned int)__ldcg(list);
#pragma unroll
            for (int k = 0; k < VEC; ++k) v[k] = __ldcg(src + k);
        }
        src += src_hop;
        list += hop;
    };
    const float scale = KVFMT != KV_MXFP4 ? __ldcg(p.scale) : 1.0f;
    fetch(v, slot);
    const float rscale = __frcp_rn(scale);
    const unsigned int general = general_from(rscale);
    for (;;) {                                                                        // the same number of steps for the whole block
        const bool mine = sub < left;
        left -= hop;
        if (AHEAD && left > 0) fetch(next, next_slot);
        const bool ok = LISTED ? slot < top : mine;                // nothing is written elsewhere
        if (LISTED) {
            if (mine && !ok && !p.write_status) *p.bad = 1;
            to = (long long)slot;
        }
        if constexpr (KVFMT == KV_E4M3) {
            static_assert(VEC == 2, "one 16-byte store");
            if (ok) {
                const uint2 a = cast_e4m3x8(v[0], scale, rscale, general), b = cast_e4m3x8(v[1], scale, rscale, general);
                reinterpret_cast<uint4*>(p.codes + to * p.codes_stride)[chunk] = make_uint4(a.x, a.y, b.x, b.y);
            }
        } else {
            uint8_t sb;
            const uint32_t codes = quant_mxfp4x8(v[0], sb);
            if (KVFMT == KV_HYBRID && chunk >= V_DIM / 8) {
                if (ok) reinterpret_cast<uint2*>(p.rope + to * p.rope_stride)[chunk - V_DIM / 8] = cast_e4m3x8(v[0], scale, rscale, general);
            } else if (ok) {
                reinterpret_cast<uint32_t*>(p.codes + to * p.codes_stride)[chunk] = codes;
                if ((chunk & 3) == 0) p.bs[to * p.bs_stride + (chunk >> 2)] = sb;
            }
        }
        if (left <= 0) break;
        to += hop;
        if constexpr (AHEAD) {
            slot = next_slot;
#pragma unroll
            for (int k = 0; k < VEC; ++k) v[k] = next[k];
        } else {
            fetch(v, slot);
        }
    }
}

// The status block counts as one of a single wave's: one block more waits for another to leave and then takes all of its steps behind
// them (us with rows in HBM, a block more and not: listed e4m3 16384 rows 7.33 and 6.96, 24000 rows 10.3 and 9.0; listed MXFP4 16384 rows
// 7.09 and 6.76).
template <int KVFMT, bool LISTED, bool AHEAD>
cudaError_t launch_waves(const AppendParams& p, long long steps, int waves, cudaStream_t stream) {
    const long long blocks = waves * 148 * resident(AHEAD) - (waves == 1 ? p.write_status : 0);
    return launch_pdl(kv_append_kernel<KVFMT, LISTED, AHEAD>, (unsigned int)((steps < blocks ? steps : blocks) + p.write_status), THREADS, 0, stream, p);
}
// Seven blocks on an SM: up to eight steps per block of a single wave the blocks stay and loop (unlisted e4m3, 16384 rows 5.7 us, 7.2 with
// a second wave); beyond that four waves even out what the blocks take (131072 rows 40.3 us, 44.5 with one).
// Listed rows of an e4m3 cache have the slot's load in front of each step: one wave of four blocks that fetch a step ahead takes them.  Up to
// five blocks on an SM have one step each, nothing to fetch ahead, and more bytes in flight without (us, seven blocks and four ahead, rows that
// a kernel has just written, i.e. in L2 | in HBM: 512 rows 1.47 and 1.56 | 2.04 and 2.09, 4736 2.88 and 3.06 | 3.38 and 3.63, 5500 3.27 and 3.27 |
// 3.71 and 4.14).  Above that four are faster for rows in L2, and for rows in HBM from 7400 on but for two to three steps a block (6000
// 3.49 and 3.40 | 3.91 and 4.26, 7104 3.93 and 3.60 | 4.38 and 4.46, 7400 4.28 and 3.71 | 4.59 and 4.51, 9000 4.59 and 4.01 | 5.00 and 4.86, 12000
// 4.89 and 4.61 | 5.61 and 5.82, 16384 6.14 and 5.86 | 6.98 and 6.98, 24000 8.36 and 8.27 | 8.97 and 8.99, 50000 17.8 and 16.2 |
// 18.3 and 16.5, 131072 41.0 and 40.3 | 40.6 and 40.5, 500000 157 and 149 | 157 and 150).
template <int KVFMT>
cudaError_t launch_format(const AppendParams& p, cudaStream_t stream) {
    const long long steps = (p.n + block_rows(KVFMT) - 1) / block_rows(KVFMT);
    constexpr bool AHEAD = KVFMT == KV_E4M3;
    if (AHEAD && p.slots && steps > 148 * 5) return launch_waves<KVFMT, true, AHEAD>(p, steps, 1, stream);
    const int waves = steps <= 8 * 148 * resident(false) ? 1 : 4;
    return p.slots ? launch_waves<KVFMT, true, false>(p, steps, waves, stream) : launch_waves<KVFMT, false, false>(p, steps, waves, stream);
}

}  // namespace

cudaError_t launch_kv_append(const void* src, long long n, long long src_stride, const int* slots, long long base_slot,
                             long long num_slots, int kv_format, void* codes, long long codes_stride, void* bs,
                             long long bs_stride, void* rope, long long rope_stride, const float* scale, int* bad,
                             bool write_status, cudaStream_t stream) {
    AppendParams p;
    p.src = (const __nv_bfloat16*)src; p.n = n; p.src_stride = src_stride;
    p.slots = slots; p.base_slot = base_slot; p.num_slots = num_slots;
    p.codes = (uint8_t*)codes; p.codes_stride = codes_stride;
    p.bs = (uint8_t*)bs; p.bs_stride = bs_stride;
    p.rope = (uint8_t*)rope; p.rope_stride = rope_stride;
    p.scale = scale; p.bad = bad; p.write_status = write_status ? 1 : 0;
    if (kv_format == KV_E4M3) return launch_format<KV_E4M3>(p, stream);
    return kv_format == KV_MXFP4 ? launch_format<KV_MXFP4>(p, stream) : launch_format<KV_HYBRID>(p, stream);
}

}  // namespace b200mla
