// Log-sum-exp combine kernels.
//
//  * combine_spans_kernel merges the partials that stage-1 CTAs wrote for sequences whose tiles
//    were spread over several KV spans (slot = cta + sequence, see mla_common.cuh), writes zeros
//    for empty sequences and leaves alone the sequences a single CTA finished by itself.
//  * combine_parts_kernel merges `parts` dense partial results [parts, rows, 512] + [parts, rows],
//    the form an all-gather of per-GPU shards produces.
//
// Math (natural-log LSE, normalised partial O):  M = max_i LSE_i,  w_i = exp(LSE_i - M),
// O = sum_i w_i O_i / sum_i w_i,  LSE = M + log(sum_i w_i); an empty part has LSE = -inf and weight 0.
// Role in the reference: _mla_mxfp4_reduce (mixed-mla/submission.py:257-294), aiter.mla_reduce_v1,
// stage 2 of competitor_submissions/dgavriloff_v114_hybrid_mxfp4k_fp8v.py:131-160.
#include "mla_common.cuh"

namespace b200mla {

namespace {

__global__ void __launch_bounds__(128) combine_spans_kernel(const MlaParams p) {
    pdl_wait();
    const int b = blockIdx.x;
    const int2 ctas = p.seq_ctas[b];
    if (ctas.x != ctas.y) merge_row<1, 4>(p, b, blockIdx.y, ctas.x, ctas.y, threadIdx.x * 4);
}

constexpr int GROUP = 8;                // parts whose loads are in flight together: the GPUs of a node

__global__ void __launch_bounds__(128) combine_parts_kernel(const float* __restrict__ o_parts,
                                                            const float* __restrict__ lse_parts, int parts,
                                                            long long rows, long long o_stride, long long lse_stride,
                                                            __nv_bfloat16* out, float* out_lse) {
    pdl_wait();
    const long long r = blockIdx.x;
    const int d = threadIdx.x * 4;
    // A row is a few kilobytes: what counts is that its loads are in flight together, those of the LSEs included (with
    // pdl_wait, 4 us less for the eight records of 256 rows behind a decode than one part after the other).
    float lse[GROUP];
    float4 v[GROUP];
    auto load = [&](int i0) {
#pragma unroll
        for (int k = 0; k < GROUP; ++k)
            if (i0 + k < parts) lse[k] = __ldcg(lse_parts + (i0 + k) * lse_stride + r);
#pragma unroll
        for (int k = 0; k < GROUP; ++k)
            if (i0 + k < parts) v[k] = __ldcg(reinterpret_cast<const float4*>(o_parts + (i0 + k) * o_stride + r * V_DIM + d));
    };
    load(0);
    float M = -INFINITY;
#pragma unroll
    for (int k = 0; k < GROUP; ++k)
        if (k < parts) M = fmaxf(M, lse[k]);
    for (int i = GROUP; i < parts; ++i) M = fmaxf(M, __ldcg(lse_parts + i * lse_stride + r));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float den = 0.f;
    if (M > -INFINITY) {
        for (int i0 = 0; i0 < parts; i0 += GROUP) {
            if (i0 > 0) load(i0);
#pragma unroll
            for (int k = 0; k < GROUP; ++k)
                if (i0 + k < parts) {
                    const float wt = expf(lse[k] - M);
                    acc.x += wt * v[k].x; acc.y += wt * v[k].y; acc.z += wt * v[k].z; acc.w += wt * v[k].w;
                    den += wt;
                }
        }
        const float inv = 1.0f / den;
        acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
    }
    store_bf16x4(out + r * V_DIM + d, acc);
    if (out_lse && threadIdx.x == 0) out_lse[r] = den > 0.f ? M + logf(den) : -INFINITY;
}

}  // namespace

cudaError_t launch_combine_spans(const MlaParams& p, cudaStream_t stream) {
    dim3 grid(p.batch, p.rows);
    return launch_pdl(combine_spans_kernel, grid, 128, 0, stream, p);
}

cudaError_t launch_combine_parts(const float* o_parts, const float* lse_parts, int parts, long long rows,
                                 long long o_stride, long long lse_stride, __nv_bfloat16* out, float* out_lse,
                                 cudaStream_t stream) {
    return launch_pdl(combine_parts_kernel, dim3((unsigned)rows), 128, 0, stream, o_parts, lse_parts, parts, rows, o_stride, lse_stride, out,
                      out_lse);
}

}  // namespace b200mla
