// fp32 MatMul on CUDA cores for products that are too small for the tensor-core form (gemm_tc32.cu), whose conversions, tensor-memory
// set-up and 64-value k-blocks cost 8 us before the first result: few rows (a short prompt, a generation step), or a batch of small
// matrices (attention spelt with MatMul).  MatMulInfo semantics (src/04kernel/src/attributes/mat_mul_info.cc:27-42), trans_a = 0.
//
// A CTA computes a 32 x 32 tile; its eight warps divide k and each computes the whole tile for its share, so that a product with a
// handful of tiles still has eight times as many independent chains, and the sum of eight short chains is closer to the exact one
// than a long chain.  Per warp, 16 values of k at a time: operands one step ahead in registers (16-byte loads where rows are aligned),
// a private piece of shared memory (no barrier between warps), 8 x 4 results per lane from three 16-byte shared loads per k: the
// multiply-adds are the bound (32 cycles of the warp's scheduler per k against 3 of the shared-memory port).  The eight partial
// tiles are added through shared memory in a fixed order.
// Against gemm_tc32.cu: 32 x 256 x 256 4.1 us and 9.0, 128 x 256 x 256 4.8 and 13.7, 16 x 256 x 688 8.3 and 12.6, 32 x 1024 x 1024 14.1 and
// 14.3, 509 x 1024 x 1024 37.4 and 20.6; the operator graph of a two-layer 256-wide model on 32 tokens 221 -> 146 us.
#include "common.cuh"
#include "gemm_dispatch.cuh"

namespace rg {

constexpr int S3_T = 32, S3_K = 16, S3_WARPS = 8, S3_PITCH = 36;// pitch: rows of 144 bytes keep 16-byte alignment

struct Small32Args {
    const float *A, *B, *C;
    float *Y;
    uint32_t m, n, k, n_tiles;
    uint64_t stride_a, stride_b, stride_c, stride_y;
    uint32_t c_row, c_col;
    float alpha, beta;
};

// Four k-consecutive values of row r (operands with k innermost) from k0; zeros outside
template<bool VEC>
__device__ __forceinline__ float4 s3_row(const float *x, uint32_t r, uint32_t rows, uint32_t k0, uint32_t k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r >= rows) return v;
    const float *p = x + static_cast<uint64_t>(r) * k + k0;
    if constexpr (VEC) {// k is a multiple of 4
        if (k0 < k) v = __ldg(reinterpret_cast<const float4 *>(p));
    } else {
        if (k0 < k) v.x = __ldg(p);
        if (k0 + 1 < k) v.y = __ldg(p + 1);
        if (k0 + 2 < k) v.z = __ldg(p + 2);
        if (k0 + 3 < k) v.w = __ldg(p + 3);
    }
    return v;
}
// Four consecutive columns of row kk of B [k, n]
template<bool VEC>
__device__ __forceinline__ float4 s3_cols(const float *x, uint32_t kk, uint32_t k, uint32_t c0, uint32_t n) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kk >= k) return v;
    const float *p = x + static_cast<uint64_t>(kk) * n + c0;
    if constexpr (VEC) {// n is a multiple of 4
        if (c0 < n) v = __ldg(reinterpret_cast<const float4 *>(p));
    } else {
        if (c0 < n) v.x = __ldg(p);
        if (c0 + 1 < n) v.y = __ldg(p + 1);
        if (c0 + 2 < n) v.z = __ldg(p + 2);
        if (c0 + 3 < n) v.w = __ldg(p + 3);
    }
    return v;
}

template<bool TRANS_B, bool VEC>
__global__ void __launch_bounds__(S3_WARPS * 32) gemm_small32_kernel(const Small32Args a) {
    __shared__ __align__(16) float smem[S3_WARPS * 2 * S3_K * S3_PITCH];// per warp A [16][36] and B [16][36]; then the partial tiles
    pdl_enter();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nt = blockIdx.x % a.n_tiles, mt = blockIdx.x / a.n_tiles, b = blockIdx.y;
    const float *A = a.A + b * a.stride_a, *B = a.B + b * a.stride_b;
    float *As = smem + warp * (2 * S3_K * S3_PITCH), *Bs = As + S3_K * S3_PITCH;
    const uint32_t steps = (a.k + S3_K - 1) / S3_K, s0 = steps * warp / S3_WARPS, s1 = steps * (warp + 1) / S3_WARPS;
    float4 ra[4], rb[4];
    auto fetch = [&](uint32_t s) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // four lanes read the 64 bytes of a row: a load touches 8 rows (with a row per lane it touched 32, and that was the bound)
            ra[i] = s3_row<VEC>(A, mt * S3_T + lane / 4 + 8 * i, a.m, s * S3_K + lane % 4 * 4, a.k);
            if constexpr (TRANS_B) rb[i] = s3_row<VEC>(B, nt * S3_T + lane / 4 + 8 * i, a.n, s * S3_K + lane % 4 * 4, a.k);
            else
                rb[i] = s3_cols<VEC>(B, s * S3_K + 4 * i + lane / 8, a.k, nt * S3_T + lane % 8 * 4, a.n);
        }
    };
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const uint32_t row = lane / 8 * 8, col = lane % 8 * 4;
    if (s0 < s1) fetch(s0);
    for (uint32_t s = s0; s < s1; ++s) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float *at = As + lane % 4 * 4 * S3_PITCH + lane / 4 + 8 * i;
            at[0] = ra[i].x, at[S3_PITCH] = ra[i].y, at[2 * S3_PITCH] = ra[i].z, at[3 * S3_PITCH] = ra[i].w;
            if constexpr (TRANS_B) {
                float *bt = Bs + lane % 4 * 4 * S3_PITCH + lane / 4 + 8 * i;
                bt[0] = rb[i].x, bt[S3_PITCH] = rb[i].y, bt[2 * S3_PITCH] = rb[i].z, bt[3 * S3_PITCH] = rb[i].w;
            } else {
                *reinterpret_cast<float4 *>(Bs + (4 * i + lane / 8) * S3_PITCH + lane % 8 * 4) = rb[i];
            }
        }
        __syncwarp();
        if (s + 1 < s1) fetch(s + 1);
#pragma unroll
        for (int kk = 0; kk < S3_K; ++kk) {
            const float4 x0 = *reinterpret_cast<const float4 *>(As + kk * S3_PITCH + row), x1 = *reinterpret_cast<const float4 *>(As + kk * S3_PITCH + row + 4);
            const float4 w = *reinterpret_cast<const float4 *>(Bs + kk * S3_PITCH + col);
            const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i][0] = fmaf(x[i], w.x, acc[i][0]), acc[i][1] = fmaf(x[i], w.y, acc[i][1]);
                acc[i][2] = fmaf(x[i], w.z, acc[i][2]), acc[i][3] = fmaf(x[i], w.w, acc[i][3]);
            }
        }
        __syncwarp();
    }
    __syncthreads();// the operands of all warps have been read: their memory takes the partial tiles [warp][32][36]
    float *mine = smem + warp * (S3_T * S3_PITCH);
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<float4 *>(mine + (row + i) * S3_PITCH + col) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    // one thread per four results
    const uint32_t tr = threadIdx.x / 8, tc = threadIdx.x % 8 * 4, gr = mt * S3_T + tr, gc = nt * S3_T + tc;
    if (gr >= a.m || gc >= a.n) return;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < S3_WARPS; ++w) {
        const float4 v = *reinterpret_cast<const float4 *>(smem + w * (S3_T * S3_PITCH) + tr * S3_PITCH + tc);
        sum[0] += v.x, sum[1] += v.y, sum[2] += v.z, sum[3] += v.w;
    }
    float *y = a.Y + b * a.stride_y + static_cast<uint64_t>(gr) * a.n + gc;
    const float *c = a.C ? a.C + b * a.stride_c + static_cast<uint64_t>(gr) * a.c_row + static_cast<uint64_t>(gc) * a.c_col : nullptr;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sum[j] *= a.alpha;
        if (c && gc + j < a.n) sum[j] += a.beta * c[static_cast<uint64_t>(j) * a.c_col];
    }
    if (gc + 4 <= a.n && (reinterpret_cast<uintptr_t>(y) & 15u) == 0) {
        *reinterpret_cast<float4 *>(y) = make_float4(sum[0], sum[1], sum[2], sum[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (gc + j < a.n) y[j] = sum[j];
    }
}

bool gemm_small32_supported(const rg_mat_mul_params *p) {
    const uint64_t tiles = static_cast<uint64_t>((p->m + S3_T - 1) / S3_T) * ((p->n + S3_T - 1) / S3_T);
    return p->dtype == RG_F32 && !p->trans_a && tiles <= 0x7fffffffull && p->batch <= 65535;
}
// Estimated time: launch and the last reduction 3 us, 12.5 ns per value of k for the first tile on an SM; each further one 0.85 us and 7.3 ns
// per value of k
float gemm_small32_us(const rg_mat_mul_params *p) {
    const uint64_t tiles = static_cast<uint64_t>((p->m + S3_T - 1) / S3_T) * ((p->n + S3_T - 1) / S3_T) * p->batch, sms = static_cast<uint64_t>(sm_count());
    return 3.f + 0.0125f * static_cast<float>(p->k) + static_cast<float>((tiles + sms - 1) / sms - 1) * (0.85f + 0.0073f * static_cast<float>(p->k));
}
int gemm_small32(const rg_mat_mul_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    if (!gemm_small32_supported(p)) return RG_ERR_UNSUPPORTED;
    Small32Args a = {};
    a.A = static_cast<const float *>(in[0]), a.B = static_cast<const float *>(in[1]), a.C = p->has_bias ? static_cast<const float *>(in[2]) : nullptr;
    a.Y = static_cast<float *>(out[0]);
    a.m = p->m, a.n = p->n, a.k = p->k, a.n_tiles = (p->n + S3_T - 1) / S3_T;
    a.stride_a = p->stride_a, a.stride_b = p->stride_b, a.stride_c = p->stride_c, a.stride_y = p->stride_y;
    a.c_row = p->bias_row_stride, a.c_col = p->bias_col_stride, a.alpha = p->alpha, a.beta = p->beta;
    const bool vec = aligned16(in[0]) && aligned16(in[1]) && p->k % 4 == 0 && (p->trans_b || p->n % 4 == 0) && p->stride_a % 4 == 0 && p->stride_b % 4 == 0;
    auto kern = p->trans_b ? (vec ? gemm_small32_kernel<true, true> : gemm_small32_kernel<true, false>)
                           : (vec ? gemm_small32_kernel<false, true> : gemm_small32_kernel<false, false>);
    RG_CHECK_CUDA(launch_pdl(kern, dim3(a.n_tiles * ((p->m + S3_T - 1) / S3_T), p->batch), dim3(S3_WARPS * 32), 0, st, a));
    count_launch();
    return launch_status();
}

}// namespace rg
