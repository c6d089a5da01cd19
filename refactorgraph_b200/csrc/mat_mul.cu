// rg_b200_mat_mul: routes a MatMul (MatMulInfo semantics, src/04kernel/src/attributes/mat_mul_info.cc:27-42)
// to one of the hand-written kernels (16 bits: streaming GEMV, skinny, tcgen05, CUDA cores; fp32: tcgen05, 32 x 32 tiles, CUDA cores).
// No vendor GEMM is linked.
#include "gemm_dispatch.cuh"
#include <cstdlib>

using namespace rg;

static bool gemv_shape(const rg_mat_mul_params *p) {
    return (p->dtype == RG_FP16 || p->dtype == RG_BF16) && !p->trans_a && p->trans_b && p->m <= 4 && p->batch == 1 &&
           !p->has_bias && p->alpha == 1.0f && p->k % 8 == 0 && p->k * 2u <= 32768u;
}

// The streaming kernel multiplies on the CUDA cores: one or two rows keep up with HBM (5.1-5.4 TB/s on large weights), three and four do
// not (3.5), while the tensor cores pay about 3 us more per launch.  At four rows: 4096 x 4096 11.0 us here, 11.6 there; 12288 x
// 4096 29.2 and 23.2; 22016 x 4096 50.9 and 36.5.  The line lies at 20 million weights.  `tc`: the tensor cores take the product
// (less than 64 x 64 results or an unaligned result they do not).
static bool gemv_preferred(const rg_mat_mul_params *p, bool tc) {
    return gemv_shape(p) && (p->m <= 2 || !tc || static_cast<uint64_t>(p->n) * p->k < 20000000ull);
}

static int run_gemv(const rg_mat_mul_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    rg_linear_params lp = {};
    lp.dtype = p->dtype;
    lp.m = p->m, lp.n = p->n, lp.k = p->k;
    const void *lin[6] = {in[0], in[1], nullptr, nullptr, nullptr, nullptr};
    void *lout[3] = {out[0], nullptr, nullptr};
    return linear_stream(&lp, lin, lout, st);
}

// 5..32 rows of A against a K-major B: the weight-streaming kernel on the warp-level tensor path (RG_B200_SKINNY=0 keeps such
// products on the tcgen05 kernel)
static bool skinny_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("RG_B200_SKINNY");
        return !(e && e[0] == '0');
    }();
    return on;
}
static bool skinny_shape(const rg_mat_mul_params *p) {
    if (p->trans_a || !p->trans_b || p->batch != 1 || p->m <= 4 || p->m > 32) return false;
    if (p->has_bias && (p->bias_col_stride > 1)) return false;
    return linear_skinny_shape(p->dtype, p->m, p->n, p->k);
}
// The automatic choice: up to 8 rows of A against few rows of B with a long k.  Here / on tcgen05 at 8 rows: 1280 x 8192 weights 10.3 / 10.4
// us, 2560 x 8192 14.2 / 15.3, 512 x 8192 7.7 / 9.0; at 16 rows 11.3 / 10.6, 15.4 / 15.5 and 9.1 / 9.1; larger products are 15-40 % faster there.
// Up to 16 rows where tcgen05 does not take the product and the CUDA cores would be left with it.
static bool skinny_preferred(const rg_mat_mul_params *p, bool tc) {
    return skinny_enabled() && skinny_shape(p) && p->m <= (tc ? 8u : 16u) && p->n <= 2560 && p->k >= 4096;
}
static int run_skinny(const rg_mat_mul_params *p, void *ws, const void *const *in, void *const *out, cudaStream_t st) {
    SkinnyCall c = {};
    c.dtype = p->dtype, c.m = p->m, c.n = p->n, c.k = p->k;
    c.epilogue = p->has_bias ? 1 : 0;
    c.alpha = p->alpha, c.beta = p->beta;
    c.c_row_stride = p->bias_row_stride, c.c_col_stride = p->bias_col_stride, c.y_row_stride = p->n;
    c.w_static = (p->flags & RG_MM_B_STATIC) != 0;
    const void *lin[5] = {in[0], in[1], p->has_bias ? in[2] : nullptr, nullptr, nullptr};
    void *lout[3] = {out[0], nullptr, nullptr};
    return linear_skinny(c, ws, lin, lout, st);
}

// The 64 x 64 tiles of the CUDA-core kernel in fp32: a CTA alone takes 1.48 us for 16 values of k; with all SMs full a tile takes its SM 0.3 us
// and 0.83 per 16 values
static float f32_simt_us(const rg_mat_mul_params *p) {
    const float tiles = static_cast<float>((p->m + 63) / 64) * static_cast<float>((p->n + 63) / 64) * static_cast<float>(p->batch);
    const float steps = p->k > 16 ? static_cast<float>(p->k) / 16.f : 1.f, alone = 1.48f * steps, full = tiles / static_cast<float>(sm_count()) * (0.3f + 0.83f * steps);
    return 3.f + (alone > full ? alone : full);
}
// fp32 (force_kernel values): the form with the smallest estimated time.  Measured (tensor cores / 32 x 32 tiles / 64 x 64 tiles):
// 32 x 256 x 256 9.0 / 4.1 / 18.2 us, 128 x 1024 x 1024 19.7 / 19.0 / 97.8, 256 x 1024 x 1024 20.1 / 19.3 / -, 32 x 32000 x 1024 49 / 66 / 295,
// 4 x 11008 x 4096 75 / 103 / -, 509 x 2752 x 1024 39 / 91 / 128; the 64 x 64 tiles have the short k of large results, where the others pay
// for every tile: 4096 x 4096 x 4 - / 111 / 34, 1024 x 1024 x 8 - / 8.5 / 3.9, 300 matrices of 100 x 100 x 10 - / 31 / 11, 512 of 64 x 64 x 64
// - / 18.1 / 14.6.  Sums of fewer than eight products stay off the tensor cores, whose dropped terms would show beside so few roundings.
static int f32_route(const rg_mat_mul_params *p) {
    if (p->trans_a || !gemm_small32_supported(p)) return p->trans_a ? 1 : 5;
    const float tc = p->k < 8 ? 1e30f : gemm_tc32_us(p), small = gemm_small32_us(p);
    if ((p->m + 63) / 64 <= 65535 && f32_simt_us(p) < (tc < small ? tc : small)) return 1;
    return tc < small ? 5 : 6;
}

extern "C" {

size_t rg_b200_mat_mul_workspace(const rg_mat_mul_params *p) {
    // the fp32 tensor-core kernel's and the skinny kernel's k-split need scratch
    if (!p || p->m == 0 || p->n == 0 || p->k == 0 || p->batch == 0) return 0;
    if (p->dtype == RG_F32) return f32_route(p) == 5 || (p->force_kernel == 5 && !p->trans_a) ? gemm_tc32_workspace(p) : 0;
    if ((p->dtype != RG_FP16 && p->dtype != RG_BF16) || p->trans_a) return 0;
    return skinny_shape(p) ? linear_skinny_workspace(p->dtype, p->m, p->n, p->k, p->has_bias ? 1 : 0, nullptr, 0) : 0;
}

int rg_b200_mat_mul(const rg_mat_mul_params *p, void *ws, const void *const *in, void *const *out, void *stream) {
    if (!p || !in || !out || !in[0] || !in[1] || !out[0]) return RG_ERR_NULL;
    if (p->has_bias && !in[2]) return RG_ERR_NULL;
    if (p->dtype != RG_F32 && p->dtype != RG_FP16 && p->dtype != RG_BF16) return RG_ERR_DTYPE;
    if (p->k == 0) return RG_ERR_SHAPE;
    if (p->m == 0 || p->n == 0 || p->batch == 0) return RG_OK;
    if (p->batch > 65535) return RG_ERR_SHAPE;
    auto st = static_cast<cudaStream_t>(stream);
    switch (p->force_kernel) {
        case 0: break;
        case 1: return gemm_simt(p, in, out, st);
        case 2: return gemv_shape(p) ? run_gemv(p, in, out, st) : RG_ERR_UNSUPPORTED;
        case 3: return gemm_tc_supported(p, in, out) ? gemm_tc(p, in, out, st) : RG_ERR_UNSUPPORTED;
        case 4: return skinny_shape(p) ? run_skinny(p, ws, in, out, st) : RG_ERR_UNSUPPORTED;
        case 5: return gemm_tc32(p, ws, in, out, st);
        case 6: return gemm_small32(p, in, out, st);
        case 7: return gemm_tc_supported(p, in, out) ? gemm_tc(p, in, out, st, true) : RG_ERR_UNSUPPORTED;
        default: return RG_ERR_UNSUPPORTED;
    }
    if (p->dtype == RG_F32) {
        const int route = f32_route(p);
        return route == 5 ? gemm_tc32(p, ws, in, out, st) : route == 6 ? gemm_small32(p, in, out, st) : gemm_simt(p, in, out, st);
    }
    const bool tc = gemm_tc_supported(p, in, out);
    if (gemv_preferred(p, tc) && aligned16(in[0]) && aligned16(in[1])) {
        const int rc = run_gemv(p, in, out, st);
        if (rc != RG_ERR_SHAPE && rc != RG_ERR_UNSUPPORTED) return rc;
    }
    if (skinny_preferred(p, tc) && aligned16(in[0]) && aligned16(in[1]) && aligned16(out[0]) &&
        (ws || linear_skinny_workspace(p->dtype, p->m, p->n, p->k, p->has_bias ? 1 : 0, nullptr, 0) == 0)) {
        const int rc = run_skinny(p, ws, in, out, st);
        if (rc != RG_ERR_SHAPE && rc != RG_ERR_UNSUPPORTED) return rc;
    }
    return tc ? gemm_tc(p, in, out, st) : gemm_simt(p, in, out, st);
}
}
