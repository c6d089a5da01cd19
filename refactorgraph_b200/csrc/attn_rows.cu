// Attention on the reference tensor layout (rg_b200_attention; semantics src/08-01llm/README.md:29-63) for everything the
// tensor-core prefill kernel does not take: single-token steps, short prompts, fp32, head dimensions 32 / 64 / 128 / 256.
// Probabilities and sums stay in fp32.
//
// The query rows that share a KV head — the heads of its group times the S positions — are contiguous in q and o, so a CTA takes R of
// them at a time and a split of the keys they see (R = 4 or 2 where there are that many rows: every K / V element loaded then serves
// R rows).  Work inside a CTA: LPK lanes share a key (16-byte chunks dealt round robin, so the lanes of a key read whole
// sectors), a warp holds 32 / LPK keys times U at once with all their K and V loads in flight, and every group of lanes keeps its
// own online-softmax state, merged once at the end: no cross-lane step per key other than the dot product's.  Splits exist
// because a step has only batch x heads rows: their number comes from the capacity, the keys of each from the device-side past,
// so a short sequence in a large cache is cut as finely as a long one.  The last split to arrive merges the records.
// Bound by HBM in a step (K and V of a group read once).  A generation step of 4 sequences x 1037 tokens, two layers of the 7B shape in
// fp16: 2.73 ms with one warp walking all keys of a row, 0.53 ms with this kernel.
#include "common.cuh"

namespace rg {

constexpr int AR_THREADS = 128, AR_WARPS = 4, AR_MAX_SPLITS = 32, AR_MIN_KEYS = 64;

struct RowsArgs {
    const void *q, *k, *v;
    void *o;
    const int64_t *past;
    float *part;   // [n][kv head][row block][split][R][2 + D]
    unsigned *cnt; // [n][kv head][row block], zero before the first call and left at zero
    uint32_t S, rows, row_blocks, splits, kv_tokens;// rows = query rows of one KV head, kv_tokens = tokens addressable per (n, KV head)
    float scale;
};

template<class T, int D> struct RowsShape {
    static constexpr int CHUNKS = D * static_cast<int>(sizeof(T)) / 16, E = 16 / static_cast<int>(sizeof(T));
    static constexpr int LPK = CHUNKS < 8 ? CHUNKS : 8, CPL = CHUNKS / LPK, KPW = 32 / LPK;
    static constexpr int U = CPL >= 4 ? 2 : 4;          // keys per lane group in flight: at most 16 loads of 16 bytes per lane
    static constexpr int VPL = CPL * E;                 // elements of a row held by a lane
    static constexpr int RMAX = VPL <= 16 ? 4 : 1;      // register file: (2 R + 2 U) VPL values
    static constexpr int KEYS = KPW * U;                // keys of one warp step
};

template<class T, bool ALIGNED>
__device__ __forceinline__ void rows_load(Vec16<T> &v, const T *p) {
    if constexpr (ALIGNED) {
        v.load(p);
    } else {
#pragma unroll
        for (int e = 0; e < Vec16<T>::N; ++e) reinterpret_cast<T *>(&v.raw)[e] = p[e];
    }
}

// ALIGNED = false: k and v start off a 16-byte boundary and are read element by element
template<class T, int D, int R, bool ALIGNED>
__global__ void __launch_bounds__(AR_THREADS) attn_rows_kernel(const RowsArgs a) {
    using Sh = RowsShape<T, D>;
    constexpr int LPK = Sh::LPK, CPL = Sh::CPL, KPW = Sh::KPW, U = Sh::U, E = Sh::E, VPL = Sh::VPL;
    __shared__ float s_acc[AR_WARPS][R][D];
    __shared__ float s_m[AR_WARPS][R], s_l[AR_WARPS][R];
    __shared__ int s_last;
    pdl_enter();
    const uint32_t split = blockIdx.x % a.splits, block = blockIdx.x / a.splits;
    const uint32_t rb = block % a.row_blocks, head = block / a.row_blocks;// head = n * KV heads + KV head
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / LPK, sub = lane % LPK;
    const uint32_t past = past_clamped(a.past, a.kv_tokens);
    const uint32_t r0 = rb * R;
    // keys that the rows of this block see: a row at position i sees keys 0 .. past + i
    uint32_t see[R], vis = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint64_t s = r0 + r < a.rows ? static_cast<uint64_t>(past) + (r0 + r) % a.S + 1u : 0u;
        see[r] = s < a.kv_tokens ? static_cast<uint32_t>(s) : a.kv_tokens;
        vis = see[r] > vis ? see[r] : vis;
    }
    uint32_t per = (vis + a.splits - 1) / a.splits;
    per = per < AR_MIN_KEYS ? AR_MIN_KEYS : (per + AR_WARPS * Sh::KEYS - 1) / (AR_WARPS * Sh::KEYS) * (AR_WARPS * Sh::KEYS);
    const uint32_t nsplit = vis ? (vis + per - 1) / per : 1;
    if (split >= nsplit) return;
    const uint32_t k0 = split * per, k1 = k0 + per < vis ? k0 + per : vis;

    const size_t qrow = static_cast<size_t>(head) * a.rows + r0;
    const T *q = static_cast<const T *>(a.q) + qrow * D;
    const T *K = static_cast<const T *>(a.k) + static_cast<size_t>(head) * a.kv_tokens * D;
    const T *V = static_cast<const T *>(a.v) + static_cast<size_t>(head) * a.kv_tokens * D;
    float qv[R][VPL], acc[R][VPL], m[R], l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                qv[r][c * E + e] = r0 + r < a.rows ? Num<T>::to_f(q[static_cast<size_t>(r) * D + (c * LPK + sub) * E + e]) * a.scale : 0.f;
                acc[r][c * E + e] = 0.f;
            }
        }
    }
    for (uint32_t kb = k0 + warp * Sh::KEYS; kb < k1; kb += AR_WARPS * Sh::KEYS) {
        Vec16<T> kr[U][CPL], vr[U][CPL];
        uint32_t key[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            key[u] = kb + u * KPW + grp;
            const size_t at = static_cast<size_t>(key[u] < k1 ? key[u] : k0) * D;// a key past the end loads a valid row and is masked
#pragma unroll
            for (int c = 0; c < CPL; ++c) rows_load<T, ALIGNED>(kr[u][c], K + at + (c * LPK + sub) * E);
#pragma unroll
            for (int c = 0; c < CPL; ++c) rows_load<T, ALIGNED>(vr[u][c], V + at + (c * LPK + sub) * E);
        }
        float s[R][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int r = 0; r < R; ++r) s[r][u] = 0.f;
#pragma unroll
            for (int c = 0; c < CPL; ++c) {
                float f[E];
                kr[u][c].unpack(f);
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int e = 0; e < E; ++e) s[r][u] = fmaf(qv[r][c * E + e], f[e], s[r][u]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int x = 1; x < LPK; x <<= 1) s[r][u] += __shfl_xor_sync(0xffffffffu, s[r][u], x);
        }
        float p[R][U];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float mn = m[r];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (key[u] < k1 && key[u] < see[r]) mn = fmaxf(mn, s[r][u]);
            const float corr = m[r] == -INFINITY ? 0.f : expf(m[r] - mn), base = mn == -INFINITY ? 0.f : mn;// only scores of -inf so far: weights of 0, not exp(inf - inf)
            l[r] *= corr;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                p[r][u] = key[u] < k1 && key[u] < see[r] ? expf(s[r][u] - base) : 0.f;
                l[r] += p[r][u];
            }
            m[r] = mn;
#pragma unroll
            for (int e = 0; e < VPL; ++e) acc[r][e] *= corr;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (key[u] >= k1) continue;// its row repeats another's: 0 x inf must not reach the sum
#pragma unroll
            for (int c = 0; c < CPL; ++c) {
                float f[E];
                vr[u][c].unpack(f);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (key[u] >= see[r]) continue;
#pragma unroll
                    for (int e = 0; e < E; ++e) acc[r][c * E + e] = fmaf(p[r][u], f[e], acc[r][c * E + e]);
                }
            }
        }
    }
    // merge the lane groups of the warp, then the warps
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float mw = m[r];
#pragma unroll
        for (int x = LPK; x < 32; x <<= 1) mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, x));
        const float f = m[r] == -INFINITY ? 0.f : expf(m[r] - mw);
        float lw = l[r] * f;
#pragma unroll
        for (int x = LPK; x < 32; x <<= 1) lw += __shfl_xor_sync(0xffffffffu, lw, x);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                float v = acc[r][c * E + e] * f;
#pragma unroll
                for (int x = LPK; x < 32; x <<= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
                if (grp == 0) s_acc[warp][r][(c * LPK + sub) * E + e] = v;
            }
        }
        if (lane == 0) s_m[warp][r] = mw, s_l[warp][r] = lw;
    }
    __syncthreads();
    T *o = static_cast<T *>(a.o) + qrow * D;
    float *rec = a.part + static_cast<size_t>(block) * a.splits * (R * (D + 2));
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float mx = -INFINITY, den = 0.f, f[AR_WARPS];
#pragma unroll
        for (int w = 0; w < AR_WARPS; ++w) mx = fmaxf(mx, s_m[w][r]);
#pragma unroll
        for (int w = 0; w < AR_WARPS; ++w) {
            f[w] = s_m[w][r] == -INFINITY ? 0.f : expf(s_m[w][r] - mx);
            den += s_l[w][r] * f[w];
        }
        for (uint32_t d = threadIdx.x; d < D; d += AR_THREADS) {
            float num = 0.f;
#pragma unroll
            for (int w = 0; w < AR_WARPS; ++w) num += s_acc[w][r][d] * f[w];
            if (nsplit > 1) rec[(split * R + r) * (D + 2) + 2 + d] = num;
            else if (r0 + r < a.rows)
                o[static_cast<size_t>(r) * D + d] = Num<T>::from_f(num / den);
        }
        if (nsplit > 1 && threadIdx.x == 0) rec[(split * R + r) * (D + 2)] = mx, rec[(split * R + r) * (D + 2) + 1] = den;
    }
    if (nsplit == 1) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.cnt + block, 1u) == nsplit - 1 ? 1 : 0;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
        if (r0 + r >= a.rows) break;
        // a lane reads the record header of one split (there are at most 32)
        float2 ml = make_float2(-INFINITY, 0.f);
        if (lane < nsplit) ml.x = __ldcg(rec + (lane * R + r) * (D + 2)), ml.y = __ldcg(rec + (lane * R + r) * (D + 2) + 1);
        const float mx = warp_max(ml.x);
        const float f = ml.x == -INFINITY ? 0.f : expf(ml.x - mx);
        const float den = warp_sum(ml.y * f);
        for (uint32_t d0 = 0; d0 < D; d0 += AR_THREADS) {
            const uint32_t d = d0 + threadIdx.x;
            float num = 0.f;
#pragma unroll 8
            for (uint32_t j = 0; j < nsplit; ++j) {
                const float w = __shfl_sync(0xffffffffu, f, j);
                if (d < D) num += __ldcg(rec + (j * R + r) * (D + 2) + 2 + d) * w;
            }
            if (d < D) o[static_cast<size_t>(r) * D + d] = Num<T>::from_f(num / den);
        }
    }
    if (threadIdx.x == 0) a.cnt[block] = 0u;
}

struct RowsPlan {
    uint32_t R, rows, row_blocks, splits;
    size_t cnt_bytes, part_bytes;
};
static uint32_t rows_rmax(int dtype, uint32_t D) {
    if (dtype == RG_F32) return D == 32 ? RowsShape<float, 32>::RMAX : D == 64 ? RowsShape<float, 64>::RMAX : D == 128 ? RowsShape<float, 128>::RMAX : RowsShape<float, 256>::RMAX;
    return D == 32 ? RowsShape<__half, 32>::RMAX : D == 64 ? RowsShape<__half, 64>::RMAX : D == 128 ? RowsShape<__half, 128>::RMAX : RowsShape<__half, 256>::RMAX;
}
static RowsPlan rows_plan(const rg_attention_params *p, bool aligned = true) {
    RowsPlan pl;
    pl.rows = p->n_heads / p->n_kv_heads * p->seq_len;
    const uint32_t rmax = aligned ? rows_rmax(p->dtype, p->head_dim) : 1;
    pl.R = pl.rows >= 4 && rmax >= 4 ? 4 : (pl.rows >= 2 && rmax >= 2 ? 2 : 1);
    pl.row_blocks = (pl.rows + pl.R - 1) / pl.R;
    const uint64_t ctas = static_cast<uint64_t>(pl.row_blocks) * p->n_kv_heads * p->batch;
    const uint32_t kv_tokens = p->has_cache ? p->max_seq : p->seq_len;
    // four CTAs per SM: 16 warps with 8 KiB of loads each in flight
    uint64_t want = ctas ? 4ull * sm_count() / ctas : 1;
    const uint32_t most = (kv_tokens + AR_MIN_KEYS - 1) / AR_MIN_KEYS;
    if (want > most) want = most;
    pl.splits = static_cast<uint32_t>(want < 1 ? 1 : want > AR_MAX_SPLITS ? AR_MAX_SPLITS : want);
    pl.cnt_bytes = pl.splits > 1 ? (ctas * 4 + 255) / 256 * 256 : 0;
    pl.part_bytes = pl.splits > 1 ? ctas * pl.splits * pl.R * (p->head_dim + 2) * 4 : 0;
    return pl;
}
// The alignment of K and V may change from call to call and with it the number of row blocks: the counters have a place of their own
// that holds those of either plan, so that no call parks sums where another one counts.
struct RowsWorkspace {
    size_t cnt_bytes, part_bytes;
};
static RowsWorkspace rows_workspace(const rg_attention_params *p) {
    const RowsPlan pl = rows_plan(p), pu = rows_plan(p, false);
    return {pl.cnt_bytes > pu.cnt_bytes ? pl.cnt_bytes : pu.cnt_bytes, pl.part_bytes > pu.part_bytes ? pl.part_bytes : pu.part_bytes};
}
size_t attn_rows_workspace(const rg_attention_params *p) {
    const RowsWorkspace w = rows_workspace(p);
    return w.cnt_bytes + w.part_bytes;
}

template<class T, int D>
static int rows_launch(const RowsPlan &pl, const RowsArgs &a, dim3 grid, cudaStream_t st) {
    void (*kern)(const RowsArgs) = attn_rows_kernel<T, D, 1, true>;
    if (!aligned16(a.k) || !aligned16(a.v)) {
        kern = attn_rows_kernel<T, D, 1, false>;
    } else if constexpr (RowsShape<T, D>::RMAX >= 4) {
        if (pl.R == 4) kern = attn_rows_kernel<T, D, 4, true>;
        else if (pl.R == 2)
            kern = attn_rows_kernel<T, D, 2, true>;
    }
    RG_CHECK_CUDA(launch_pdl(kern, grid, dim3(AR_THREADS), 0, st, a));
    count_launch();
    return launch_status();
}
template<class T>
static int rows_dim(uint32_t D, const RowsPlan &pl, const RowsArgs &a, dim3 grid, cudaStream_t st) {
    switch (D) {
        case 32: return rows_launch<T, 32>(pl, a, grid, st);
        case 64: return rows_launch<T, 64>(pl, a, grid, st);
        case 128: return rows_launch<T, 128>(pl, a, grid, st);
        case 256: return rows_launch<T, 256>(pl, a, grid, st);
        default: return RG_ERR_SHAPE;
    }
}
// ws may be NULL: the keys are then not split
int attn_rows(const rg_attention_params *p, void *ws, const void *q, const void *k, const void *v, void *o, const int64_t *past, uint32_t kv_tokens, cudaStream_t st) {
    RowsPlan pl = rows_plan(p, aligned16(k) && aligned16(v));
    if (!ws) pl.splits = 1;
    RowsArgs a = {};
    a.q = q, a.k = k, a.v = v, a.o = o, a.past = past;
    a.cnt = static_cast<unsigned *>(ws), a.part = reinterpret_cast<float *>(static_cast<uint8_t *>(ws) + rows_workspace(p).cnt_bytes);
    a.S = p->seq_len, a.rows = pl.rows, a.row_blocks = pl.row_blocks, a.splits = pl.splits, a.kv_tokens = kv_tokens;
    a.scale = 1.0f / sqrtf(static_cast<float>(p->head_dim));
    const uint64_t ctas = static_cast<uint64_t>(pl.row_blocks) * pl.splits * p->n_kv_heads * p->batch;
    if (ctas > 0x7fffffffull) return RG_ERR_SHAPE;
    const dim3 grid(static_cast<unsigned>(ctas));
    switch (p->dtype) {
        case RG_F32: return rows_dim<float>(p->head_dim, pl, a, grid, st);
        case RG_FP16: return rows_dim<__half>(p->head_dim, pl, a, grid, st);
        default: return rows_dim<__nv_bfloat16>(p->head_dim, pl, a, grid, st);
    }
}

}// namespace rg
