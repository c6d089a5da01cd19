// TopK and top-k sampling over vocabulary-sized rows (no reference counterpart; the ordering rule is
// "value descending, ties by lower index, NaN below every number").
//
// One CTA per row.  The row is turned into order-preserving 32-bit keys staged in shared memory (one HBM read),
// the k-th largest key is found by an MSB-first radix select (4 passes of 8 bits with shared-memory
// histograms); if the k-th key is tied, four more passes over ~index pick the lowest indices, so the
// selection is a radix select over the distinct 64-bit composite (key, ~index) and is deterministic.
// The k winners are then rank-sorted and written out.
//
// In front of it, for rows of up to 16 16-byte chunks per thread: the row stays in registers (one read), every thread finds the
// largest key of its own elements, and the k-th largest of those maxima is a key that at least k elements reach.  The elements that
// reach it — k of them and a few more, unless values repeat a lot — are ranked against one another.  In a row with more than 512
// of them, bisection finds the k-th largest key, and a pass in the order of the indices its first ties.
// The histogram passes of the radix select serialise on the few distinct leading bytes that logits have:
// one row of 32000 fp16 values 40 us, 509 rows of fp32 120 us, and a 4-token step of a two-layer decoder 527 -> 502 us without them.
#include "common.cuh"

namespace rg {

constexpr int TOPK_MAX = 64;
constexpr int TOPK_THREADS = 1024;
constexpr int TOPK_REG_THREADS = 512;// rows in registers: up to 64 of them hold the row
constexpr uint32_t TOPK_STAGE_MAX = 40960;// keys staged in smem (160 KiB)

template<class T> __device__ __forceinline__ uint32_t key_of(T v) {
    const float f = Num<T>::to_f(v);
    if (f != f) return 0u;
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float float_of_key(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct TopkShared {
    uint32_t hist[256];
    uint32_t bin, kk, cnt_eq, count;
    uint32_t cand_key[TOPK_MAX];
    uint32_t cand_idx[TOPK_MAX];
    uint32_t sort_key[TOPK_MAX];
    uint32_t sort_idx[TOPK_MAX];
    float red[33];
};

// Selects the k largest (key, ~idx) composites of the row into sh.sort_key/sort_idx (descending).
// `skeys` holds the staged keys when staged != 0, else keys are recomputed from x.
template<class T>
__device__ void topk_select(const T *__restrict__ xr, uint32_t n, uint32_t k, uint32_t *skeys, bool staged,
                            TopkShared &sh) {
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    if (staged)
        for (uint32_t i = tid; i < n; i += nt) skeys[i] = key_of<T>(xr[i]);
    __syncthreads();
    auto key_at = [&](uint32_t i) -> uint32_t { return staged ? skeys[i] : key_of<T>(xr[i]); };

    uint32_t prefix = 0, mask = 0, prefix2 = 0, mask2 = 0, kk = k;
    bool tie_break = false;
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = 24 - 8 * (pass & 3);
        for (uint32_t b = tid; b < 256; b += nt) sh.hist[b] = 0;
        __syncthreads();
        if (pass < 4) {
            for (uint32_t i = tid; i < n; i += nt) {
                const uint32_t key = key_at(i);
                if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & 255u], 1u);
            }
        } else {
            for (uint32_t i = tid; i < n; i += nt) {
                const uint32_t key = key_at(i), inv = ~i;
                if (key == prefix && (inv & mask2) == prefix2) atomicAdd(&sh.hist[(inv >> shift) & 255u], 1u);
            }
        }
        __syncthreads();
        if (tid < 32) {
            // lane L owns bins 255-8L .. 248-8L (descending); find the bin holding the kk-th largest
            uint32_t local = 0;
            const int top = 255 - 8 * static_cast<int>(tid);
#pragma unroll
            for (int j = 0; j < 8; ++j) local += sh.hist[top - j];
            uint32_t incl = local;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (static_cast<int>(tid) >= o) incl += t;
            }
            const uint32_t excl = incl - local;
            if (excl < kk && kk <= incl) {
                uint32_t above = excl;
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = sh.hist[top - j];
                    if (above + c >= kk) {
                        sh.bin = static_cast<uint32_t>(top - j);
                        sh.kk = kk - above;
                        sh.cnt_eq = c;
                        break;
                    }
                    above += c;
                }
            }
        }
        __syncthreads();
        kk = sh.kk;
        if (pass < 4) {
            prefix |= sh.bin << shift;
            mask |= 255u << shift;
            if (pass == 3) {
                if (sh.cnt_eq == kk) break;// every element equal to the k-th key is taken
                tie_break = true;
            }
        } else {
            prefix2 |= sh.bin << shift;
            mask2 |= 255u << shift;
        }
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0) sh.count = 0;
    __syncthreads();
    for (uint32_t i = tid; i < n; i += nt) {
        const uint32_t key = key_at(i);
        const bool take = key > prefix || (key == prefix && (!tie_break || (~i) >= prefix2));
        if (take) {
            const uint32_t pos = atomicAdd(&sh.count, 1u);
            if (pos < TOPK_MAX) {
                sh.cand_key[pos] = key;
                sh.cand_idx[pos] = i;
            }
        }
    }
    __syncthreads();
    const uint32_t cnt = sh.count < k ? sh.count : k;
    if (tid < cnt) {
        const uint32_t mk = sh.cand_key[tid], mi = sh.cand_idx[tid];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < cnt; ++j) {
            const uint32_t ok = sh.cand_key[j], oi = sh.cand_idx[j];
            rank += (ok > mk || (ok == mk && oi < mi)) ? 1u : 0u;
        }
        sh.sort_key[rank] = mk;
        sh.sort_idx[rank] = mi;
    }
    __syncthreads();
}

// The row in registers: CH 16-byte chunks per thread, chunk threadIdx.x + c * blockDim.x.
template<class T, int CH> struct TopkRow {
    static constexpr int N = Vec16<T>::N;
    Vec16<T> raw[CH];
    uint32_t chunks;
    __device__ __forceinline__ void load(const T *xr, uint32_t n) {
        chunks = n / N;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const uint32_t i = threadIdx.x + c * blockDim.x;
            if (i < chunks) raw[c].load(xr + static_cast<size_t>(i) * N);
        }
    }
    template<class F> __device__ __forceinline__ void each(F &&f) const {
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const uint32_t i = threadIdx.x + c * blockDim.x;
            if (i < chunks) {
                float v[N];
                raw[c].unpack(v);
#pragma unroll
                for (int j = 0; j < N; ++j) f(v[j], i * N + j);
            }
        }
    }
};
constexpr uint32_t TOPK_CAND = 512;
struct TopkCand {
    uint32_t key[TOPK_CAND], idx[TOPK_CAND], count, top[32];
};
// The sum of v over the block, for every thread; buf alternates between calls
__device__ __forceinline__ uint32_t topk_block_count(uint32_t v, TopkCand &cd, uint32_t buf) {
    const uint32_t lane = threadIdx.x & 31u, warps = blockDim.x >> 5;// at most 16
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) cd.top[buf * 16 + (threadIdx.x >> 5)] = v;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < warps ? cd.top[buf * 16 + lane] : 0u);
}
// The k winners to cd, of a row in which many keys reach `least`; `mine` is the largest key of the calling thread's elements.  A function of
// its own that reads the row again (from L1 or L2), so that the common case has the registers to itself.  The k-th largest key by
// bisection between `least` and the largest key (which are the same where those values repeat), then a pass in the order of the
// indices that ends when enough ties are found.  A row of 32000 equal halves 47 us on the radix select.
template<class T> static __device__ __noinline__ void topk_many_ties(const T *__restrict__ xr, uint32_t n, uint32_t k, uint32_t least, uint32_t mine, TopkCand &cd) {
    constexpr uint32_t N = Vec16<T>::N;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, chunks = n / N;
    mine = __reduce_max_sync(0xffffffffu, mine);
    if (lane == 0) cd.top[16 + warp] = mine;
    __syncthreads();// every thread has seen cd.count by now
    if (threadIdx.x == 0) cd.count = 0;
    // at least k keys reach lo, `above` (less than k) reach hi
    uint32_t lo = least, hi = __reduce_max_sync(0xffffffffu, lane < warps ? cd.top[16 + lane] : 0u) + 1, above = 0, buf = 0;
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        uint32_t c = 0;
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < chunks; i += blockDim.x) {
            Vec16<T> a;
            float v[N];
            a.load(xr + static_cast<size_t>(i) * N);
            a.unpack(v);
#pragma unroll
            for (uint32_t j = 0; j < N; ++j) c += key_of<float>(v[j]) >= mid ? 1u : 0u;
        }
        c = topk_block_count(c, cd, buf);
        buf ^= 1u;
        if (c >= k) lo = mid;
        else
            hi = mid, above = c;
    }
    const uint32_t need = k - above;// ties, the first of them
    uint32_t seen = 0;              // ties in the chunks before i0
    for (uint32_t i0 = 0; i0 < chunks && (above || seen < need); i0 += blockDim.x, buf ^= 1u) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t key[N], ties = 0;
        if (i < chunks) {
            Vec16<T> a;
            float v[N];
            a.load(xr + static_cast<size_t>(i) * N);
            a.unpack(v);
#pragma unroll
            for (uint32_t j = 0; j < N; ++j) key[j] = key_of<float>(v[j]), ties += key[j] == lo ? 1u : 0u;
        }
        uint32_t upto = ties;// of this warp's lanes so far
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, upto, d);
            upto += lane >= d ? o : 0u;
        }
        if (lane == 31) cd.top[buf * 16 + warp] = upto;
        __syncthreads();
        const uint32_t w = lane < warps ? cd.top[buf * 16 + lane] : 0u;
        uint32_t rank = seen + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + upto - ties;
        seen += __reduce_add_sync(0xffffffffu, w);
        if (i < chunks) {
#pragma unroll
            for (uint32_t j = 0; j < N; ++j) {
                if (key[j] > lo || (key[j] == lo && rank++ < need)) {
                    const uint32_t at = atomicAdd(&cd.count, 1u);// k of them in all
                    cd.key[at] = key[j], cd.idx[at] = i * N + j;
                }
            }
        }
    }
    __syncthreads();
}
// The k winners of the row to sh.sort_key / sort_idx
template<class T, int CH>
__device__ __forceinline__ void topk_from_registers(const TopkRow<T, CH> &row, const T *__restrict__ xr, uint32_t n, uint32_t k, TopkShared &sh, TopkCand &cd) {
    const uint32_t tid = threadIdx.x;
    uint32_t mine = 0u;
    row.each([&](float v, uint32_t) {
        const uint32_t key = key_of<float>(v);
        mine = key > mine ? key : mine;
    });
    if (tid == 0) cd.count = 0;
    uint32_t least = 0u;
    if (k == 1) {
        const uint32_t w = __reduce_max_sync(0xffffffffu, mine);
        if (tid < 32) cd.top[tid] = 0u;
        __syncthreads();
        if ((tid & 31u) == 0) cd.top[tid >> 5] = w;
        __syncthreads();
        least = __reduce_max_sync(0xffffffffu, cd.top[tid & 31u]);
    } else {
        // the leading 20 bits of the k-th largest maximum (sign, exponent and 11 bits below: ties beyond that add candidates)
        for (int bit = 31; bit >= 12; --bit) {
            const uint32_t t = least | (1u << bit);
            if (static_cast<uint32_t>(__syncthreads_count(mine >= t)) >= k) least = t;
        }
    }
    if (mine >= least) {
        row.each([&](float v, uint32_t i) {
            const uint32_t key = key_of<float>(v);
            if (key >= least) {
                const uint32_t at = atomicAdd(&cd.count, 1u);
                if (at < TOPK_CAND) cd.key[at] = key, cd.idx[at] = i;
            }
        });
    }
    __syncthreads();
    uint32_t count = cd.count;
    if (count > TOPK_CAND) {
        topk_many_ties<T>(xr, n, k, least, mine, cd);
        count = cd.count;// k
    }
    for (uint32_t c = tid; c < count; c += blockDim.x) {
        const uint32_t mk = cd.key[c], mi = cd.idx[c];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < count; ++j) rank += (cd.key[j] > mk || (cd.key[j] == mk && cd.idx[j] < mi)) ? 1u : 0u;
        if (rank < k) sh.sort_key[rank] = mk, sh.sort_idx[rank] = mi;
    }
    __syncthreads();
}

// CH != 0: rows of CH chunks per thread, in registers
template<class T, bool SOFTMAX, int CH>
__global__ void __launch_bounds__(CH ? TOPK_REG_THREADS : TOPK_THREADS) topk_kernel(const T *__restrict__ x, void *__restrict__ values,
                                                            int64_t *__restrict__ indices, uint32_t n, uint32_t k,
                                                            int staged) {
    pdl_enter();
    extern __shared__ __align__(16) uint32_t skeys[];
    __shared__ TopkShared sh;
    __shared__ TopkCand cd;
    const T *xr = x + static_cast<size_t>(blockIdx.x) * n;
    TopkRow<T, CH ? CH : 1> row;
    if constexpr (CH != 0) {
        row.load(xr, n);
        topk_from_registers(row, xr, n, k, sh, cd);
    } else {
        topk_select<T>(xr, n, k, skeys, staged != 0, sh);
    }
    float inv_sum = 0.f, mx = 0.f;
    if constexpr (SOFTMAX) {
        mx = float_of_key(sh.sort_key[0]);
        float s = 0.f;
        if constexpr (CH != 0) {
            row.each([&](float f, uint32_t) {
                if (f == f) s += expf(f - mx);
            });
        } else {
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
                const float f = staged ? float_of_key(skeys[i]) : Num<T>::to_f(xr[i]);
                if (f == f) s += expf(f - mx);
            }
        }
        s = block_sum(s, sh.red);
        inv_sum = 1.f / s;
    }
    if (threadIdx.x < k) {
        const uint32_t idx = sh.sort_idx[threadIdx.x];
        const size_t o = static_cast<size_t>(blockIdx.x) * k + threadIdx.x;
        indices[o] = static_cast<int64_t>(idx);
        if constexpr (SOFTMAX) static_cast<float *>(values)[o] = expf(Num<T>::to_f(xr[idx]) - mx) * inv_sum;
        else
            static_cast<T *>(values)[o] = xr[idx];
    }
}

// Philox-4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC'11).
__device__ __forceinline__ uint32_t philox_u32(uint64_t seed, uint32_t row, uint64_t step) {
    uint32_t c0 = row, c1 = 0u, c2 = static_cast<uint32_t>(step), c3 = static_cast<uint32_t>(step >> 32);
    uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
        c0 = n0, c1 = n1, c2 = n2, c3 = n3;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c0;
}

template<class T, int CH>
__global__ void __launch_bounds__(CH ? TOPK_REG_THREADS : TOPK_THREADS) topk_sample_kernel(const T *__restrict__ x,
                                                                   const uint64_t *__restrict__ step,
                                                                   int64_t *__restrict__ token, uint32_t n, uint32_t k,
                                                                   float inv_temp, uint64_t seed, int staged) {
    pdl_enter();
    extern __shared__ __align__(16) uint32_t skeys[];
    __shared__ TopkShared sh;
    __shared__ TopkCand cd;
    const T *xr = x + static_cast<size_t>(blockIdx.x) * n;
    if constexpr (CH != 0) {
        TopkRow<T, CH> row;
        row.load(xr, n);
        topk_from_registers(row, xr, n, k, sh, cd);
    } else {
        topk_select<T>(xr, n, k, skeys, staged != 0, sh);
    }
    if (threadIdx.x == 0) {
        const float x0 = float_of_key(sh.sort_key[0]);
        float total = 0.f;
        for (uint32_t j = 0; j < k; ++j) total += expf((float_of_key(sh.sort_key[j]) - x0) * inv_temp);
        const uint32_t r = philox_u32(seed, blockIdx.x, *step);
        const float u = static_cast<float>(r >> 8) * (1.0f / 16777216.0f);
        const float target = u * total;
        float cum = 0.f;
        uint32_t pick = k - 1;
        for (uint32_t j = 0; j < k; ++j) {
            cum += expf((float_of_key(sh.sort_key[j]) - x0) * inv_temp);
            if (cum > target) {
                pick = j;
                break;
            }
        }
        token[blockIdx.x] = static_cast<int64_t>(sh.sort_idx[pick]);
    }
}

static uint32_t topk_threads(uint32_t n) {
    uint32_t t = (n + 31) / 32 * 32;
    if (t > TOPK_THREADS) t = TOPK_THREADS;
    if (t < 64) t = 64;
    return t;
}
// Chunks per thread of the form that keeps the row in registers, or 0: whole aligned 16-byte chunks, at most 16 a thread
template<class T> static int topk_chunks(const void *x, uint32_t n) {
    constexpr uint32_t N = 16 / sizeof(T);
    if (!aligned16(x) || n % N != 0 || n < 1024) return 0;
    const uint32_t per = (n / N + TOPK_REG_THREADS - 1) / TOPK_REG_THREADS;
    return per <= 4 ? 4 : per <= 8 ? 8 : per <= 16 ? 16 : 0;
}
struct TopkLaunch {
    int staged;
    size_t smem;
    uint32_t threads;
};
// Keys are staged for the radix select
static TopkLaunch topk_shape(uint32_t n, int ch) {
    TopkLaunch l;
    l.staged = n <= TOPK_STAGE_MAX && !ch;
    l.smem = l.staged ? static_cast<size_t>(n) * 4 : 0;
    l.threads = ch ? static_cast<uint32_t>(TOPK_REG_THREADS) : topk_threads(n);
    return l;
}

template<class T, bool SOFTMAX, int CH>
static int topk_go(const rg_topk_params *p, const T *x, void *values, int64_t *idx, cudaStream_t st) {
    const TopkLaunch l = topk_shape(p->n, CH);
    RG_CHECK_CUDA(cudaFuncSetAttribute(topk_kernel<T, SOFTMAX, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 163840));
    RG_CHECK_CUDA(launch_pdl(topk_kernel<T, SOFTMAX, CH>, dim3(p->rows), dim3(l.threads), l.smem, st, x, values, idx, p->n, p->k, l.staged));
    count_launch();
    return launch_status();
}
template<class T>
static int topk_launch(const rg_topk_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    auto x = static_cast<const T *>(in[0]);
    auto idx = static_cast<int64_t *>(out[1]);
#define RG_TOPK(CH) (p->softmax ? topk_go<T, true, CH>(p, x, out[0], idx, st) : topk_go<T, false, CH>(p, x, out[0], idx, st))
    switch (topk_chunks<T>(x, p->n)) {
        case 4: return RG_TOPK(4);
        case 8: return RG_TOPK(8);
        case 16: return RG_TOPK(16);
        default: return RG_TOPK(0);
    }
#undef RG_TOPK
}

template<class T, int CH>
static int topk_sample_go(const rg_topk_sample_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    const TopkLaunch l = topk_shape(p->n, CH);
    RG_CHECK_CUDA(cudaFuncSetAttribute(topk_sample_kernel<T, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 163840));
    RG_CHECK_CUDA(launch_pdl(topk_sample_kernel<T, CH>, dim3(p->rows), dim3(l.threads), l.smem, st, static_cast<const T *>(in[0]), static_cast<const uint64_t *>(in[1]),
                             static_cast<int64_t *>(out[0]), p->n, p->k, 1.0f / p->temperature, p->seed, l.staged));
    count_launch();
    return launch_status();
}
template<class T>
static int topk_sample_launch(const rg_topk_sample_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    switch (topk_chunks<T>(in[0], p->n)) {
        case 4: return topk_sample_go<T, 4>(p, in, out, st);
        case 8: return topk_sample_go<T, 8>(p, in, out, st);
        case 16: return topk_sample_go<T, 16>(p, in, out, st);
        default: return topk_sample_go<T, 0>(p, in, out, st);
    }
}

}// namespace rg

using namespace rg;

extern "C" {

size_t rg_b200_topk_workspace(const rg_topk_params *) { return 0; }
int rg_b200_topk(const rg_topk_params *p, void *, const void *const *in, void *const *out, void *stream) {
    if (!p || !in || !out || !in[0] || !out[0] || !out[1]) return RG_ERR_NULL;
    if (p->k == 0 || p->k > TOPK_MAX || p->k > p->n) return RG_ERR_SHAPE;
    if (p->rows == 0) return RG_OK;
    auto st = static_cast<cudaStream_t>(stream);
    switch (p->dtype) {
        case RG_F32: return topk_launch<float>(p, in, out, st);
        case RG_FP16: return topk_launch<__half>(p, in, out, st);
        case RG_BF16: return topk_launch<__nv_bfloat16>(p, in, out, st);
        default: return RG_ERR_DTYPE;
    }
}

size_t rg_b200_topk_sample_workspace(const rg_topk_sample_params *) { return 0; }
int rg_b200_topk_sample(const rg_topk_sample_params *p, void *, const void *const *in, void *const *out, void *stream) {
    if (!p || !in || !out || !in[0] || !in[1] || !out[0]) return RG_ERR_NULL;
    if (p->k == 0 || p->k > TOPK_MAX || p->k > p->n || !(p->temperature > 0.f)) return RG_ERR_SHAPE;
    if (p->rows == 0) return RG_OK;
    auto st = static_cast<cudaStream_t>(stream);
    switch (p->dtype) {
        case RG_F32: return topk_sample_launch<float>(p, in, out, st);
        case RG_FP16: return topk_sample_launch<__half>(p, in, out, st);
        case RG_BF16: return topk_sample_launch<__nv_bfloat16>(p, in, out, st);
        default: return RG_ERR_DTYPE;
    }
}
}
