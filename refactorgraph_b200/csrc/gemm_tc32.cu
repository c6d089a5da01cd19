// fp32 MatMul on the fifth-generation tensor cores:  Y = alpha * A B (+ beta * C) with fp32 operands, results and partial sums
// (MatMulInfo semantics, src/04kernel/src/attributes/mat_mul_info.cc:27-42).  The CUDA cores bound the tiled kernel it stands in
// for at 72 TFLOP/s; six bf16 products per fp32 product leave the tensor cores a bound of 265.
//
// Every operand x is written as hi + mid + lo, three bf16 values: hi is x rounded to eight significand bits, mid the rest rounded to eight,
// lo what is left of it.  bf16 ends at 2^-133 and fp32 at 2^-149, so 2^16 x is what is taken apart: the three parts are then exactly
// 2^16 x for every x below 2^112, subnormal numbers included, and the sums are 2^32 times as large until the last step.  Of the nine
// products of two such sums the six largest are computed (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi); |mid| is at most 2^-8 |x| and
// |lo| 2^-17 |x|, so the other three are together at most 2^-24 of the product of the values, as much as one rounding, with either sign.  The
// tensor core adds into fp32 but does not round to nearest, so the large product is not left to accumulate there: its sum over 64
// values of k goes to registers and is added with ordinary fp32 additions.  The five small products accumulate in tensor memory over
// the whole k range, where their error is 2^-8 smaller.  Error against 64 bits (2-norm, normal data) here / of a chain of fp32
// multiply-adds: k = 1 2.57e-8 / 2.52e-8, 2 2.6e-8 / 3.1e-8, 8 3.0e-8 / 5.3e-8, 64 0.69e-7 / 1.4e-7, 1024 0.91e-7 / 5.7e-7, 11008 1.3e-7 /
// 1.9e-6; the automatic route leaves sums of fewer than eight products to the CUDA cores.  With all nine products but lo lo a single
// product is as close as a multiply-add, and 509 x 32000 x 1024 takes 280 us.
// Infinities, NaNs, operands from 2^112 and sums from 2^96 on leave a result that is not finite; such results are computed again
// from the operands in fp32 multiply-adds, so they are what fp32 gives.
//
// D[i, j] = sum_k P[i, k] Q[j, k] on tiles of 128 x BN.  P = A and Q = B with BN = 128; up to 64 rows of A change sides, so that the
// weights fill the 128 rows of the instruction and are converted once (BN = 32 or 64).  Either operand may be stored with k or with
// i / j innermost (K-major or MN-major in shared memory; nothing is transposed).  Roles of the warps:
//   converters  eight warps (two such groups on alternate k-blocks for up to 32 rows, a form bound by the weights' stream):
//               16-byte loads one k-block ahead in registers, three 16-byte stores per eight values into the swizzled planes
//   drainers    add the large product's accumulator (double-buffered) to registers after every 64 values of k; one thread of the
//               first issues the 24 tcgen05.mma (kind::f16, 128 x BN x 16) of the k-block after the one it is about to drain (a
//               seventeenth warp for that would take a quarter of everybody's registers; the skinny forms have it)
// FAST: rows on 16 bytes and k, and n where it is innermost, multiples of 8.  Addresses are then 32-bit offsets kept per item, rows past the
// edge repeat the last one (they only reach results that are not stored) and only the last k-block looks at the end of k.  With
// bounds and addresses worked out per piece the converters executed twice the instructions and set the pace: 509 x 2752 x 1024 45.3 us then,
// 38.4 without; 509 x 32000 x 1024 281 and 235.  The factor of 2^16 costs them 3 to 5 % where weights are stored [k, n] (41 and 249 us,
// 134 TFLOP/s) and up to 10 % in the skinny forms.
// k is split between CTAs where tiles are few; the last to arrive adds the parked sums in order.
// Measured against the 64 x 64 CUDA-core tiles: 509 x 32000 x 1024 1433 us, 509 x 2752 x 1024 128, 32 x 32000 x 1024 295 (54 here).
#include "gemm_dispatch.cuh"
#include "tcgen05.cuh"

namespace rg {

static __device__ int s_tc32_error;

constexpr int T3_BM = 128, T3_BK = 64;
constexpr float T3_SCALE = 65536.f, T3_UNSCALE = 1.f / (65536.f * 65536.f);// of the operands, and of the sums of their products

template<int BN> struct Tc32Shape {
    static constexpr int STAGES = BN == 128 ? 2 : 3, GROUPS = BN == 32 ? 2 : 1, CONV = 8 * GROUPS, EPI = BN == 128 ? 8 : 4;
    static constexpr int COLS = BN * 4 / EPI;// accumulator columns of a drainer thread
    static constexpr bool ISSUER = BN != 128;// a warp of its own for the thread that issues the products
    static constexpr int THREADS = (CONV + EPI + (ISSUER ? 1 : 0)) * 32;
    static constexpr uint32_t P_TILE = T3_BM * T3_BK * 2, Q_TILE = BN * T3_BK * 2, STAGE = 3 * (P_TILE + Q_TILE);
    static constexpr size_t SMEM = STAGES * STAGE + (2 * STAGES + 6) * 8 + 16 + 1024;
};

struct Tc32Operand {
    const float *x;                // k innermost: element (i, k) at x[i * ld + k]; i innermost: x[k * ld + i]
    uint64_t stride;               // elements between the matrices of a batch
    uint32_t outer, inner, ld, vec;// vec: rows start on 16 bytes
};
struct Tc32Args {
    Tc32Operand p, q;
    float *Y;
    const float *C;
    float *partial;   // [item][BN][128], used when splits > 1
    unsigned *counter;// [tile], zero before the first call and left at zero
    uint32_t rows, cols, k;// D is rows x cols
    uint32_t m_tiles, n_tiles, tiles, splits;
    uint64_t stride_y, stride_c, y_i, y_j, c_i, c_j;
    float alpha, beta;
};

__device__ __forceinline__ uint32_t tc32_round(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// eight values -> one 16-byte piece of each plane
__device__ __forceinline__ void tc32_planes(const float (&v)[8], uint4 &hi, uint4 &mid, uint4 &lo) {
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float a = v[2 * j] * T3_SCALE, b = v[2 * j + 1] * T3_SCALE;
        const uint32_t h = tc32_round(a, b);
        const float a1 = a - __uint_as_float(h << 16), b1 = b - __uint_as_float(h & 0xffff0000u);
        const uint32_t m = tc32_round(a1, b1);
        const float a2 = a1 - __uint_as_float(m << 16), b2 = b1 - __uint_as_float(m & 0xffff0000u);
        w[0][j] = h, w[1][j] = m, w[2][j] = __byte_perm(__float_as_uint(a2), __float_as_uint(b2), 0x7632);// at most 7 bits are left: cutting is exact
    }
    hi = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]);
    mid = make_uint4(w[1][0], w[1][1], w[1][2], w[1][3]);
    lo = make_uint4(w[2][0], w[2][1], w[2][2], w[2][3]);
}
// Eight innermost-consecutive values of an operand at (outer, inner); zeros outside the matrix.
__device__ __forceinline__ void tc32_load(const Tc32Operand &o, const float *base, uint32_t outer, uint32_t inner, float (&v)[8]) {
    const float *src = base + static_cast<uint64_t>(outer) * o.ld + inner;
    if (o.vec && outer < o.outer && inner + 8 <= o.inner) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(src)), b = __ldg(reinterpret_cast<const float4 *>(src) + 1);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = outer < o.outer && inner + j < o.inner ? __ldg(src + j) : 0.f;
    }
}
__device__ __forceinline__ bool t3_warp_wait(uint64_t *bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity) ? 1 : 0) != 0; }

// Walks a CTA's items (tile, split of k) and the k-blocks inside them.
struct Tc32Walk {
    uint32_t item, b, mt, nt, kb, kb0, kb1;
    __device__ __forceinline__ bool open(const Tc32Args &a, uint32_t kblocks) {
        if (item >= a.tiles * a.splits) return false;
        const uint32_t ks = item % a.splits, tile = item / a.splits, per = a.m_tiles * a.n_tiles, in = tile % per;
        b = tile / per, mt = in % a.m_tiles, nt = in / a.m_tiles;// neighbours share a column tile
        kb0 = kb = static_cast<uint32_t>(static_cast<uint64_t>(kblocks) * ks / a.splits), kb1 = static_cast<uint32_t>(static_cast<uint64_t>(kblocks) * (ks + 1) / a.splits);
        return true;
    }
    __device__ __forceinline__ bool next(const Tc32Args &a, uint32_t kblocks) {
        if (++kb < kb1) return true;
        item += gridDim.x;
        return open(a, kblocks);
    }
};

// Results j0 + j of this lane's row i, j a bit of its `odd`, once more as chains of fp32 multiply-adds: the parts of an infinity are not
// numbers, and the scaled values and sums overflow where those of the operands do not.  All lanes work on the columns that any of
// them needs, eight at a time, so that a value of Q serves 32 rows and one of P eight columns.  A function of its own behind the
// stores of the others, so that it takes no registers from the converters' loop (inlined, 509 x 32000 x 1024 took 313 us instead
// of 249).
template<int COLS, bool P_MN, bool Q_MN> static __device__ __noinline__ void tc32_mend(const Tc32Args &a, uint32_t b, uint32_t i, uint32_t j0, uint64_t odd) {
    const uint64_t p_k = P_MN ? a.p.ld : 1, q_k = Q_MN ? a.q.ld : 1, q_j = Q_MN ? 1 : a.q.ld;
    const uint32_t row = i < a.rows ? i : a.rows - 1;// a row past the edge repeats the last one and stores nothing
    const float *p = a.p.x + b * a.p.stride + (P_MN ? row : static_cast<uint64_t>(row) * a.p.ld);
    const uint64_t any = static_cast<uint64_t>(__reduce_or_sync(0xffffffffu, static_cast<uint32_t>(odd >> 32))) << 32 | __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(odd));
    for (uint32_t g = 0; g < COLS; g += 8) {
        if ((any >> g & 0xffu) == 0) continue;
        const float *q = a.q.x + b * a.q.stride;
        uint64_t at[8];
        float s[8];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) {
            const uint32_t j = j0 + g + e;
            at[e] = (j < a.cols ? j : a.cols - 1) * q_j, s[e] = 0.f;
        }
#pragma unroll 4
        for (uint32_t k = 0; k < a.k; ++k, p += p_k, q += q_k) {
            const float x = __ldg(p);
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e) s[e] = fmaf(x, __ldg(q + at[e]), s[e]);
        }
        p -= a.k * p_k;
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) {
            const uint32_t j = j0 + g + e;
            if ((odd >> (g + e) & 1u) == 0) continue;
            float y = s[e] * a.alpha;
            if (a.C) y += a.beta * a.C[b * a.stride_c + row * a.c_i + j * a.c_j];
            a.Y[b * a.stride_y + row * a.y_i + j * a.y_j] = y;
        }
    }
}

template<int BN, bool P_MN, bool Q_MN, bool FAST>
__global__ void __launch_bounds__(Tc32Shape<BN>::THREADS, 1) gemm_tc32_kernel(const __grid_constant__ Tc32Args a) {
    using Sh = Tc32Shape<BN>;
    constexpr int STAGES = Sh::STAGES, GROUPS = Sh::GROUPS, EPI = Sh::EPI, COLS = Sh::COLS;
    constexpr uint32_t P_TILE = Sh::P_TILE, Q_TILE = Sh::Q_TILE, STAGE = Sh::STAGE;
    constexpr int NP = T3_BM * T3_BK / 8 / 256, NQ = BN * T3_BK / 8 / 256;// pieces of eight values per converter thread and k-block
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE);
    uint64_t *empty = full + STAGES;
    uint64_t *big_full = empty + STAGES;  // [2] the large product's accumulator holds 64 values of k
    uint64_t *big_empty = big_full + 2;   // [2]
    uint64_t *small_empty = big_empty + 2;// [2] the small products' accumulator of an item has been read
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(small_empty + 2);
    int *failed = reinterpret_cast<int *>(tmem_slot + 1);
    __shared__ int s_last;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t kblocks = (a.k + T3_BK - 1) / T3_BK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 8), mbar_init(&empty[s], 1);
        for (int s = 0; s < 2; ++s) mbar_init(&big_full[s], 1), mbar_init(&big_empty[s], EPI), mbar_init(&small_empty[s], EPI);
        *failed = 0;
        fence_mbar_init();
    }
    if (warp == EPI) {
        tmem_alloc(tmem_slot, 4 * BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;// columns: large product 0 / 1, small products 0 / 1, BN each
    pdl_enter();
    Tc32Walk w;
    w.item = blockIdx.x;

    if (warp >= EPI && warp < EPI + Sh::CONV) {
        // ---- converters ----
        const uint32_t group = (warp - EPI) / 8, t = threadIdx.x - EPI * 32 - group * 256;
        // piece c of a tile: K-major (row, 8 k) = (c / 8, c % 8); MN-major (k, 8 rows) = (c / (rows / 8), c % (rows / 8))
        uint32_t offp[NP], offq[NQ];// FAST: offsets of this thread's pieces from the k-block's first element
        auto aim = [&]() {
            if constexpr (FAST) {
                auto offset = [&](const Tc32Operand &o, bool mn, uint32_t rows, uint32_t tile, int i) {
                    const uint32_t c = t + i * 256;
                    if (mn) {
                        const uint32_t col = tile * rows + c % (rows / 8) * 8;
                        return c / (rows / 8) * o.ld + (col < o.inner ? col : o.inner - 8);
                    }
                    const uint32_t row = tile * rows + c / 8;
                    return (row < o.outer ? row : o.outer - 1) * o.ld + c % 8 * 8;
                };
#pragma unroll
                for (int i = 0; i < NP; ++i) offp[i] = offset(a.p, P_MN, T3_BM, w.mt, i);
#pragma unroll
                for (int i = 0; i < NQ; ++i) offq[i] = offset(a.q, Q_MN, BN, w.nt, i);
            }
        };
        auto fetch = [&](float (&v)[NP + NQ][8], int i) {
            const bool first = i < NP, mn = first ? P_MN : Q_MN;
            const uint32_t c = t + (first ? i : i - NP) * 256, rows = first ? T3_BM : BN, tile = first ? w.mt : w.nt;
            const Tc32Operand &o = first ? a.p : a.q;
            const float *base = o.x + w.b * o.stride;
            if constexpr (FAST) {
                const float4 *src = reinterpret_cast<const float4 *>(base + (mn ? static_cast<uint64_t>(w.kb * T3_BK) * o.ld : w.kb * T3_BK) + (first ? offp[i] : offq[i - NP]));
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
                if ((w.kb + 1) * T3_BK <= a.k) {// the same for every thread
                    x = __ldg(src), y = __ldg(src + 1);
                } else if (w.kb * T3_BK + (mn ? c / (rows / 8) : c % 8 * 8) < a.k) {
                    x = __ldg(src), y = __ldg(src + 1);
                }
                v[i][0] = x.x, v[i][1] = x.y, v[i][2] = x.z, v[i][3] = x.w, v[i][4] = y.x, v[i][5] = y.y, v[i][6] = y.z, v[i][7] = y.w;
            } else {
                if (mn) tc32_load(o, base, w.kb * T3_BK + c / (rows / 8), tile * rows + c % (rows / 8) * 8, v[i]);
                else
                    tc32_load(o, base, tile * rows + c / 8, w.kb * T3_BK + c % 8 * 8, v[i]);
            }
        };
        bool more = w.open(a, kblocks), ok = true;
        for (uint32_t g = 0; more && g < group; ++g) more = w.next(a, kblocks);
        float v[NP + NQ][8];
        if (more) {
            aim();
#pragma unroll
            for (int i = 0; i < NP + NQ; ++i) fetch(v, i);
        }
        for (uint32_t it = group; more; it += GROUPS) {
            const uint32_t s = it % STAGES;
            ok = ok && t3_warp_wait(&empty[s], ((it / STAGES) & 1u) ^ 1u);
            if (!ok) {
                *failed = 1;
                break;
            }
            const uint32_t item = w.item;
            for (int g = 0; more && g < GROUPS; ++g) more = w.next(a, kblocks);// the block fetched while this one is converted
            if (more && w.item != item) aim();
            uint8_t *st = smem + s * STAGE;
#pragma unroll
            for (int i = 0; i < NP + NQ; ++i) {
                const uint32_t c = t + (i < NP ? i : i - NP) * 256;
                const bool mn = i < NP ? P_MN : Q_MN;
                const uint32_t per = (i < NP ? T3_BM : BN) / 8;
                // 128-byte rows: K-major one per row of the tile, MN-major one per k and block of 64 rows; 16-byte pieces permuted by the row
                const uint32_t r = mn ? c / per : c / 8, piece = mn ? c % per % 8 : c % 8, block = mn ? c % per / 8 : 0;
                uint8_t *dst = st + (i < NP ? 0 : 3 * P_TILE) + block * (T3_BK * 128) + r * 128 + ((piece ^ (r & 7u)) << 4);
                const uint32_t plane = i < NP ? P_TILE : Q_TILE;
                uint4 hi, mid, lo;
                tc32_planes(v[i], hi, mid, lo);
                *reinterpret_cast<uint4 *>(dst) = hi;
                *reinterpret_cast<uint4 *>(dst + plane) = mid;
                *reinterpret_cast<uint4 *>(dst + 2 * plane) = lo;
                if (more) fetch(v, i);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");// the tensor core reads shared memory through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else {
        // the products of the next k-block of this CTA's schedule (one thread)
        Tc32Walk wi = w;
        uint32_t issued = 0, items_issued = 0, d_small = 0;
        bool to_issue = warp == (Sh::ISSUER ? EPI + Sh::CONV : 0) && lane == 0 && wi.open(a, kblocks);
        auto issue = [&]() {
            const uint32_t idesc = instr_desc(1, T3_BM, BN) | (P_MN ? 1u << 15 : 0u) | (Q_MN ? 1u << 16 : 0u);
            const uint32_t s = issued % STAGES, buf = issued & 1u, d_big = tmem + buf * BN;
            const bool fresh = wi.kb == wi.kb0;
            bool good = true;
            if (fresh) {
                d_small = tmem + (2 + (items_issued & 1u)) * BN;
                good = mbar_wait(&small_empty[items_issued & 1u], ((items_issued >> 1) & 1u) ^ 1u);
                ++items_issued;
            }
            good = good && mbar_wait(&big_empty[buf], ((issued >> 1) & 1u) ^ 1u) && mbar_wait(&full[s], (issued / STAGES) & 1u);
            if (!good) {
                *failed = 3;
                to_issue = false;
                return;
            }
            tc_fence_after();
            const uint32_t ps = smem_u32(smem + s * STAGE), qs = ps + 3 * P_TILE;
            auto product = [&](uint32_t d, uint32_t pp, uint32_t qp, bool first) {
#pragma unroll
                for (uint32_t kk = 0; kk < T3_BK / 16; ++kk) {
                    const uint32_t pt = ps + pp * P_TILE, qt = qs + qp * Q_TILE;
                    const uint64_t pd = P_MN ? smem_desc_sw128_mn(pt + kk * 2048, T3_BK * 128) : smem_desc_sw128(pt + kk * 32);
                    const uint64_t qd = Q_MN ? smem_desc_sw128_mn(qt + kk * 2048, T3_BK * 128) : smem_desc_sw128(qt + kk * 32);
                    tc_mma_f16(d, pd, qd, idesc, first && kk == 0 ? 0u : 1u);
                }
            };
            product(d_big, 0, 0, true);
            product(d_small, 0, 2, fresh);
            product(d_small, 2, 0, false);
            product(d_small, 1, 1, false);
            product(d_small, 0, 1, false);
            product(d_small, 1, 0, false);
            tc_commit(&empty[s]);
            tc_commit(&big_full[buf]);
            ++issued;
            to_issue = wi.next(a, kblocks);
        };
        if constexpr (Sh::ISSUER) {
            while (to_issue) issue();
            if (warp >= EPI) w.item = a.tiles * a.splits;// nothing to drain
        } else if (to_issue) {
            issue();
        }
        __syncwarp();
        // ---- drainers: warp w reads the tensor-memory lanes of quarter w % 4 (tile rows), COLS columns of them ----
        const uint32_t quarter = warp & 3u, col = (warp >> 2) * COLS, trow = quarter * 32 + lane, lanes = (quarter * 32u) << 16;
        uint32_t it = 0, local = 0;
        bool ok = true;// after a wait that ran out nothing is waited for any more, but every barrier of the block is still met
        for (bool more = w.open(a, kblocks); more; ++local) {
            float acc[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
            const uint32_t item = w.item, tile = item / a.splits, mt = w.mt, nt = w.nt, b = w.b;
            for (uint32_t kb = w.kb0; kb < w.kb1; ++kb, ++it) {
                const uint32_t buf = it & 1u;
                if constexpr (!Sh::ISSUER) {
                    if (to_issue) issue();
                    __syncwarp();
                }
                ok = ok && t3_warp_wait(&big_full[buf], (it >> 1) & 1u);
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    uint32_t r[16];
                    tmem_ld_32x16(tmem + buf * BN + col + c + lanes, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&big_empty[buf]);
            }
#pragma unroll
            for (int c = 0; c < COLS; c += 16) {
                uint32_t r[16];
                tmem_ld_32x16(tmem + (2 + (local & 1u)) * BN + col + c + lanes, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&small_empty[local & 1u]);
            if (!ok) *failed = 4;
            w.item += gridDim.x;
            more = w.open(a, kblocks);
            const uint32_t i = mt * T3_BM + trow, j0 = nt * BN + col;
            if (a.splits > 1) {
                // park this split's sums, column by column so that a warp writes whole lines; the last split of the tile to arrive
                // adds all of them in split order
                float *mine = a.partial + static_cast<size_t>(item) * (T3_BM * BN) + col * T3_BM + trow;
#pragma unroll
                for (int j = 0; j < COLS; ++j) mine[j * T3_BM] = acc[j];
                asm volatile("bar.sync 2, %0;" ::"n"(EPI * 32) : "memory");
                if (threadIdx.x == 0) {
                    unsigned old;
                    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.counter + tile) : "memory");
                    s_last = old == a.splits - 1 ? 1 : 0;
                }
                asm volatile("bar.sync 2, %0;" ::"n"(EPI * 32) : "memory");
                const bool last = s_last != 0;
                asm volatile("bar.sync 2, %0;" ::"n"(EPI * 32) : "memory");
                if (!last) continue;
                const float *base = a.partial + static_cast<size_t>(tile) * a.splits * (T3_BM * BN) + col * T3_BM + trow;
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
                for (uint32_t s = 0; s < a.splits; ++s) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j) acc[j] += __ldcg(base + static_cast<size_t>(s) * (T3_BM * BN) + j * T3_BM);
                }
                if (threadIdx.x == 0) a.counter[tile] = 0u;
            }
            uint64_t odd = 0;// results of this row that are not finite
            if (i < a.rows) {
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] *= T3_UNSCALE;
                float probe = 0.f;
#pragma unroll
                for (int j = 0; j < COLS; ++j) probe = fmaf(acc[j], 0.f, probe);
                if (probe != 0.f) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (!(fabsf(acc[j]) <= 3.402823466e38f) && j0 + j < a.cols) odd |= 1ull << j;
                }
                float *y = a.Y + b * a.stride_y + i * a.y_i + j0 * a.y_j;
#pragma unroll
                for (int j = 0; j < COLS; ++j) acc[j] *= a.alpha;
                if (a.C) {
                    const float *c = a.C + b * a.stride_c + i * a.c_i + j0 * a.c_j;
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (j0 + j < a.cols) acc[j] += a.beta * c[j * a.c_j];
                }
                if (odd == 0 && a.y_j == 1 && j0 + COLS <= a.cols && (reinterpret_cast<uintptr_t>(y) & 15u) == 0) {
#pragma unroll
                    for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4 *>(y + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (j0 + j < a.cols && (odd >> j & 1u) == 0) y[j * a.y_j] = acc[j];
                }
            }
            if (__any_sync(0xffffffffu, odd != 0)) tc32_mend<COLS, P_MN, Q_MN>(a, b, i, j0, odd);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == EPI) {
        tc_fence_after();
        tmem_dealloc(tmem, 4 * BN);
    }
    if (threadIdx.x == 0 && *failed) atomicExch(&s_tc32_error, *failed);
}

// ---- host ------------------------------------------------------------------------------------------------------
struct Tc32Plan {
    bool swap;
    uint32_t bn, m_tiles, n_tiles, tiles, splits;
    size_t counter_bytes, partial_bytes;
};
static Tc32Plan tc32_plan(const rg_mat_mul_params *p) {
    Tc32Plan pl;
    const uint32_t sms = static_cast<uint32_t>(sm_count()), kblocks = (p->k + T3_BK - 1) / T3_BK;
    pl.swap = p->m <= 64;
    pl.bn = !pl.swap ? 128 : p->m <= 32 ? 32 : 64;
    pl.m_tiles = ((pl.swap ? p->n : p->m) + T3_BM - 1) / T3_BM, pl.n_tiles = ((pl.swap ? p->m : p->n) + pl.bn - 1) / pl.bn;
    pl.tiles = pl.m_tiles * pl.n_tiles * p->batch;
    // split k where that shortens the longest chain of k-blocks on an SM by more than the parked sums cost (about three blocks,
    // and one more for every two of them to add)
    pl.splits = 1;
    uint64_t best = (static_cast<uint64_t>(pl.tiles) + sms - 1) / sms * kblocks;
    for (uint32_t s = 2; s <= 16 && s * 2 <= kblocks; ++s) {
        const uint64_t cost = (static_cast<uint64_t>(pl.tiles) * s + sms - 1) / sms * ((kblocks + s - 1) / s) + 3 + s / 2;
        if (cost < best) best = cost, pl.splits = s;
    }
    pl.counter_bytes = pl.splits > 1 ? (static_cast<size_t>(pl.tiles) * 4 + 255) / 256 * 256 : 0;
    pl.partial_bytes = pl.splits > 1 ? static_cast<size_t>(pl.tiles) * pl.splits * T3_BM * pl.bn * 4 : 0;
    return pl;
}
// 8 us before the first result, then the longest chain of k-blocks on an SM at 1.8 us (128 columns), 1.45 or 1.4 us, 4.3 us (fewer columns: 1.2) for
// every tile but the last on an SM (its results are stored while the next tile waits for the drainers), and the parked sums.  Rows off 16
// bytes: 2.2 us a k-block, and 7 us a tile where it is the results' (16 x 509 x 509 x 64 28.5 us)
float gemm_tc32_us(const rg_mat_mul_params *p) {
    const Tc32Plan pl = tc32_plan(p);
    const uint32_t sms = static_cast<uint32_t>(sm_count()), kblocks = (p->k + T3_BK - 1) / T3_BK;
    const uint64_t rounds = (static_cast<uint64_t>(pl.tiles) * pl.splits + sms - 1) / sms;
    return 8.f + static_cast<float>(rounds) * static_cast<float>((kblocks + pl.splits - 1) / pl.splits) * (pl.bn == 32 ? 1.4f : pl.bn == 64 ? 1.45f : p->k % 8 == 0 && (p->trans_b || p->n % 8 == 0) ? 1.8f : 2.2f) +
           (pl.bn == 128 ? 4.3f : 1.2f) * static_cast<float>(rounds - 1) + (pl.bn == 128 && p->n % 4 ? 7.f * static_cast<float>(rounds) : 0.f) +
           (pl.splits > 1 ? 2.f + 0.6f * static_cast<float>(pl.splits) : 0.f);
}
size_t gemm_tc32_workspace(const rg_mat_mul_params *p) {
    const Tc32Plan pl = tc32_plan(p);
    return pl.counter_bytes + pl.partial_bytes;
}

template<int BN, bool P_MN, bool Q_MN, bool FAST>
static int tc32_launch(const Tc32Args &a, cudaStream_t st) {
    auto kern = gemm_tc32_kernel<BN, P_MN, Q_MN, FAST>;
    constexpr size_t smem = Tc32Shape<BN>::SMEM;
    RG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const uint32_t items = a.tiles * a.splits, sms = static_cast<uint32_t>(sm_count());
    RG_CHECK_CUDA(launch_pdl(kern, dim3(items < sms ? items : sms), dim3(Tc32Shape<BN>::THREADS), smem, st, a));
    count_launch();
    return launch_status();
}
// ws may be NULL: k is then not split
int gemm_tc32(const rg_mat_mul_params *p, void *ws, const void *const *in, void *const *out, cudaStream_t st) {
    if (p->dtype != RG_F32 || p->trans_a) return RG_ERR_UNSUPPORTED;
    Tc32Plan pl = tc32_plan(p);
    if (!ws) pl.splits = 1;
    if (static_cast<uint64_t>(pl.m_tiles) * pl.n_tiles * p->batch * pl.splits > 0x7fffffffull) return RG_ERR_SHAPE;
    Tc32Operand oa = {static_cast<const float *>(in[0]), p->stride_a, p->m, p->k, p->k, 0};
    Tc32Operand ob = {static_cast<const float *>(in[1]), p->stride_b, p->trans_b ? p->n : p->k, p->trans_b ? p->k : p->n, p->trans_b ? p->k : p->n, 0};
    for (Tc32Operand *o : {&oa, &ob}) o->vec = aligned16(o->x) && o->ld % 4 == 0 && o->stride % 4 == 0;
    Tc32Args a = {};
    a.p = pl.swap ? ob : oa, a.q = pl.swap ? oa : ob;
    a.Y = static_cast<float *>(out[0]), a.C = p->has_bias ? static_cast<const float *>(in[2]) : nullptr;
    a.counter = static_cast<unsigned *>(ws), a.partial = reinterpret_cast<float *>(static_cast<uint8_t *>(ws) + pl.counter_bytes);
    a.rows = pl.swap ? p->n : p->m, a.cols = pl.swap ? p->m : p->n, a.k = p->k;
    a.m_tiles = pl.m_tiles, a.n_tiles = pl.n_tiles, a.tiles = pl.tiles, a.splits = pl.splits;
    a.stride_y = p->stride_y, a.stride_c = p->stride_c;
    a.y_i = pl.swap ? 1 : p->n, a.y_j = pl.swap ? p->n : 1;
    a.c_i = pl.swap ? p->bias_col_stride : p->bias_row_stride, a.c_j = pl.swap ? p->bias_row_stride : p->bias_col_stride;
    a.alpha = p->alpha, a.beta = p->beta;
    const auto small = [](const Tc32Operand &o) { return static_cast<uint64_t>(o.outer + 128) * o.ld < (1ull << 31); };
    const bool fast = oa.vec && ob.vec && p->k % 8 == 0 && (p->trans_b || p->n % 8 == 0) && small(oa) && small(ob);
#define RG_TC32(BN, P_MN, Q_MN) (fast ? tc32_launch<BN, P_MN, Q_MN, true>(a, st) : tc32_launch<BN, P_MN, Q_MN, false>(a, st))
    if (!pl.swap) return p->trans_b ? RG_TC32(128, false, false) : RG_TC32(128, false, true);
    if (pl.bn == 32) return p->trans_b ? RG_TC32(32, false, false) : RG_TC32(32, true, false);
    return p->trans_b ? RG_TC32(64, false, false) : RG_TC32(64, true, false);
#undef RG_TC32
}

int gemm_tc32_error_word(bool clear) { return error_symbol(s_tc32_error, clear); }

}// namespace rg
