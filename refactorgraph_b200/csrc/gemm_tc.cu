// Tensor-core GEMM for sm_100a:  Y[m,n] = alpha * A[m,k] * B[n,k]^T (+ beta * C),  fp16 / bf16 operands (both
// K-major: activations [tokens, k] and weights [out, in], the reference MatMul with transB = 1), fp32 accumulation
// in tensor memory.  Replaces the cublasGemmEx call of MatMulCublas
// (src/04kernel/src/kernels/mat_mul/cublas_kernel.cu:48-55) for prefill-sized products.
//
// Persistent CTAs (one per SM) walk 128 x BN output tiles (BN = 256 or 128; 64 / 32 with the operands swapped so that a
// skinny activation matrix becomes the N side of the instruction) in an L2-friendly grouped order:
//   warp 4  (one thread): TMA producer — cp.async.bulk.tensor.2d loads of the A tile [128 x 64] and B tile [BN x 64]
//                         with the 128-byte swizzle into a STAGES-deep shared-memory ring (full[] mbarriers).
//   warp 5  (one thread): MMA issuer — per stage four tcgen05.mma.cta_group::1.kind::f16 (M 128, N BN, K 16) whose
//                         shared-memory descriptors advance 32 bytes along K inside the swizzle atom; tcgen05.commit
//                         releases the stage (empty[]) and finally signals the accumulator (acc_full).
//   warps 0-3:            epilogue — tcgen05.ld of each warp's 32 TMEM lanes, alpha/beta/bias, conversion, stores.
// The accumulator is double-buffered in tensor memory (2 x BN columns, acc_full[] / acc_empty[] mbarriers), so a tile's
// epilogue overlaps the next tile's main loop.  Warp 5 also allocates and frees the TMEM columns.  Every mbarrier wait is bounded; on expiry the CTA records
// an error word, still frees its tensor memory and exits.
// Large products (512 rows and more, where tc_wide_tile says so) run on CTA pairs (template flag PAIR, tcgen05 ... cta_group::2): see
// the comment above the kernel.
#include "gemm_dispatch.cuh"
#include "tcgen05.cuh"
#include "ar_slots.cuh"
#include <atomic>
#include <cstdlib>
#include <type_traits>
#include <cuda.h>

namespace rg {

static __device__ int s_tc_error;
static __device__ int s_tc_index_error;// a cache-append position or block-table entry was out of range (store skipped)

constexpr int TC_BM = 128;
constexpr int TC_BK = 64;// 64 x 2 B = one 128-byte swizzle row
constexpr int TC_THREADS = 192;
__host__ __device__ constexpr uint32_t tc_recv_bytes(int bn) { return bn <= 64 ? 128u * bn * 4u : 0u; }// a tile's sums, from all CTAs of a cluster
constexpr uint32_t TC_MN_BLOCK = 64 * TC_BK * 2;// one box of an MN-major operand: 64 columns x 64 k-rows

struct TcArgs {
    void *Y;
    const void *C;
    uint32_t m, n, k;// problem as the kernel sees it: D[m,n] = A[m,k] B[n,k]^T
    float alpha, beta;
    uint32_t c_row_stride, c_col_stride;
    uint64_t y_row_stride, y_col_stride;// element strides of Y over the kernel's (row, col) = lets swapped runs write Y^T
    int is_bf16;
    uint32_t ksplit;   // CTAs of a cluster that share a tile, each with its part of k (skinny forms; 1 elsewhere)
    uint32_t group_m;  // row tiles per group of the tile order
    uint32_t early;    // operand that no earlier kernel of the stream writes (a weight): 1 = A, 2 = B, 0 = neither
    // QKV epilogue (rope != 0): columns are [q heads | k heads | v heads] of head_dim 128, rows are tokens; q is rotated into
    // q_out[token, nq * 128], k rotated and v copied into the caches at pos[token] of sequence token / tokens_per_seq
    uint32_t swiglu;   // != 0: B tile = 128 gate rows + the matching 128 up rows (swiglu rows further down B); Y[m, n / 2] = silu(g) * u
    uint32_t rope, nq, tokens_per_seq;
    float log2_theta;
    const int64_t *pos;
    const int32_t *table;
    void *q_out, *kc, *vc;
    rg_kv_layout kv;
    // push != 0 (weights on the M side only): the finished 16-bit values do not go to Y; paired with the flag of the all-reduce
    // call in flight they are stored into this rank's input slot in the allocation of every rank (1, one-shot) or of the rank
    // that owns the run of chunks (2, two-shot), over NVLink with ordinary 8-byte stores — the row-parallel product and the send
    // half of the all-reduce are one kernel
    uint32_t push;
    ArPeers ar;
};

// Row `feat` of the kernel's output (an output feature; a.m of them) for token `tok`: even lanes take the value of the next
// lane (feature feat + 1: both lie in one 16-byte chunk of the token's row) and store {two 16-bit values, flag}.  Called by all
// 32 lanes of a warp; `live` = this lane's row exists.
template<class T>
__device__ __forceinline__ void tc_push_value(const TcArgs &a, uint32_t flag, unsigned q, uint32_t feat, uint32_t tok, float v, bool live, uint32_t lane) {
    const float vn = __shfl_down_sync(0xffffffffu, v, 1);
    if ((lane & 1u) || !live) return;
    const T lo = Num<T>::from_f(v), hi = Num<T>::from_f(vn);
    const uint32_t data = static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&lo)) | (static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&hi)) << 16);
    const uint64_t e = static_cast<uint64_t>(tok) * a.m + feat, chunk = e >> 3;
    const size_t off = ar_slot_offset(a.ar.capacity, a.ar.world, q, a.ar.rank) + chunk * 32 + ((e & 7u) >> 1) * 8;
    if (a.push == 2) {
        const int owner = static_cast<int>((chunk / 32) % static_cast<uint64_t>(a.ar.world));
        asm volatile("st.global.cg.v2.u32 [%0], {%1, %2};" ::"l"(a.ar.peer[owner] + off), "r"(data), "r"(flag) : "memory");
    } else {
#pragma unroll
        for (int r = 0; r < AR_MAX_RANKS; ++r)
            if (r < a.ar.world) asm volatile("st.global.cg.v2.u32 [%0], {%1, %2};" ::"l"(a.ar.peer[r] + off), "r"(data), "r"(flag) : "memory");
    }
}

// Tile order: groups of TC_GROUP_M row tiles are walked column by column, so the CTAs running at the same time share
// a few A row-panels and B column-panels in L2 instead of streaming all of B once per row tile.
constexpr uint32_t TC_GROUP_M = 16;
__device__ __forceinline__ void tile_coords(uint32_t t, uint32_t m_tiles, uint32_t n_tiles, uint32_t &mt, uint32_t &nt, uint32_t group_m = TC_GROUP_M) {
    const uint32_t per_group = group_m * n_tiles;
    const uint32_t grp = t / per_group, first = grp * group_m;
    const uint32_t rows = m_tiles - first < group_m ? m_tiles - first : group_m;
    const uint32_t r = t - grp * per_group;
    mt = first + r % rows;
    nt = r / rows;
}

// A unit's work: tiles unit, unit + units, ... over the k-blocks [kb0, kb1).  A unit is a CTA, a pair of CTAs (pair mode) or a cluster
// of ksplit CTAs that divide the k-blocks of each tile between them.
struct TcWalk {
    uint32_t tiles, units, item, kb0, kb1, tile;
    __device__ __forceinline__ void init(uint32_t tiles_, uint32_t kblocks, uint32_t unit, uint32_t units_, uint32_t part, uint32_t parts) {
        tiles = tiles_, units = units_, item = unit;
        kb0 = kblocks * part / parts, kb1 = kblocks * (part + 1) / parts;
    }
    __device__ __forceinline__ bool next() {
        if (item >= tiles) return false;
        tile = item;
        item += units;
        return true;
    }
};

// Persistent: CTA c computes tiles c, c + gridDim.x, ...  The accumulator is double-buffered in tensor memory (2 x BN
// columns), so the epilogue of one tile (tcgen05.ld, conversion, stores) overlaps the MMA main loop of the next.
// PAIR: two CTAs (a cluster of two on neighbouring SMs) compute one 256 x BN tile with tcgen05 ... cta_group::2: each CTA loads its
// 128 rows of A and HALF of the B tile, the even CTA issues the products for both, each CTA's tensor memory receives its 128 rows of
// the accumulator and its epilogue warps store them.  Per SM and k-block that is 32 KiB from L2 instead of 48 for the same 128 x 256
// outputs: the single-CTA kernel is bound by requests to L2 (ncu: 68 % of request cycles, tensor pipe 80 %; an extra L2 prefetch
// per box made it 22 % slower).  No load is multicast.
//
// k-split (skinny forms): a 128-row tile per CTA leaves most SMs idle or the last round nearly empty, so a cluster of 2, 4 or 8 CTAs
// shares each tile, every CTA streaming its part of k.  CTA r finishes columns (tokens) [r W, r W + W), W = BN / ksplit: the others
// store their sums of those columns into its receive buffer over distributed shared memory (st.shared::cluster, counted on its
// recv_full mbarrier; recv_free, counted on the senders', hands the buffer back), it adds them in rank order and runs the
// epilogue of its W columns.  Two receive buffers, so the exchange of a tile overlaps the stream of the next.  The wide forms do the
// same for products with fewer tiles than SMs, one tile per cluster: the receive buffer is then the ring itself, and
// recv_free says that all CTAs have read their last stage.
// Measured with stream-K / parked partial sums in global memory before: 8 tokens x 4096 x 4096 16.4 -> 11.6 us, 4096 x 11008 24.9 ->
// 19.8, 12288 x 4096 26.6 -> 23.2, 22016 x 4096 37.7 -> 36.5, 32000 x 4096 49.4 -> 47.1; an 8-layer 7B step of 8 sequences 1.37 -> 1.17 ms.
//
// MN: the weight matrix is stored [k, out] (MatMul with transB = 0, as exporters write it): its tile is loaded as boxes of 64 output
// columns x 64 k-rows, one 8 KiB block per 64 columns, and enters the instruction as an MN-major operand (the M side of the skinny
// forms, the N side otherwise).  A K step of 16 is then 16 rows = 2 KiB further inside each block; the next 64 columns are one
// block further (leading offset), the next 8 rows 1 KiB further (stride offset).  Nothing is transposed in memory.  These products ran
// on the CUDA cores before: a two-layer 7B decoder on a 300-token prompt, fp16, all weights [k, out], 11.3 ms then, 0.81 ms now.
template<class T, int BN, int STAGES, bool PUSH = false, bool PAIR = false, bool MN = false>// PUSH: the epilogue that stores into the all-reduce slots is compiled in
__global__ void __launch_bounds__(TC_THREADS) gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_a,
                                                              const __grid_constant__ CUtensorMap tmap_b, const TcArgs a) {
    constexpr uint32_t A_BYTES = TC_BM * TC_BK * 2, B_BYTES = (PAIR ? BN / 2 : BN) * TC_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr uint32_t ROWS = PAIR ? 2 * TC_BM : TC_BM;// rows of a tile
    constexpr bool MN_A = MN && BN <= 64, MN_B = MN && BN > 64;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;// 0 = the CTA that issues the products
    const uint32_t S = PAIR ? 1u : a.ksplit, part = S > 1 ? cluster_ctarank() : 0u;
    const uint32_t unit = PAIR ? blockIdx.x >> 1 : blockIdx.x / S, units = PAIR ? gridDim.x >> 1 : gridDim.x / S;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // the swizzled tiles need 1024-byte alignment
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t *recv = smem + STAGES * STAGE_BYTES;// [2][sender][4-column group][128 rows][4] fp32
    constexpr uint32_t RECV_BYTES = tc_recv_bytes(BN);
    uint64_t *full = reinterpret_cast<uint64_t *>(recv + 2 * RECV_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *acc_full = empty + STAGES; // [2]
    uint64_t *acc_empty = acc_full + 2;  // [2]
    uint64_t *recv_full = acc_empty + 2; // [2]
    uint64_t *recv_free = recv_full + 2; // [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(recv_free + 2);
    int *failed = reinterpret_cast<int *>(tmem_slot + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t m_tiles = (a.m + ROWS - 1) / ROWS, n_tiles = (a.n + BN - 1) / BN, tiles = m_tiles * n_tiles;
    const uint32_t kblocks = (a.k + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], PAIR ? 8 : 4);// one arrival per epilogue warp (pair mode: of both CTAs, on the even CTA's barrier)
            mbar_init(&recv_full[b], 4 * S);       // one per epilogue warp of every CTA of the cluster
            mbar_init(&recv_free[b], 4 * S);
        }
        *failed = 0;
        fence_mbar_init();
    }
    if (warp == 5) {
        if constexpr (PAIR) {
            tmem_alloc_pair(tmem_slot, 2 * BN);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(tmem_slot, 2 * BN);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();// the partner's barriers are initialised before anything arrives on them
    if (S > 1) cluster_arrive();       // the same; waited for where the first arrival is made
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Programmatic dependent launch: everything up to here, and the first stages of a weight operand, overlap the previous
    // kernel of the stream; each role waits for that kernel right before it first touches memory the kernel may write.
    pdl_launch_dependents();

    if (warp == 4) {
        if (lane == 0) {
            uint32_t it = 0, pre = 0;
            // B tile of column tile nt: BN consecutive rows of B, or (SiLU-gate form) 128 gate rows and their 128 up rows
            auto load_b = [&](uint8_t *dst, uint32_t kb, uint32_t nt, uint64_t *bar) {
                if constexpr (MN_B) {
#pragma unroll
                    for (uint32_t c = 0; c < BN / 64; ++c) tma_load_2d(dst + c * TC_MN_BLOCK, &tmap_b, nt * BN + c * 64, kb * TC_BK, bar);
                } else if (BN == 256 && a.swiglu) {
                    tma_load_2d(dst, &tmap_b, kb * TC_BK, nt * 128, bar);
                    tma_load_2d(dst + 128 * TC_BK * 2, &tmap_b, kb * TC_BK, a.swiglu + nt * 128, bar);
                } else {
                    tma_load_2d(dst, &tmap_b, kb * TC_BK, nt * BN, bar);
                }
            };
            // A tile of row tile mt: 128 consecutive rows of A, or (SiLU-gate form with the weights on the A side) 64 gate rows
            // and their 64 up rows: two boxes of a 64-row tensor map, one behind the other
            auto load_a = [&](uint8_t *dst, uint32_t kb, uint32_t mt, uint64_t *bar) {
                if constexpr (MN_A) {
#pragma unroll
                    for (uint32_t c = 0; c < TC_BM / 64; ++c) tma_load_2d(dst + c * TC_MN_BLOCK, &tmap_a, mt * TC_BM + c * 64, kb * TC_BK, bar);
                } else if (BN <= 64 && a.swiglu) {
                    tma_load_2d(dst, &tmap_a, kb * TC_BK, mt * 64, bar);
                    tma_load_2d(dst + 64 * TC_BK * 2, &tmap_a, kb * TC_BK, a.swiglu + mt * 64, bar);
                } else {
                    tma_load_2d(dst, &tmap_a, kb * TC_BK, mt * TC_BM, bar);
                }
            };
            TcWalk walk;
            walk.init(tiles, kblocks, unit, units, part, S);
            if (!PAIR && a.early) {
                // weight tiles of this CTA's first segment go in flight before the wait; their partner tiles follow after it
                TcWalk peek = walk;
                if (peek.next()) {
                    uint32_t mt, nt;
                    tile_coords(peek.tile, m_tiles, n_tiles, mt, nt, a.group_m);
                    for (uint32_t kb = walk.kb0; kb < walk.kb1 && pre < STAGES; ++kb, ++pre) {
                        mbar_arrive_expect_tx(&full[pre], STAGE_BYTES);
                        uint8_t *st = smem + pre * STAGE_BYTES;
                        if (a.early == 1) load_a(st, kb, mt, &full[pre]);
                        else
                            load_b(st + A_BYTES, kb, nt, &full[pre]);
                    }
                }
            }
            pdl_wait();
            bool good = true;
            while (good && walk.next()) {
                uint32_t mt, nt;
                tile_coords(walk.tile, m_tiles, n_tiles, mt, nt, a.group_m);
                for (uint32_t kb = walk.kb0; kb < walk.kb1; ++kb, ++it) {
                    const uint32_t s = it % STAGES, ph = (it / STAGES) & 1u;
                    uint8_t *st = smem + s * STAGE_BYTES;
                    if (it < pre) {// stage armed and half filled above
                        if (a.early == 1) load_b(st + A_BYTES, kb, nt, &full[s]);
                        else
                            load_a(st, kb, mt, &full[s]);
                        continue;
                    }
                    if (!mbar_wait(&empty[s], ph ^ 1u)) {
                        *failed = 1;
                        good = false;
                        break;
                    }
                    if constexpr (PAIR) {
                        // both CTAs' bytes are counted on the even CTA's barrier, which its producer arms for the two of them
                        const uint32_t bar = cluster_map(&full[s], 0);
                        if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * STAGE_BYTES);
                        tma_load_2d_pair(st, &tmap_a, kb * TC_BK, (mt * 2 + rank) * TC_BM, bar);
                        const uint32_t brow = a.swiglu ? (rank ? a.swiglu + nt * 128 : nt * 128) : nt * BN + rank * (BN / 2);
                        if constexpr (MN_B) {
#pragma unroll
                            for (uint32_t c = 0; c < BN / 128; ++c)
                                tma_load_2d_pair(st + A_BYTES + c * TC_MN_BLOCK, &tmap_b, brow + c * 64, kb * TC_BK, bar);
                        } else {
                            tma_load_2d_pair(st + A_BYTES, &tmap_b, kb * TC_BK, brow, bar);
                        }
                        continue;
                    }
                    mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
                    load_a(st, kb, mt, &full[s]);
                    load_b(st + A_BYTES, kb, nt, &full[s]);
                }
            }
            // a wait ran out: the copies in flight land before the block may go
            if (!PAIR && !good)
                for (uint32_t j = it < STAGES ? 0 : it - STAGES; j < it; ++j) mbar_wait(&full[j % STAGES], (j / STAGES) & 1u);
        }
    } else if (warp == 5) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = instr_desc(a.is_bf16, ROWS, BN) | (MN_A ? 1u << 15 : 0u) | (MN_B ? 1u << 16 : 0u);
            uint32_t it = 0, local = 0;
            bool ok = true;
            TcWalk walk;
            walk.init(tiles, kblocks, unit, units, part, S);
            for (; ok && walk.next(); ++local) {
                const uint32_t buf = local & 1u, kb0 = walk.kb0, kb1 = walk.kb1;
                if (!mbar_wait(&acc_empty[buf], ((local >> 1) & 1u) ^ 1u)) {
                    *failed = 4;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (uint32_t kb = kb0; kb < kb1; ++kb, ++it) {
                    const uint32_t s = it % STAGES, ph = (it / STAGES) & 1u;
                    if (!mbar_wait(&full[s], ph)) {
                        *failed = 2;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < TC_BK / 16; ++kk) {
                        const uint64_t ad = MN_A ? smem_desc_sw128_mn(a_addr + kk * 2048, TC_MN_BLOCK) : smem_desc_sw128(a_addr + kk * 32);
                        const uint64_t bd = MN_B ? smem_desc_sw128_mn(b_addr + kk * 2048, TC_MN_BLOCK) : smem_desc_sw128(b_addr + kk * 32);
                        if constexpr (PAIR) tc_mma_f16_pair(d_tmem, ad, bd, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
                        else
                            tc_mma_f16(d_tmem, ad, bd, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
                    }
                    // frees the stage once these MMAs have read it (pair mode: in both CTAs)
                    if constexpr (PAIR) tc_commit_pair(&empty[s], 3);
                    else
                        tc_commit(&empty[s]);
                }
                // this tile's accumulator is complete when it arrives
                if constexpr (PAIR) tc_commit_pair(&acc_full[buf], 3);
                else
                    tc_commit(&acc_full[buf]);
            }
        }
    } else {
        // ---- epilogue warps 0..3: TMEM lanes [32*warp, 32*warp + 32) = tile rows ----
        pdl_wait();// C and Y may still be in use by the previous kernel
        T *Y = static_cast<T *>(a.Y);
        const T *C = static_cast<const T *>(a.C);
        const bool c_rowmajor = C && a.c_col_stride == 1 && (a.c_row_stride % 8) == 0 && (reinterpret_cast<uintptr_t>(C) & 15u) == 0;// 16-byte loads
        if (S > 1) cluster_wait();
        // the all-reduce call this product feeds: its number stays put until the receiving kernel behind this one has run
        uint32_t ar_flag_v = 0;
        unsigned ar_q = 0;
        if constexpr (PUSH) {
            const unsigned long long seq = *reinterpret_cast<const volatile unsigned long long *>(a.ar.mine);
            ar_flag_v = ar_flag(seq), ar_q = static_cast<unsigned>(seq & 1ull);
        }
        // SiLU gate with the weights on the A side: tile rows [0, 64) are gate rows, [64, 128) their up rows; the up half hands
        // its values to the gate half through this buffer
        constexpr int UPW = BN <= 64 ? BN : 1;
        __shared__ float s_up[BN <= 64 ? 64 : 1][UPW + 1];
        // v[0..W) = this thread's row, columns c_first ..; every one of the 128 epilogue threads calls it
        auto swiglu_rows = [&](const float *v, auto width, uint32_t mt, uint32_t c_first) {
            constexpr int W = decltype(width)::value;
            const uint32_t trow = warp * 32 + lane, f = a.swiglu;
            if (trow >= 64) {
#pragma unroll
                for (int j = 0; j < W; ++j) s_up[trow - 64][j] = v[j];
            }
            asm volatile("bar.sync 2, 128;" ::: "memory");
            if (trow < 64) {
                const uint32_t feat = mt * 64 + trow;
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const uint32_t tok = c_first + j;
                    if (feat < f && tok < a.n) {
                        const float g = a.alpha * v[j], u = a.alpha * s_up[trow][j];
                        Y[static_cast<uint64_t>(tok) * f + feat] = Num<T>::from_f(g / (1.f + expf(-g)) * u);
                    }
                }
            }
            asm volatile("bar.sync 2, 128;" ::: "memory");
        };
        // QKV split + rotation + cache append with the weights on the A side: a tile of 128 rows is one head (head_dim 128), tile
        // rows i and i + 64 are a rotation pair.  The upper half hands its values to the lower half, which rotates the pair with
        // the token's angle and stores both results: into the q buffer, or into the K / V cache row of the token's position
        // (checked against the layout; a bad position or block id skips the store and raises the index error).
        auto rope_rows = [&](const float *v, auto width, uint32_t mt, uint32_t c_first) {
            constexpr int W = decltype(width)::value;
            const uint32_t trow = warp * 32 + lane, nkv = a.kv.n_kv_heads;
            if (trow >= 64) {
#pragma unroll
                for (int j = 0; j < W; ++j) s_up[trow - 64][j] = v[j];
            }
            asm volatile("bar.sync 2, 128;" ::: "memory");
            if (trow < 64 && mt < a.nq + 2 * nkv) {
                const uint32_t gh = mt;
                const bool is_q = gh < a.nq, rotate = gh < a.nq + nkv;
                const uint32_t kvh = is_q ? 0u : (rotate ? gh - a.nq : gh - a.nq - nkv);
                const float inv_freq = exp2f(-a.log2_theta * (2.0f * static_cast<float>(trow) / 128.0f));
#pragma unroll 1
                for (int j = 0; j < W; ++j) {
                    const uint32_t tok = c_first + j;
                    if (tok >= a.n) break;
                    float lo = a.alpha * v[j], hi = a.alpha * s_up[trow][j];
                    const int64_t p = a.pos[tok];
                    if (rotate) {
                        float sn, cs;
                        sincosf(static_cast<float>(p) * inv_freq, &sn, &cs);
                        const float r0 = lo * cs - hi * sn, r1 = hi * cs + lo * sn;
                        lo = r0, hi = r1;
                    }
                    T *dst;
                    if (is_q) {
                        dst = static_cast<T *>(a.q_out) + (static_cast<uint64_t>(tok) * a.nq + gh) * 128u;
                    } else {
                        if (!kv_pos_ok(p, a.kv, a.table != nullptr)) {
                            s_tc_index_error = 1;
                            continue;
                        }
                        const uint32_t seq = a.tokens_per_seq > 1 ? tok / a.tokens_per_seq : tok;
                        uint64_t cache_row;
                        uint32_t head_pitch;
                        if (a.table) {
                            const uint32_t page = a.kv.page_size;
                            const int32_t blk = a.table[static_cast<uint64_t>(seq) * a.kv.max_blocks_per_seq + static_cast<uint32_t>(p) / page];
                            if (!kv_block_ok(blk, a.kv)) {
                                s_tc_index_error = 1;
                                continue;
                            }
                            cache_row = (static_cast<uint64_t>(blk) * nkv * page + static_cast<uint32_t>(p) % page) * 128u;
                            head_pitch = page * 128u;
                        } else {
                            cache_row = (static_cast<uint64_t>(seq) * nkv * a.kv.max_seq + static_cast<uint64_t>(p)) * 128u;
                            head_pitch = a.kv.max_seq * 128u;
                        }
                        dst = static_cast<T *>(rotate ? a.kc : a.vc) + cache_row + static_cast<uint64_t>(kvh) * head_pitch;
                    }
                    dst[trow] = Num<T>::from_f(lo);
                    dst[trow + 64] = Num<T>::from_f(hi);
                }
            }
            asm volatile("bar.sync 2, 128;" ::: "memory");
        };
        uint32_t local = 0;
        TcWalk walk;
        walk.init(tiles, kblocks, unit, units, part, S);
        // hands an accumulator buffer back to the thread that issues the products (pair mode: in the even CTA)
        auto release_acc = [&](uint32_t buf) {
            if constexpr (PAIR) mbar_arrive_cluster(cluster_map(&acc_empty[buf], 0));
            else
                mbar_arrive(&acc_empty[buf]);
        };
        // Epilogue of columns [c_first, c_first + W) of this thread's row in the skinny forms, from their finished sums
        auto finish = [&](const float *v, auto width, uint32_t mt, uint32_t row, uint32_t c_first) {
            constexpr int W = decltype(width)::value;
            if constexpr (PUSH) {
#pragma unroll
                for (int j = 0; j < W; ++j)
                    if (c_first + j < a.n) tc_push_value<T>(a, ar_flag_v, ar_q, row, c_first + j, a.alpha * v[j], row < a.m, lane);
            } else if (a.swiglu) {
                swiglu_rows(v, width, mt, c_first);
            } else if (a.rope) {
                rope_rows(v, width, mt, c_first);
            } else if (row < a.m) {
                // all of C before the first store: behind the stores of Y, which may be the same memory as far as the compiler knows,
                // each load would wait for its own round trip
                float add[W];
#pragma unroll
                for (int j = 0; j < W; ++j)
                    add[j] = C && c_first + j < a.n ? Num<T>::to_f(C[static_cast<uint64_t>(row) * a.c_row_stride + static_cast<uint64_t>(c_first + j) * a.c_col_stride]) : 0.f;
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    if (c_first + j < a.n) {
                        float o = a.alpha * v[j];
                        if (C) o += a.beta * add[j];
                        Y[static_cast<uint64_t>(row) * a.y_row_stride + static_cast<uint64_t>(c_first + j) * a.y_col_stride] = Num<T>::from_f(o);
                    }
                }
            }
        };
        // W columns per CTA of the cluster, WC of them at a time, from the receive buffer
        auto finish_received = [&](auto chunk, const uint8_t *from, uint32_t W, uint32_t mt, uint32_t row, uint32_t c_first) {
            constexpr int WC = decltype(chunk)::value;
            const uint32_t trow = warp * 32 + lane;
            for (uint32_t c = 0; c < W; c += WC) {
                if (c_first + c >= a.n) break;// the same for every thread of the block
                float v[WC];
#pragma unroll
                for (int j = 0; j < WC; ++j) v[j] = 0.f;
                for (uint32_t src = 0; src < S; ++src) {
#pragma unroll
                    for (int g = 0; g < WC / 4; ++g) {
                        const float4 x = *reinterpret_cast<const float4 *>(from + (((src * W + c) / 4 + g) * 128 + trow) * 16);
                        v[4 * g] += x.x, v[4 * g + 1] += x.y, v[4 * g + 2] += x.z, v[4 * g + 3] += x.w;
                    }
                }
                finish(v, chunk, mt, row, c_first + c);
            }
        };
        bool ok = true;// after a wait that ran out nothing is waited for any more, but every barrier of the block is still met
        for (; walk.next(); ++local) {
            uint32_t mt, nt;
            tile_coords(walk.tile, m_tiles, n_tiles, mt, nt, a.group_m);
            const uint32_t buf = local & 1u, phase = (local >> 1) & 1u, m0 = PAIR ? (mt * 2 + rank) * TC_BM : mt * TC_BM, n0 = nt * BN;
            const uint32_t row = m0 + warp * 32 + lane;
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], phase) ? 1 : 0);
            if (!ok) *failed = 3;
            tc_fence_after();
            if constexpr (BN <= 64) {
                if (S > 1) {
                    const uint32_t W = BN / S, shift = __ffs(W) - 1, trow = warp * 32 + lane;// a power of two
                    ok = ok && __all_sync(0xffffffffu, mbar_wait_cluster(&recv_free[buf], phase ^ 1u) ? 1 : 0);
                    uint8_t *box = recv + buf * RECV_BYTES;
#pragma unroll 1
                    for (int c0 = 0; c0 < BN; c0 += 32) {
                        uint32_t r[32];
                        tmem_ld_32x32(tmem_base + buf * BN + ((warp * 32u) << 16) + c0, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int g = 0; g < 8; ++g) {
                            const uint32_t c = c0 + 4 * g, to = c >> shift;
                            if (n0 + c < a.n)
                                st_cluster_v4(cluster_map(box + (((part * W + (c & (W - 1))) / 4) * 128 + trow) * 16, to), r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
                        }
                    }
                    tc_fence_before();
                    fence_cluster();
                    __syncwarp();
                    if (lane == 0) release_acc(buf);
                    if (lane < S) mbar_arrive_cluster(cluster_map(&recv_full[buf], lane));
                    ok = ok && __all_sync(0xffffffffu, mbar_wait_cluster(&recv_full[buf], phase) ? 1 : 0);
                    if (!ok) *failed = 5;
                    if (W >= 8) finish_received(std::integral_constant<int, 8>{}, box, W, mt, row, n0 + part * W);
                    else
                        finish_received(std::integral_constant<int, 4>{}, box, W, mt, row, n0 + part * W);
                    __syncwarp();
                    if (lane < S) mbar_arrive_cluster(cluster_map(&recv_free[buf], lane));
                    continue;
                }
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld_32x32(tmem_base + buf * BN + ((warp * 32u) << 16) + c0, r);
                    tmem_ld_wait();
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                    finish(v, std::integral_constant<int, 32>{}, mt, row, n0 + c0);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) release_acc(buf);
                continue;
            }
            if constexpr (BN == 256) {
                if (a.swiglu) {
                    // accumulator columns [0, 128) = gate, [128, 256) = up of output columns n0/2 .. n0/2 + 127
                    const uint32_t j0 = (n0 / 256) * 128, f = a.n / 2;
#pragma unroll 1
                    for (int c0 = 0; c0 < 128; c0 += 32) {
                        uint32_t gt[32], up[32];
                        const uint32_t taddr = tmem_base + buf * BN + ((warp * 32u) << 16) + c0;
                        tmem_ld_32x32(taddr, gt);
                        tmem_ld_32x32(taddr + 128, up);
                        tmem_ld_wait();
                        if (row < a.m && j0 + c0 < f) {
                            T *dst = Y + static_cast<uint64_t>(row) * f + j0 + c0;
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                float o[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) {
                                    const float g = a.alpha * __uint_as_float(gt[j + e]), u = a.alpha * __uint_as_float(up[j + e]);
                                    o[e] = g / (1.f + expf(-g)) * u;
                                }
                                Vec16<T> v;
                                v.pack(o);
                                v.store(dst + j);
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) release_acc(buf);
                    continue;
                }
            }
            if constexpr (BN >= 128) {
                if (a.rope) {
                    // this thread's token: rotate the pairs (i, i + 64) of every q and k head of the tile, copy v heads, and
                    // write each head straight to its destination (q buffer or KV cache, contiguous or paged)
                    const bool live = row < a.m;
                    const int64_t p = live ? a.pos[row] : 0;
                    const uint32_t seq = a.tokens_per_seq > 1 ? row / a.tokens_per_seq : row, nkv = a.kv.n_kv_heads;
                    uint64_t cache_row = 0;// element offset of (seq, kv head 0, p) in a cache, without the head term
                    uint32_t head_pitch = 0;
                    bool cache_ok = live;// false: this token's k / v heads are not stored
                    if (live && !kv_pos_ok(p, a.kv, a.table != nullptr)) {
                        s_tc_index_error = 1;
                        cache_ok = false;
                    }
                    if (cache_ok) {
                        if (a.table) {
                            const uint32_t page = a.kv.page_size;
                            const int32_t blk = a.table[static_cast<uint64_t>(seq) * a.kv.max_blocks_per_seq + static_cast<uint32_t>(p) / page];
                            if (!kv_block_ok(blk, a.kv)) {
                                s_tc_index_error = 1;
                                cache_ok = false;
                            }
                            cache_row = (static_cast<uint64_t>(cache_ok ? blk : 0) * nkv * page + static_cast<uint32_t>(p) % page) * 128u;
                            head_pitch = page * 128u;
                        } else {
                            cache_row = (static_cast<uint64_t>(seq) * nkv * a.kv.max_seq + static_cast<uint64_t>(p)) * 128u;
                            head_pitch = a.kv.max_seq * 128u;
                        }
                    }
#pragma unroll 1
                    for (int pc = 0; pc < 2; ++pc) {
                        float cs[32], sn[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float inv_freq = exp2f(-a.log2_theta * (2.0f * static_cast<float>(pc * 32 + j) / 128.0f));
                            sincosf(static_cast<float>(p) * inv_freq, &sn[j], &cs[j]);
                        }
#pragma unroll 1
                        for (int hh = 0; hh < BN / 128; ++hh) {
                            const uint32_t col0 = n0 + hh * 128;
                            if (col0 >= a.n) break;
                            uint32_t lo[32], hi[32];
                            const uint32_t taddr = tmem_base + buf * BN + ((warp * 32u) << 16) + hh * 128 + pc * 32;
                            tmem_ld_32x32(taddr, lo);
                            tmem_ld_32x32(taddr + 64, hi);
                            tmem_ld_wait();
                            if (!live) continue;
                            const uint32_t gh = col0 / 128;
                            T *dst;
                            if (gh < a.nq) {
                                dst = static_cast<T *>(a.q_out) + (static_cast<uint64_t>(row) * a.nq + gh) * 128u;
                            } else {
                                if (!cache_ok) continue;
                                const bool is_k = gh < a.nq + nkv;
                                const uint32_t kvh = is_k ? gh - a.nq : gh - a.nq - nkv;
                                dst = static_cast<T *>(is_k ? a.kc : a.vc) + cache_row + static_cast<uint64_t>(kvh) * head_pitch;
                            }
                            const bool rotate = gh < a.nq + nkv;
#pragma unroll
                            for (int j = 0; j < 32; j += 8) {
                                float fl[8], fh[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e) {
                                    const float x0 = a.alpha * __uint_as_float(lo[j + e]), x1 = a.alpha * __uint_as_float(hi[j + e]);
                                    fl[e] = rotate ? x0 * cs[j + e] - x1 * sn[j + e] : x0;
                                    fh[e] = rotate ? x1 * cs[j + e] + x0 * sn[j + e] : x1;
                                }
                                Vec16<T> vl, vh;
                                vl.pack(fl), vh.pack(fh);
                                vl.store(dst + pc * 32 + j);
                                vh.store(dst + 64 + pc * 32 + j);
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) release_acc(buf);
                    continue;
                }
            }
            // 32 columns at a time.  What is added from C is fetched ahead of the accumulator (behind the stores of the columns before,
            // which may be the same memory as far as the compiler knows, every load would wait for its own round trip): one residual
            // tile of 128 x 256 took 12 us longer than the plain product with a load in front of every store.
            // Rows of a multiple of 8 columns end between two 16-byte pieces, which are then there or not, and past the last column there is
            // nothing to do: straight-line code for single columns costs more than its stores when it comes from a cold instruction cache
            // (128 x 64 x 64 7.5 us with it and 2.9 without, 1945 x 8040 x 312 33.4 and 24.4).
            const bool rows_wide = a.y_col_stride == 1 && (a.n % 8) == 0 && (a.y_row_stride % 8) == 0 && (!C || c_rowmajor);
            Vec16<T> cnext[4];
            auto fetch_c = [&](uint32_t col0) {
                if (C && rows_wide && row < a.m) {
                    const T *csrc = C + static_cast<uint64_t>(row) * a.c_row_stride + col0;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (col0 + 8 * j < a.n) cnext[j].load(csrc + 8 * j);
                }
            };
            auto store_columns = [&](const float (&r)[32], const Vec16<T> (&cv)[4], uint32_t col0) {
                if (row >= a.m) return;
                if (rows_wide) {
                    // contiguous 64-byte run of this thread's row: four 16-byte stores
                    T *dst = Y + static_cast<uint64_t>(row) * a.y_row_stride + col0;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        if (col0 + j >= a.n) break;
                        float f[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) f[e] = a.alpha * r[j + e];
                        if (C) {
                            float cf[8];
                            cv[j / 8].unpack(cf);
#pragma unroll
                            for (int e = 0; e < 8; ++e) f[e] += a.beta * cf[e];
                        }
                        Vec16<T> v;
                        v.pack(f);
                        v.store(dst + j);
                    }
                } else {
                    float add[32];
                    if (C) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const uint32_t col = col0 + j;
                            add[j] = col < a.n ? Num<T>::to_f(C[static_cast<uint64_t>(row) * a.c_row_stride + static_cast<uint64_t>(col) * a.c_col_stride]) : 0.f;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const uint32_t col = col0 + j;
                        if (col < a.n) {
                            float v = a.alpha * r[j];
                            if (C) v += a.beta * add[j];
                            Y[static_cast<uint64_t>(row) * a.y_row_stride + static_cast<uint64_t>(col) * a.y_col_stride] = Num<T>::from_f(v);
                        }
                    }
                }
            };
            if constexpr (BN > 64 && !PAIR) {
                if (S > 1) {
                    const uint32_t W = BN / S, shift = __ffs(W) - 1, trow = warp * 32 + lane, mine = n0 + part * W;// W: 32, 64 or 128
                    if (lane < S) mbar_arrive_cluster(cluster_map(&recv_free[0], lane));// this CTA's products are done: its ring may be written
                    fetch_c(mine);
                    ok = ok && __all_sync(0xffffffffu, mbar_wait_cluster(&recv_free[0], 0) ? 1 : 0);
                    if (!ok) {
                        *failed = 5;
                        continue;// nothing is stored into a ring that may still be in use
                    }
#pragma unroll 1
                    for (int c0 = 0; c0 < BN; c0 += 32) {
                        uint32_t r[32];
                        tmem_ld_32x32(tmem_base + buf * BN + ((warp * 32u) << 16) + c0, r);
                        tmem_ld_wait();
                        if (n0 + c0 >= a.n) break;
                        const uint32_t to = cluster_map(smem + ((part * W + (c0 & (W - 1))) / 4 * 128 + trow) * 16, c0 >> shift);
#pragma unroll
                        for (int g = 0; g < 8; ++g) st_cluster_v4(to + g * 2048, r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
                    }
                    fence_cluster();
                    __syncwarp();
                    if (lane < S) mbar_arrive_cluster(cluster_map(&recv_full[0], lane));
                    ok = ok && __all_sync(0xffffffffu, mbar_wait_cluster(&recv_full[0], 0) ? 1 : 0);
                    if (!ok) *failed = 5;
                    for (uint32_t c = 0; c < W && mine + c < a.n; c += 32) {
                        Vec16<T> cv[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) cv[j] = cnext[j];
                        if (c + 32 < W) fetch_c(mine + c + 32);
                        float v[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = 0.f;
                        for (uint32_t src = 0; src < S; ++src) {
                            const float4 *from = reinterpret_cast<const float4 *>(smem) + ((src * W + c) / 4 * 128 + trow);
#pragma unroll
                            for (int g = 0; g < 8; ++g) {
                                const float4 x = from[g * 128];
                                v[4 * g] += x.x, v[4 * g + 1] += x.y, v[4 * g + 2] += x.z, v[4 * g + 3] += x.w;
                            }
                        }
                        store_columns(v, cv, mine + c);
                    }
                    continue;
                }
            }
            fetch_c(n0);
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                if (n0 + c0 >= a.n) break;// the same for every thread
                uint32_t r[32];
                Vec16<T> cv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) cv[j] = cnext[j];
                if (c0 + 32 < BN) fetch_c(n0 + c0 + 32);
                tmem_ld_32x32(tmem_base + buf * BN + ((warp * 32u) << 16) + c0, r);
                tmem_ld_wait();
                float v[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                store_columns(v, cv, n0 + c0);
            }
            // hand the accumulator buffer back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) release_acc(buf);
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();// the partner has read its accumulators and received every arrival meant for it
    if (S > 1) {
        if (warp >= 4) cluster_wait();// of the arrival at the start
        cluster_sync();// every store and arrival meant for this CTA's shared memory has been made
    }
    if (warp == 5) {
        tc_fence_after();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 2 * BN);
        else
            tmem_dealloc(tmem_base, 2 * BN);
    }
    if (threadIdx.x == 0 && *failed) atomicExch(&s_tc_error, *failed);
}

// ---- host -----------------------------------------------------------------------------------------------------
// rows x k matrix, K-major (row stride = ld elements); box = 64 (k) x box_rows, 128-byte swizzle
static bool make_map(CUtensorMap *map, const void *base, int is_bf16, uint64_t rows, uint64_t k, uint64_t ld, uint32_t box_rows) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {k, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {TC_BK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A K-major matrix W[rows, k] seen as (64 columns, rows, k / 64 column blocks): one request then loads a box of box_rows rows
// x box_blocks column blocks, stored [block][row][128 bytes] with the 128-byte swizzle (the streaming skinny kernel's unit).
bool tma_encode_rows_by_blocks(void *map, const void *base, int is_bf16, uint64_t rows, uint64_t k, uint32_t box_rows, uint32_t box_blocks) {
    EncodeFn fn = encode_fn();
    if (!fn || k % 64 != 0) return false;
    const cuuint64_t dims[3] = {64, rows, k / 64};
    const cuuint64_t strides[2] = {k * 2, 128};
    const cuuint32_t box[3] = {64, box_rows, box_blocks};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(static_cast<CUtensorMap *>(map), is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
              const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A weight matrix stored [k, n] as the kernel's MN-major operand: boxes of 64 columns x 64 k-rows
static bool make_map_mn(CUtensorMap *map, const void *base, int is_bf16, uint64_t k, uint64_t n) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {n, k};
    const cuuint64_t strides[1] = {n * 2};
    const cuuint32_t box[2] = {64, TC_BK};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool gemm_tc_supported(const rg_mat_mul_params *p, const void *const *in, void *const *out) {
    if (p->dtype != RG_FP16 && p->dtype != RG_BF16) return false;
    if (p->trans_a) return false;
    if (!p->trans_b) {
        if (p->n % 8 != 0) return false;// rows of an MN-major B start on 16 bytes
        // a batch is one launch per matrix here and one launch altogether on the CUDA cores (~15 TFLOP/s), which keep the batches of
        // products that would take them less than about 9 us each
        if (p->batch > 1 && static_cast<uint64_t>(p->m) * p->n * p->k < (1ull << 26)) return false;
    }
    if (p->k % 8 != 0 || p->k < 64) return false;
    if (!aligned16(in[0]) || !aligned16(in[1]) || !aligned16(out[0])) return false;
    if (p->batch > 1 && ((p->stride_a % 8) || (p->stride_b % 8) || (p->stride_y % 8))) return false;
    // worth a tensor-core launch only when there is a tile's worth of work
    if (static_cast<uint64_t>(p->m) * p->n < 64ull * 64ull) return false;
    return encode_fn() != nullptr;
}

// Skinny products (the tokens on the instruction's N side): up to 64 tokens against at least one tile of weight rows
static bool tc_swapped(const rg_mat_mul_params *p) { return p->m <= 64 && p->n >= 128; }
// CTAs of a cluster that share a tile: 1, 2, 4 or 8, whichever the model below says is done first.  A k-block (16 KiB of weights) takes an
// SM 0.345 us when all of them stream and never less than 0.31; every round of tiles pays for what its exchange does not hide
// behind the next tile's stream (about 4 us less 0.12 per k-block); launch and drain 3 us.  Measured at 8 tokens with
// 1 / 2 / 4 / 8 CTAs: 4096 x 4096 21.4 / 13.6 / 11.7 / 14.3 us (model 22.8 / 13.1 / 10.1 / 14.4), 22016 x 4096 45.7 / 36.5 / 41.5 / 54.1 us,
// 32000 x 1024 14.5 / 20.1 / 31.6 / 57.2 us, 57344 x 8192 174 / 156 / 151 / 193 us, 8192 x 28672 130 / 75 / 75 / 87 us.
static uint32_t tc_ksplit(uint32_t tiles, uint32_t kblocks, const int (&clusters)[4]) {
    const float sms = static_cast<float>(sm_count());
    uint32_t best = 1;
    float best_us = 1e30f;
    for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t s = 1u << i, c = static_cast<uint32_t>(clusters[i]);
        if (c == 0 || (s > 1 && s > kblocks)) continue;
        const float rounds = static_cast<float>((tiles + c - 1) / c), busy = static_cast<float>((tiles < c ? tiles : c) * s) / sms;
        const float kb = static_cast<float>((kblocks + s - 1) / s), kb_us = 0.345f * busy > 0.31f ? 0.345f * busy : 0.31f;
        float seen = s > 1 ? 4.0f - 0.12f * kb : 0.f;
        if (seen < 0.f) seen = 0.f;
        const float us = rounds * (kb * kb_us + seen);
        if (us < best_us) best_us = us, best = s;
    }
    return best;
}

// The wide forms: clusters share a tile only where every tile has one to itself, at least four k-blocks and 32 columns per CTA.  Shared
// memory fills at 64 bytes a cycle, which makes a k-block 0.33 us (128 columns) or 0.43 us (256); launch and drain 4 us, exchange 3 us.
static float tc_wide_us(uint32_t tiles, uint32_t kblocks, uint32_t bn, uint32_t s, uint32_t slots) {
    const float kb_us = bn > 128 ? 0.43f : 0.33f, crowd = bn > 128 ? 0.57f : 0.33f;// 144 CTAs of the large tile share what L2 delivers
    const uint32_t busy = tiles * s < slots ? tiles * s : slots;
    const float us = busy * 2 > slots ? kb_us + (crowd - kb_us) * (2.f * busy / slots - 1.f) : kb_us;
    return 4.f + static_cast<float>((static_cast<uint64_t>(tiles) * s + slots - 1) / slots) * static_cast<float>((kblocks + s - 1) / s) * us + (s > 1 ? 3.f : 0.f);
}
static uint32_t tc_ksplit_wide(uint32_t tiles, uint32_t kblocks, uint32_t bn, const int (&clusters)[4]) {
    uint32_t best = 1;
    float best_us = tc_wide_us(tiles, kblocks, bn, 1, static_cast<uint32_t>(sm_count()));
    for (uint32_t i = 1; i < 4; ++i) {
        const uint32_t s = 1u << i;
        if (s * 4 > kblocks || s * 32 > bn || static_cast<int>(tiles) > clusters[i]) continue;
        const float us = tc_wide_us(tiles, kblocks, bn, s, static_cast<uint32_t>(sm_count()));
        if (us < best_us) best_us = us, best = s;
    }
    return best;
}

// Measured on one rank's share of a tensor-parallel-8 decode step (16 tokens, 80 layers, one GPU, no exchange; 9.55 ms):
// 5 stages for the up-to-32-token products, so that a CTA of the next kernel fits beside one of this kernel and fetches its
// first weight tiles early: 10.55 ms; 10 stages: 9.57 ms; asking L2 for 16 / 48 further weight tiles of the CTA's run before the
// dependency wait (cp.async.bulk.prefetch.tensor): 9.62 / 9.69 ms.  None is kept.
// Also measured and not kept, on the 32-token x 22016 x 4096 product (41.3 us = 4.4 TB/s; a TMA-only stream of the same tiles
// from 148 CTAs with 192 KiB in flight reaches 5.8 TB/s): 10 stages (42.1 us); the four k-steps of a k-block into four separate
// accumulators added in the epilogue, so that consecutive instructions do not depend on one another (41.0 us).  Cycle counters:
// the issuing thread spends ~340 cycles per k-block (4 instructions + commit) and waits for data 41 % of the time, the producer
// waits for a free stage 41 % of the time.  Leaving the activation-tile loads out altogether (timing only): 41.3 us.  What is
// left is the fill and drain of the memory pipeline around the dependency on the previous kernel (~10 us per launch): the
// TMA-only stream has no such dependency, so its launches overlap.
// As many clusters of `size` CTAs as the device holds at once (0 where it cannot say)
template<class... K>
static int tc_resident_clusters(void (*kern)(K...), unsigned size, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(sm_count()) / size * size), cfg.blockDim = dim3(TC_THREADS), cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 0) {
        cudaGetLastError();
        n = 0;
    }
    return n;
}
template<class T, int BN, int STAGES, bool PUSH = false, bool MN = false>
static int tc_launch(const CUtensorMap &ma, const CUtensorMap &mb, const TcArgs &a_in, cudaStream_t st) {
    TcArgs a = a_in;
    a.group_m = TC_GROUP_M;
    constexpr size_t smem = STAGES * (TC_BM * TC_BK * 2 + BN * TC_BK * 2) + 2 * tc_recv_bytes(BN) + (2 * STAGES + 8) * 8 + 16 + 1024;
    auto kern = gemm_tc_kernel<T, BN, STAGES, PUSH, false, MN>;
    RG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    // the whole shared-memory carve-out, so that a CTA of the next kernel can sit beside one of this kernel when both fit
    RG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, static_cast<int>(cudaSharedmemCarveoutMaxShared)));
    const uint32_t tiles = ((a.n + BN - 1) / BN) * ((a.m + TC_BM - 1) / TC_BM), sms = static_cast<uint32_t>(sm_count());
    // per device and cluster size 1, 2, 4, 8; asked once (or by every thread that comes before the first answer, which is the same);
    // the entry of size 1 says that the others are there
    static std::atomic<int> clusters[64][4] = {};
    int dev = 0;
    RG_CHECK_CUDA(cudaGetDevice(&dev));
    int here[4] = {static_cast<int>(sms), 0, 0, 0};
    if (dev >= 0 && dev < 64) {
        if (clusters[dev][0].load(std::memory_order_acquire) == 0) {
            for (int i = 3; i >= 1; --i) clusters[dev][i].store(tc_resident_clusters(kern, 1u << i, smem), std::memory_order_relaxed);
            clusters[dev][0].store(static_cast<int>(sms), std::memory_order_release);
        }
        for (int i = 0; i < 4; ++i) here[i] = clusters[dev][i].load(std::memory_order_relaxed);
    }
    const uint32_t kblocks = (a.k + TC_BK - 1) / TC_BK;
    if constexpr (BN <= 64) a.ksplit = tc_ksplit(tiles, kblocks, here);
    else
        a.ksplit = a.rope || a.swiglu ? 1u : tc_ksplit_wide(tiles, kblocks, BN, here);
    if (a.ksplit > 1) {
        const uint32_t c = static_cast<uint32_t>(here[a.ksplit == 2 ? 1 : a.ksplit == 4 ? 2 : 3]);
        RG_CHECK_CUDA(launch_pdl_cluster(kern, dim3((tiles < c ? tiles : c) * a.ksplit), dim3(TC_THREADS), smem, st, a.ksplit, ma, mb, a));
        count_launch();
        return launch_status();
    }
    RG_CHECK_CUDA(launch_pdl(kern, dim3(tiles < sms ? tiles : sms), dim3(TC_THREADS), smem, st, ma, mb, a));
    count_launch();
    return launch_status();
}

// Pair mode: clusters of two CTAs, one 256 x BN tile per pair (B's tensor map has boxes of BN / 2 rows).  RG_B200_GEMM_PAIR=0 keeps
// the single-CTA kernel.
static bool tc_pair_enabled() {
    static const bool on = !(std::getenv("RG_B200_GEMM_PAIR") && std::getenv("RG_B200_GEMM_PAIR")[0] == '0');
    return on;
}
template<class T, bool MN = false>
static int tc_launch_pair(const CUtensorMap &ma, const CUtensorMap &mb, const TcArgs &a_in, cudaStream_t st) {
    constexpr int BN = 256, STAGES = 6;
    TcArgs a = a_in;
    a.group_m = TC_GROUP_M;// of 256-row tiles; measured on 8192 x 12288 x 4096: 4 / 8 / 16 / 32 row tiles per group 577 / 557 / 550 / 605 us
    constexpr size_t smem = STAGES * (TC_BM * TC_BK * 2 + (BN / 2) * TC_BK * 2) + (2 * STAGES + 8) * 8 + 16 + 1024;
    auto kern = gemm_tc_kernel<T, BN, STAGES, false, true, MN>;
    RG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const uint32_t items = ((a.n + BN - 1) / BN) * ((a.m + 2 * TC_BM - 1) / (2 * TC_BM));
    // as many pairs as the device can hold at once (asked once per device; half the SM count where the question fails)
    static std::atomic<int> resident[64] = {};
    int dev = 0;
    RG_CHECK_CUDA(cudaGetDevice(&dev));
    int most = dev >= 0 && dev < 64 ? resident[dev].load(std::memory_order_relaxed) : sm_count() / 2;
    if (most == 0) {
        const int n = tc_resident_clusters(kern, 2, smem);
        most = n > 0 ? n : sm_count() / 2;
        resident[dev].store(most, std::memory_order_relaxed);
    }
    const uint32_t pairs = static_cast<uint32_t>(most);
    const uint32_t grid = 2 * (items < pairs ? items : pairs);
    RG_CHECK_CUDA(launch_pdl_cluster(kern, dim3(grid), dim3(TC_THREADS), smem, st, 2u, ma, mb, a));
    count_launch();
    return launch_status();
}

// Tile of the products of more than 64 tokens: 128 x 256 on single CTAs, 256 x 256 on pairs (512 tokens and more) or 128 x 128, whichever
// tc_wide_us says is done first.  Shared memory fills at 64 bytes a cycle and SM and L2 delivers 10 to 12 TB/s in all, so the
// smaller tile costs more per product; it wins where the large ones leave SMs idle.  128 / 256 columns / pair with residual, the
// first two with the split they get: 333 x 4096 x 4096 26.1 / 22.0 / 29.8 us (30.4 unsplit), 333 x 4096 x 11008 60.5 / 44.3 / 62.9 (70.5),
// 333 x 12288 x 4096 47.8 / 39.8 / 52.9, 128 x 4096 x 4096 15.1 / 17.9 / 29.5, 300 x 1024 x 2752 12.0 / 15.1 / 22.0 (18.0 and 22.3 unsplit),
// 700 x 4096 x 4096 44.7 / 30.9 / 31.6, 2000 x 10240 x 8192 367 / 281 / 256.
enum : int { TC_TILE_128, TC_TILE_256, TC_TILE_PAIR };
static int tc_wide_tile(uint32_t m, uint32_t n, uint32_t k) {
    if (n < 256) return TC_TILE_128;
    const uint32_t sms = static_cast<uint32_t>(sm_count()), kblocks = (k + TC_BK - 1) / TC_BK;
    auto up = [](uint32_t v, uint32_t t) { return (v + t - 1) / t; };
    // clusters that the device is sure to hold at once: one CTA in nine is left over where SMs do not divide evenly
    const int clusters[4] = {static_cast<int>(sms), static_cast<int>(sms / 2), static_cast<int>(sms * 8 / 9 / 4), static_cast<int>(sms * 7 / 9 / 8)};
    auto us = [&](uint32_t bn) {
        const uint32_t tiles = up(m, 128) * up(n, bn);
        return tc_wide_us(tiles, kblocks, bn, tc_ksplit_wide(tiles, kblocks, bn, clusters), sms);
    };
    const float small = us(128), large = us(256);
    if (m >= 512 && tc_pair_enabled()) {
        const uint64_t pairs = static_cast<uint64_t>(up(m, 256)) * up(n, 256);
        const float pair = 4.f + static_cast<float>((pairs + sms / 2 - 1) / (sms / 2)) * static_cast<float>(kblocks) * 0.385f;
        if (pair <= large && pair <= small) return TC_TILE_PAIR;
    }
    return small < large ? TC_TILE_128 : TC_TILE_256;
}

int gemm_tc(const rg_mat_mul_params *p, const void *const *in, void *const *out, cudaStream_t st, bool pairs) {
    if (pairs && !tc_pair_enabled()) return RG_ERR_UNSUPPORTED;
    const int is_bf16 = p->dtype == RG_BF16;
    const size_t es = 2;
    const bool mn = !p->trans_b;
    auto map_b = [&](CUtensorMap *map, const void *base, uint32_t box_rows) {
        return mn ? make_map_mn(map, base, is_bf16, p->k, p->n) : make_map(map, base, is_bf16, p->n, p->k, p->k, box_rows);
    };
    for (uint32_t b = 0; b < p->batch; ++b) {
        const uint8_t *A = static_cast<const uint8_t *>(in[0]) + b * p->stride_a * es;
        const uint8_t *B = static_cast<const uint8_t *>(in[1]) + b * p->stride_b * es;
        uint8_t *Y = static_cast<uint8_t *>(out[0]) + b * p->stride_y * es;
        const uint8_t *C = p->has_bias ? static_cast<const uint8_t *>(in[2]) + b * p->stride_c * es : nullptr;
        TcArgs a = {};
        a.alpha = p->alpha, a.beta = p->beta, a.is_bf16 = is_bf16, a.k = p->k;
        CUtensorMap ma, mb;
        // a skinny activation matrix (m <= 64) goes on the N side of the instruction: D^T[n, m] = W[n,k] X[m,k]^T
        const bool swap = !pairs && tc_swapped(p);
        uint32_t bn;
        if (!swap) {
            const int tile = pairs ? TC_TILE_PAIR : tc_wide_tile(p->m, p->n, p->k);
            bn = tile == TC_TILE_128 ? 128 : 256;
            a.m = p->m, a.n = p->n;
            a.early = (p->flags & RG_MM_B_STATIC) ? 2u : 0u;
            a.Y = Y, a.y_row_stride = p->n, a.y_col_stride = 1;
            a.C = C, a.c_row_stride = p->bias_row_stride, a.c_col_stride = p->bias_col_stride;
            if (tile == TC_TILE_PAIR) {
                if (!make_map(&ma, A, is_bf16, p->m, p->k, p->k, TC_BM) || !map_b(&mb, B, 128)) return RG_ERR_CUDA;
                const int rc = mn ? (is_bf16 ? tc_launch_pair<__nv_bfloat16, true>(ma, mb, a, st) : tc_launch_pair<__half, true>(ma, mb, a, st))
                                  : (is_bf16 ? tc_launch_pair<__nv_bfloat16>(ma, mb, a, st) : tc_launch_pair<__half>(ma, mb, a, st));
                if (rc != RG_OK) return rc;
                continue;
            }
            if (!make_map(&ma, A, is_bf16, p->m, p->k, p->k, TC_BM) || !map_b(&mb, B, bn)) return RG_ERR_CUDA;
        } else {
            bn = p->m <= 32 ? 32 : 64;
            a.m = p->n, a.n = p->m;
            a.early = (p->flags & RG_MM_B_STATIC) ? 1u : 0u;
            a.Y = Y, a.y_row_stride = 1, a.y_col_stride = p->n;
            a.C = C, a.c_row_stride = p->bias_col_stride, a.c_col_stride = p->bias_row_stride;
            if (!map_b(&ma, B, TC_BM) || !make_map(&mb, A, is_bf16, p->m, p->k, p->k, bn)) return RG_ERR_CUDA;
        }
        int rc;
#define RG_TC(T, MN)                                                                                                           \
    (bn == 256 ? tc_launch<T, 256, 4, false, MN>(ma, mb, a, st) : bn == 128 ? tc_launch<T, 128, 6, false, MN>(ma, mb, a, st) \
     : bn == 64 ? tc_launch<T, 64, 6, false, MN>(ma, mb, a, st) : tc_launch<T, 32, 8, false, MN>(ma, mb, a, st))
        rc = mn ? (is_bf16 ? RG_TC(__nv_bfloat16, true) : RG_TC(__half, true)) : (is_bf16 ? RG_TC(__nv_bfloat16, false) : RG_TC(__half, false));
#undef RG_TC
        if (rc != RG_OK) return rc;
    }
    return RG_OK;
}

// Y = X W^T with the QKV split, rotation and cache append in the epilogue (rg_b200_linear, epilogue 3, more than 64 tokens).
int gemm_tc_qkv_rope(const rg_linear_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    if (p->dtype != RG_FP16 && p->dtype != RG_BF16) return RG_ERR_DTYPE;
    const uint32_t nq = p->n_heads, nkv = p->kv.n_kv_heads;
    if (p->kv.head_dim != 128 || nkv == 0 || nq == 0 || p->n != (nq + 2 * nkv) * 128u || p->m <= 64) return RG_ERR_SHAPE;
    if (p->prologue != 0 || p->k % 8 != 0 || p->k < 64 || !(p->theta > 0.f)) return RG_ERR_UNSUPPORTED;
    if (!in[0] || !in[1] || !in[4] || !out[0] || !out[1] || !out[2]) return RG_ERR_NULL;
    if (in[5] && p->kv.page_size == 0) return RG_ERR_SHAPE;
    if (!aligned16(in[0]) || !aligned16(in[1]) || !aligned16(out[0]) || !aligned16(out[1]) || !aligned16(out[2])) return RG_ERR_ALIGN;
    if (!encode_fn()) return RG_ERR_UNSUPPORTED;
    const int is_bf16 = p->dtype == RG_BF16;
    TcArgs a = {};
    a.alpha = 1.f, a.beta = 0.f, a.is_bf16 = is_bf16, a.k = p->k, a.m = p->m, a.n = p->n;
    a.early = 2;
    a.Y = out[0], a.y_row_stride = p->n, a.y_col_stride = 1;
    a.rope = 1, a.nq = nq, a.tokens_per_seq = p->tokens_per_seq, a.log2_theta = log2f(p->theta);
    a.pos = static_cast<const int64_t *>(in[4]), a.table = static_cast<const int32_t *>(in[5]);
    a.q_out = out[0], a.kc = out[1], a.vc = out[2], a.kv = p->kv;
    CUtensorMap ma, mb;
    const bool pair = p->m >= 512 && tc_pair_enabled();// a pair of CTAs per 256-token tile: each loads half of the B tile
    if (!make_map(&ma, in[0], is_bf16, p->m, p->k, p->k, TC_BM) || !make_map(&mb, in[1], is_bf16, p->n, p->k, p->k, pair ? 128 : 256)) return RG_ERR_CUDA;
    if (pair) return is_bf16 ? tc_launch_pair<__nv_bfloat16>(ma, mb, a, st) : tc_launch_pair<__half>(ma, mb, a, st);
    return is_bf16 ? tc_launch<__nv_bfloat16, 256, 4>(ma, mb, a, st) : tc_launch<__half, 256, 4>(ma, mb, a, st);
}

// Y[m, n/2] = silu(X Wg^T) * (X Wu^T), W = [gate rows ; up rows] (rg_b200_linear, epilogue 2, more than 64 tokens): one B tile
// pairs 128 gate rows with their 128 up rows, so both halves of an output column meet in one accumulator.
// Up to 64 tokens: the weights go on the instruction's M side (a tile = 64 gate rows + their 64 up rows), the tokens on its N
// side, k divided over clusters as for the plain skinny product; the up half of a tile hands its sums to the gate half.
bool gemm_tc_swiglu_small_shape(const rg_linear_params *p) {
    return (p->dtype == RG_FP16 || p->dtype == RG_BF16) && p->epilogue == 2 && p->prologue == 0 && p->m > 4 && p->m <= 64 &&
           p->n % 128 == 0 && p->n >= 128 && p->k % 8 == 0 && p->k >= 64 && encode_fn() != nullptr;
}
int gemm_tc_swiglu_small(const rg_linear_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    if (!gemm_tc_swiglu_small_shape(p)) return RG_ERR_SHAPE;
    if (!in[0] || !in[1] || !out[0]) return RG_ERR_NULL;
    if (!aligned16(in[0]) || !aligned16(in[1]) || !aligned16(out[0])) return RG_ERR_ALIGN;
    const int is_bf16 = p->dtype == RG_BF16;
    TcArgs a = {};
    a.alpha = 1.f, a.beta = 0.f, a.is_bf16 = is_bf16, a.k = p->k;
    a.m = p->n, a.n = p->m;// kernel rows = weight rows (gate and up interleaved by tile), kernel columns = tokens
    a.early = 1, a.swiglu = p->n / 2;
    a.Y = out[0], a.y_row_stride = 1, a.y_col_stride = p->n / 2;
    CUtensorMap ma, mb;
    const uint32_t bn = p->m <= 32 ? 32 : 64;
    if (!make_map(&ma, in[1], is_bf16, p->n, p->k, p->k, 64) || !make_map(&mb, in[0], is_bf16, p->m, p->k, p->k, bn)) return RG_ERR_CUDA;
    if (bn == 32) return is_bf16 ? tc_launch<__nv_bfloat16, 32, 8>(ma, mb, a, st) : tc_launch<__half, 32, 8>(ma, mb, a, st);
    return is_bf16 ? tc_launch<__nv_bfloat16, 64, 6>(ma, mb, a, st) : tc_launch<__half, 64, 6>(ma, mb, a, st);
}

// Row-parallel product feeding an all-reduce: the plain skinny product (weights on the M side) whose epilogue stores into the
// communicator's slots.  m <= 64 tokens, n a multiple of 8, no C operand.
int gemm_tc_push(const rg_mat_mul_params *p, const void *const *in, const ArPeers &peers, cudaStream_t st) {
    if (p->dtype != RG_FP16 && p->dtype != RG_BF16) return RG_ERR_UNSUPPORTED;
    if (p->trans_a || !p->trans_b || p->batch != 1 || p->has_bias || p->m == 0 || p->m > 64 || p->n < 128 || p->n % 8 != 0 || p->k % 8 != 0 || p->k < 64)
        return RG_ERR_UNSUPPORTED;
    if (!aligned16(in[0]) || !aligned16(in[1]) || !encode_fn()) return RG_ERR_UNSUPPORTED;
    const int is_bf16 = p->dtype == RG_BF16;
    TcArgs a = {};
    a.alpha = p->alpha, a.beta = 0.f, a.is_bf16 = is_bf16, a.k = p->k;
    a.m = p->n, a.n = p->m;// kernel rows = output features, kernel columns = tokens
    a.early = (p->flags & RG_MM_B_STATIC) ? 1u : 0u;
    a.push = peers.two_shot ? 2u : 1u, a.ar = peers;
    CUtensorMap ma, mb;
    const uint32_t bn = p->m <= 32 ? 32 : 64;
    if (!make_map(&ma, in[1], is_bf16, p->n, p->k, p->k, TC_BM) || !make_map(&mb, in[0], is_bf16, p->m, p->k, p->k, bn)) return RG_ERR_CUDA;
    if (bn == 32) return is_bf16 ? tc_launch<__nv_bfloat16, 32, 8, true>(ma, mb, a, st) : tc_launch<__half, 32, 8, true>(ma, mb, a, st);
    return is_bf16 ? tc_launch<__nv_bfloat16, 64, 6, true>(ma, mb, a, st) : tc_launch<__half, 64, 6, true>(ma, mb, a, st);
}

// The same for the QKV projection with its split / rotation / cache-append epilogue on 5..64 tokens (a 128-row tile = one head).
bool gemm_tc_qkv_rope_small_shape(const rg_linear_params *p) {
    const uint32_t nq = p->n_heads, nkv = p->kv.n_kv_heads;
    return (p->dtype == RG_FP16 || p->dtype == RG_BF16) && p->epilogue == 3 && p->prologue == 0 && p->m > 4 && p->m <= 64 && p->kv.head_dim == 128 &&
           nq > 0 && nkv > 0 && p->n == (nq + 2 * nkv) * 128u && p->k % 8 == 0 && p->k >= 64 && p->theta > 0.f && encode_fn() != nullptr;
}
int gemm_tc_qkv_rope_small(const rg_linear_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    if (!gemm_tc_qkv_rope_small_shape(p)) return RG_ERR_SHAPE;
    if (!in[0] || !in[1] || !in[4] || !out[0] || !out[1] || !out[2]) return RG_ERR_NULL;
    if (in[5] && p->kv.page_size == 0) return RG_ERR_SHAPE;
    if (!aligned16(in[0]) || !aligned16(in[1])) return RG_ERR_ALIGN;
    const int is_bf16 = p->dtype == RG_BF16;
    TcArgs a = {};
    a.alpha = 1.f, a.beta = 0.f, a.is_bf16 = is_bf16, a.k = p->k;
    a.m = p->n, a.n = p->m;// kernel rows = output features (a tile = a head), kernel columns = tokens
    a.early = 1;
    a.rope = 1, a.nq = p->n_heads, a.tokens_per_seq = p->tokens_per_seq, a.log2_theta = log2f(p->theta);
    a.pos = static_cast<const int64_t *>(in[4]), a.table = static_cast<const int32_t *>(in[5]);
    a.q_out = out[0], a.kc = out[1], a.vc = out[2], a.kv = p->kv;
    CUtensorMap ma, mb;
    const uint32_t bn = p->m <= 32 ? 32 : 64;
    if (!make_map(&ma, in[1], is_bf16, p->n, p->k, p->k, TC_BM) || !make_map(&mb, in[0], is_bf16, p->m, p->k, p->k, bn)) return RG_ERR_CUDA;
    if (bn == 32) return is_bf16 ? tc_launch<__nv_bfloat16, 32, 8>(ma, mb, a, st) : tc_launch<__half, 32, 8>(ma, mb, a, st);
    return is_bf16 ? tc_launch<__nv_bfloat16, 64, 6>(ma, mb, a, st) : tc_launch<__half, 64, 6>(ma, mb, a, st);
}

int gemm_tc_swiglu(const rg_linear_params *p, const void *const *in, void *const *out, cudaStream_t st) {
    if (p->dtype != RG_FP16 && p->dtype != RG_BF16) return RG_ERR_DTYPE;
    const uint32_t f = p->n / 2;
    if (p->m <= 64 || p->n % 2 != 0 || f % 128 != 0) return RG_ERR_SHAPE;
    if (p->prologue != 0 || p->k % 8 != 0 || p->k < 64) return RG_ERR_UNSUPPORTED;
    if (!in[0] || !in[1] || !out[0]) return RG_ERR_NULL;
    if (!aligned16(in[0]) || !aligned16(in[1]) || !aligned16(out[0])) return RG_ERR_ALIGN;
    if (!encode_fn()) return RG_ERR_UNSUPPORTED;
    const int is_bf16 = p->dtype == RG_BF16;
    TcArgs a = {};
    a.alpha = 1.f, a.beta = 0.f, a.is_bf16 = is_bf16, a.k = p->k, a.m = p->m, a.n = p->n;
    a.early = 2, a.swiglu = f;
    a.Y = out[0], a.y_row_stride = f, a.y_col_stride = 1;
    CUtensorMap ma, mb;
    if (!make_map(&ma, in[0], is_bf16, p->m, p->k, p->k, TC_BM) || !make_map(&mb, in[1], is_bf16, p->n, p->k, p->k, 128)) return RG_ERR_CUDA;
    // pair mode: the even CTA of a pair loads the tile's gate rows, the odd one its up rows
    if (p->m >= 512 && tc_pair_enabled()) return is_bf16 ? tc_launch_pair<__nv_bfloat16>(ma, mb, a, st) : tc_launch_pair<__half>(ma, mb, a, st);
    return is_bf16 ? tc_launch<__nv_bfloat16, 256, 4>(ma, mb, a, st) : tc_launch<__half, 256, 4>(ma, mb, a, st);
}

int gemm_tc_error_word(bool clear) { return error_symbol(s_tc_error, clear); }
int gemm_tc_index_error_word(bool clear) { return error_symbol(s_tc_index_error, clear); }

}// namespace rg
