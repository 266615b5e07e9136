// y = x . W^T for prompt portions on the fifth-generation tensor cores, with the work
// that follows a projection folded into its epilogue.
//
//   x [M, K] bfloat16 (activations, K contiguous), W [N, K] bfloat16 (a projection's
//   weight as the checkpoint stores it, K contiguous), float32 accumulation.
//
// Epilogues (what the reference does in separate kernels after cublasSgemm,
// backend/model.cu:496-503 for the products, :477-483 for the gated activation,
// :97-110 for the residual sum):
//   0  y[M, N] bfloat16 = acc
//   1  y[M, N] float32  = acc
//   2  y[M, N] float32 += acc                        (residual stream)
//   3  y[M, N] bfloat16 = silu(acc_gate) * acc_up    (W = gate rows, W_up = up rows)
//   4  the same with g = min(acc_gate, limit), u = clamp(acc_up, -limit, limit): g sigmoid(alpha g) (u + 1)
//   5  y[M, N] bfloat16 = relu(acc)^2
//
// The gated epilogues (3 and 4) run on pairs of CTAs, further down.  For the others a
// persistent CTA per SM walks output tiles of 128 x BN.  BN, the accumulator's width,
// is a multiple of 16 up to 256.  Measured on this GPU, an M = 128 instruction takes the same time whatever its
// N, so anything narrower than 256 leaves the tensor core partly idle: 256 is the
// default and narrower tiles are for matrices with fewer columns.  Ten warps, three roles:
//   warp 0   producer: one lane issues TMA loads (cp.async.bulk.tensor, 128-byte
//            swizzle) of the x and W tiles of a 64-wide k block into a ring of
//            shared-memory stages, each guarded by a full/empty pair of mbarriers;
//   warp 1   one lane issues tcgen05.mma (M = 128, N = BN, K = 16; four per k block)
//            from the stage into one of two accumulators in tensor memory and commits
//            the stage back to the producer; after the last k block it commits the
//            accumulator to the epilogue;
//   warps 2-9  epilogue: a thread owns one row of one half of the tile's columns, reads
//            it from tensor memory 32 columns at a time (tcgen05.ld), applies the
//            epilogue and stores.  With two accumulators the epilogue of a tile overlaps
//            the products of the next.
// A row of the result is a sum over k in one fixed order, whatever else is in the batch.
//
// Every wait on an mbarrier is bounded by a cycle count; a wait that runs out raises a
// flag in shared memory and sets *status, all roles leave their loops, the producer
// waits (bounded) for copies it still has in flight, and the CTA frees its tensor
// memory and returns.
#include "common.cuh"

KLLM_EXPORT_LAST_ERROR(gemm_tcgen05)

#include "tc5_common.cuh"

namespace {

constexpr int BM = 128;                    // rows of a tile = lanes of tensor memory
constexpr int BK = TC5_BK;                 // k block: 64 bfloat16 = one 128-byte swizzled row
constexpr int THREADS = 320;
constexpr int EPI_THREADS = 256;
constexpr int A_BYTES = BM * 128;
constexpr int MAX_BN = 256;                // accumulators sit 256 columns apart in tensor memory
constexpr int TMEM_COLS = 2 * MAX_BN;
constexpr int MAX_STAGES = 8;
constexpr int SMEM_BYTES = 1024 + 4 * (A_BYTES + MAX_BN * 128);    // four stages of the widest tile

enum Epilogue { EPI_BF16 = 0, EPI_F32 = 1, EPI_ADD_F32 = 2, EPI_SWIGLU = 3, EPI_CLAMPED = 4, EPI_RELU2 = 5 };
constexpr bool is_gated(int epi) { return epi == EPI_SWIGLU || epi == EPI_CLAMPED; }
constexpr bool is_bf16(int epi) { return epi != EPI_F32 && epi != EPI_ADD_F32; }

// 32 consecutive results of one row, columns col..col+31 of the output, those below
// `limit` (the end of the tile or of the matrix); res: what the float32 destination held
template <int EPI>
__device__ __forceinline__ void store_chunk(void* y, int64_t ldy, int row, int col, int limit, const float (&v)[32],
                                            const float4 (&res)[8]) {
    if (is_bf16(EPI)) {
        bf16* p = (bf16*)y + (int64_t)row * ldy + col;
        if (col + 32 <= limit) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint4 pk;
                pk.x = pack_bf16(v[8 * c], v[8 * c + 1]);
                pk.y = pack_bf16(v[8 * c + 2], v[8 * c + 3]);
                pk.z = pack_bf16(v[8 * c + 4], v[8 * c + 5]);
                pk.w = pack_bf16(v[8 * c + 6], v[8 * c + 7]);
                *reinterpret_cast<uint4*>(p + 8 * c) = pk;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (col + j < limit) p[j] = __float2bfloat16_rn(v[j]);
        }
    } else {
        float* p = (float*)y + (int64_t)row * ldy + col;
        if (col + 32 <= limit) {
#pragma unroll
            for (int c = 0; c < 8; c++) {
                float4 o = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
                if (EPI == EPI_ADD_F32) { o.x += res[c].x; o.y += res[c].y; o.z += res[c].z; o.w += res[c].w; }
                *reinterpret_cast<float4*>(p + 4 * c) = o;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (col + j < limit) p[j] = (EPI == EPI_ADD_F32 ? p[j] : 0.f) + v[j];
        }
    }
}

// what the destination holds at columns col..col+31 of a row (whole chunks only; a
// ragged chunk is read where it is added)
__device__ __forceinline__ void load_residual(const void* y, int64_t ldy, int row, int col, int limit, bool row_ok,
                                              float4 (&res)[8]) {
    if (row_ok && col + 32 <= limit) {
        const float* p = (const float*)y + (int64_t)row * ldy + col;
#pragma unroll
        for (int c = 0; c < 8; c++) res[c] = *reinterpret_cast<const float4*>(p + 4 * c);
    }
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                void* __restrict__ y, int64_t ldy, int M, int N, int K,
                int bn, int stages, int* status) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_acc_full[2], bar_acc_empty[2];
    __shared__ unsigned s_tmem;
    __shared__ int s_abort;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int nout = bn;                                       // output columns of a tile
    const int b_bytes = bn * 128, stage_bytes = A_BYTES + b_bytes;
    const int m_tiles = (M + BM - 1) / BM;
    const int n_tiles = (N + nout - 1) / nout;
    const int tiles = m_tiles * n_tiles;
    const int kblocks = (K + BK - 1) / BK;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int a = 0; a < 2; a++) { mbar_init(&bar_acc_full[a], 1); mbar_init(&bar_acc_empty[a], EPI_THREADS); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    griddep_launch();

    if (warp == 0) {
        // ---- producer ----------------------------------------------------------
        if (elect_one()) {
            prefetch_map(&map_a);
            prefetch_map(&map_b);
        }
        griddep_wait();
        int s = 0;
        unsigned ph = 0;
        int issued = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * nout;
            for (int kb = 0; kb < kblocks; kb++) {
                ok = mbar_wait_warp(&bar_empty[s], ph ^ 1u, abort_flag, status, 1);
                if (!ok) break;
                if (elect_one()) {
                    const unsigned a = base + (unsigned)(s * stage_bytes), b = a + A_BYTES;
                    mbar_expect_tx(&bar_full[s], (unsigned)stage_bytes);
                    tma_load_2d(a, &map_a, kb * BK, m0, &bar_full[s]);
                    tma_load_2d(b, &map_b, kb * BK, n0, &bar_full[s]);
                }
                __syncwarp();
                issued++;
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
        }
        if (!ok || *abort_flag) {
            // copies still in flight must land before the shared memory goes away: wait,
            // with the same bound, for the stages armed last
            const int back = issued < stages ? issued : stages;
            for (int j = 0; j < back; j++) {
                int sj = s - 1 - j;
                unsigned pj = ph;
                if (sj < 0) { sj += stages; pj ^= 1u; }
                const long long t0 = clock64();
                while (!mbar_try_wait(&bar_full[sj], pj) && clock64() - t0 < kCycleLimit) {}
            }
        }
    } else if (warp == 1) {
        // ---- tensor-core issuer ------------------------------------------------
        const uint32_t idesc = make_idesc(BM, bn);
        griddep_wait();
        int s = 0, acc = 0;
        unsigned ph = 0, acc_ph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            ok = mbar_wait_warp(&bar_acc_empty[acc], acc_ph ^ 1u, abort_flag, status, 2);
            if (!ok) break;
            tc_fence_after();
            const unsigned d = tmem + (unsigned)(acc * MAX_BN);
            for (int kb = 0; kb < kblocks; kb++) {
                ok = mbar_wait_warp(&bar_full[s], ph, abort_flag, status, 3);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const unsigned a = base + (unsigned)(s * stage_bytes), b = a + A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++)
                        umma(d, make_desc(a + kk * 32), make_desc(b + kk * 32), idesc, kb > 0 || kk > 0);
                    umma_commit(&bar_empty[s]);
                }
                __syncwarp();
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            if (elect_one()) umma_commit(&bar_acc_full[acc]);
            __syncwarp();
            acc ^= 1;
            if (acc == 0) acc_ph ^= 1u;
        }
    } else {
        // ---- epilogue ----------------------------------------------------------
        griddep_wait();
        const int quarter = warp & 3;                      // the 32 lanes of tensor memory this warp may read
        const int half = (warp - 2) >> 2;                  // which half of the tile's 32-column chunks
        const unsigned lane_base = (unsigned)(quarter * 32) << 16;
        const int chunks = (nout + 31) / 32;
        const int c_lo = half == 0 ? 0 : (chunks + 1) / 2, c_hi = half == 0 ? (chunks + 1) / 2 : chunks;
        int acc = 0;
        unsigned acc_ph = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * nout;
            const int row = m0 + quarter * 32 + lane;
            const bool row_ok = row < M;
            const int limit = min(N, n0 + nout);
            float4 res[8];
            if (EPI == EPI_ADD_F32) load_residual(y, ldy, row, n0 + c_lo * 32, limit, row_ok, res);   // under the products
            if (!mbar_wait(&bar_acc_full[acc], acc_ph, abort_flag, status, 4)) break;
            tc_fence_after();
            const unsigned t = tmem + lane_base + (unsigned)(acc * MAX_BN);
#pragma unroll 1
            for (int c = c_lo; c < c_hi; c++) {
                float v[32];
                float4 res_next[8];
                tmem_ld32(t + c * 32, v);
                if (EPI == EPI_ADD_F32 && c + 1 < c_hi) load_residual(y, ldy, row, n0 + (c + 1) * 32, limit, row_ok, res_next);
                tmem_ld_wait();
                if (EPI == EPI_RELU2) {
#pragma unroll
                    for (int j = 0; j < 32; j++) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
                }
                const int col = n0 + c * 32;
                if (row_ok && col < limit) store_chunk<EPI>(y, ldy, row, col, limit, v, res);
                if (EPI == EPI_ADD_F32) {
#pragma unroll
                    for (int j = 0; j < 8; j++) res[j] = res_next[j];
                }
            }
            tc_fence_before();
            mbar_arrive(&bar_acc_empty[acc]);
            acc ^= 1;
            if (acc == 0) acc_ph ^= 1u;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
}

// ---- the gated epilogues on pairs of CTAs ----------------------------------------
// A gated product's tile is PAIR_F output columns (as many gate and up rows of W) by bn rows of x, bn a multiple of 16 up to 256.
// W is the 256-row operand of a cta_group::2 instruction and x the one of bn rows, so that the tile's second size follows the
// number of rows of a step: 845 rows run as five tiles of 176, three even waves, where tiles of 128 x rows had 308 tiles for
// 148 SMs.  A CTA holds 64 gate rows, the 64 up rows behind them and half of x's rows: 64 bytes a cycle of operands from shared
// memory at the full rate, where a CTA alone needs 96 and reached 77 % of it.  Roles as above; the leader's warp 1 issues for
// both, either CTA's producer loads its own operands and announces them on the leader's barriers.  A column's gate and up values
// lie 64 lanes apart: the two warps that read them exchange half of each through shared memory and finish half of the rows each.
// (Interleaved by 16 rows they would be a shuffle apart, but eight copies of 16 rows a stage instead of two took longer than
// the products.)  The results meet in shared memory and leave as whole 128-byte rows.  Sixteen warps finish them: what a warp waits for
// is its chain of exchange, expf and division, and with eight a tile of 256 rows took 9 us, longer than the products of K up to
// 1300 that it runs beside (768 x 3072, 4096 rows: 60.9 us with eight warps, 31.6 with sixteen, 38.0 for the kernel of
// CTAs alone that this one replaced; 1024 x 2816: 45.0, 33.9, 40.5; 2048 x 5632: 124.8, 120.8, 139.8).
//
// A tile's rows are the fastest in the order of tiles, so that neighbouring pairs share W's rows; x stays in L2.  The last tile of
// rows is moved back to end with x and leaves what it shares with the tile before to that one: rows behind x's end, which the copy
// fills with zeros, took longer than rows that are there (64 rows in a tile of 256: 27 us, in one of 64: 14).
constexpr int PAIR_F = 128;
constexpr int PAIR_STAGE_ROW = 144;                                  // bytes of a row of results in shared memory, 128 in use
constexpr int PAIR_SWAP_BYTES = 8 * 2 * 8 * 32 * 4;                  // what the eight pairs of epilogue warps exchange
constexpr int PAIR_OUT_BYTES = MAX_BN * PAIR_STAGE_ROW + PAIR_SWAP_BYTES;
constexpr int PAIR_SMEM = 1024 + PAIR_OUT_BYTES + 5 * (A_BYTES + MAX_BN / 2 * 128);
constexpr int PAIR_EPI_WARPS = 16, PAIR_THREADS = 64 + 32 * PAIR_EPI_WARPS;

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_up, bf16* __restrict__ y, int64_t ldy, int M, int N, int K, int bn, int stages,
                 float act_limit, float act_alpha, int* status) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_acc_full[2], bar_acc_empty[2];
    __shared__ unsigned s_tmem;
    __shared__ int s_abort;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int b_rows = bn / 2;
    const unsigned stage_bytes = (unsigned)(A_BYTES + b_rows * 128);         // a multiple of the swizzle's 1024, as bn is of 16
    unsigned char* results = smem_raw + (base - smem_u32(smem_raw)) + stages * stage_bytes;
    const int t_tiles = (M + bn - 1) / bn, f_tiles = (N + PAIR_F - 1) / PAIR_F;
    const int tiles = t_tiles * f_tiles, pairs = gridDim.x >> 1, first = blockIdx.x >> 1;
    const int kblocks = (K + BK - 1) / BK;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int a = 0; a < 2; a++) { mbar_init(&bar_acc_full[a], 1); mbar_init(&bar_acc_empty[a], 2 * PAIR_EPI_WARPS); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    griddep_launch();

    if (warp == 0) {
        // ---- producer: this CTA's rows of W and of x ----
        int s = 0, issued = 0;
        unsigned ph = 0;
        bool ok = true;
        const unsigned full0 = leader_addr(&bar_full[0]);             // the leader's barriers, 8 bytes apart
        auto load_w = [&](int s, int f0, int kb) {
            const unsigned a = base + s * stage_bytes, bar = full0 + 8u * s;
            if (rank == 0) mbar_expect_tx(&bar_full[s], 2u * stage_bytes);
            tma_load_2d_pair(a, &map_w, kb * BK, f0, bar);
            tma_load_2d_pair(a + A_BYTES / 2, &map_up, kb * BK, f0, bar);
        };
        auto load_x = [&](int s, int t0, int kb) {
            tma_load_2d_pair(base + s * stage_bytes + A_BYTES, &map_x, kb * BK, t0, full0 + 8u * s);
        };
        auto col0 = [&](int tile) { return tile / t_tiles * PAIR_F + (int)rank * 64; };
        auto row0 = [&](int tile) { return min(tile % t_tiles * bn, max(0, M - bn)) + (int)rank * b_rows; };
        // the first stages' weights do not depend on the kernel before
        const int early = first < tiles ? min(stages, kblocks) : 0;
        if (elect_one()) {
            prefetch_map(&map_x);
            prefetch_map(&map_w);
            prefetch_map(&map_up);
            for (int kb = 0; kb < early; kb++) load_w(kb, col0(first), kb);
        }
        griddep_wait();
        if (elect_one())
            for (int kb = 0; kb < early; kb++) load_x(kb, row0(first), kb);
        __syncwarp();
        issued = early;
        s = early % stages;
        ph = early == stages ? 1u : 0u;
        for (int tile = first; ok && tile < tiles; tile += pairs) {
            const int f0 = col0(tile), t0 = row0(tile);
            for (int kb = tile == first ? early : 0; kb < kblocks; kb++) {
                ok = mbar_wait_warp(&bar_empty[s], ph ^ 1u, abort_flag, status, 1);
                if (!ok) break;
                if (elect_one()) {
                    load_w(s, f0, kb);
                    load_x(s, t0, kb);
                }
                __syncwarp();
                issued++;
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
        }
        if (ok && !*abort_flag) {
            // the other CTA's products arrive at these barriers: stay until the last has
            for (int j = 0; ok && j < stages; j++) {
                ok = mbar_wait_warp(&bar_empty[s], ph ^ 1u, abort_flag, status, 1);
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
        } else if (rank == 0) {
            // copies still in flight must land before the shared memory goes away: wait, with the same bound, for the
            // stages armed last (the leader for both CTAs; the other one is held by the cluster's barrier)
            const int back = issued < stages ? issued : stages;
            for (int j = 0; j < back; j++) {
                int sj = s - 1 - j;
                unsigned pj = ph;
                if (sj < 0) { sj += stages; pj ^= 1u; }
                const long long t0 = clock64();
                while (!mbar_try_wait(&bar_full[sj], pj) && clock64() - t0 < kCycleLimit) {}
            }
        }
    } else if (warp == 1) {
        // ---- tensor-core issuer ----
        if (rank == 0) {
            const uint32_t idesc = make_idesc(256, bn);
            int s = 0, acc = 0;
            unsigned ph = 0, acc_ph = 0;
            bool ok = true;
            for (int tile = first; ok && tile < tiles; tile += pairs) {
                ok = mbar_wait_warp(&bar_acc_empty[acc], acc_ph ^ 1u, abort_flag, status, 2);
                if (!ok) break;
                tc_fence_after();
                const unsigned d = tmem + (unsigned)(acc * MAX_BN);
                for (int kb = 0; kb < kblocks; kb++) {
                    ok = mbar_wait_warp(&bar_full[s], ph, abort_flag, status, 3);
                    if (!ok) break;
                    if (elect_one()) {
                        const unsigned a = base + s * stage_bytes, b = a + A_BYTES;
#pragma unroll
                        for (int kk = 0; kk < BK / 16; kk++)
                            umma_pair(d, make_desc(a + kk * 32), make_desc(b + kk * 32), idesc, kb > 0 || kk > 0);
                        umma_commit_pair(&bar_empty[s]);
                    }
                    __syncwarp();
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) umma_commit_pair(&bar_acc_full[acc]);
                __syncwarp();
                acc ^= 1;
                if (acc == 0) acc_ph ^= 1u;
            }
        }
    } else {
        // ---- epilogue ----
        griddep_wait();
        // four warps of each quarter of the lanes; set `part` of them has a quarter of the tile's rows of x, 16 at a time
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const unsigned lane_base = (unsigned)(quarter * 32) << 16;
        const int c_lo = bn / 16 * part / 4, c_hi = bn / 16 * (part + 1) / 4;
        // quarters 0 and 1 hold the gate values of columns 0-31 and 32-63, quarters 2 and 3 the up values
        const bool up = quarter >= 2;
        const int group = quarter & 1, swap_id = 5 + part * 2 + group, in_part = threadIdx.x - 64 - part * 128;
        float* swap = reinterpret_cast<float*>(results + MAX_BN * PAIR_STAGE_ROW) + (part * 2 + group) * 2 * 8 * 32 + lane;
        int acc = 0;
        unsigned acc_ph = 0;
        for (int tile = first; tile < tiles; tile += pairs) {
            const int t_own = tile % t_tiles * bn, t0 = min(t_own, max(0, M - bn)), f0 = tile / t_tiles * PAIR_F + (int)rank * 64;
            // all threads of the set go on or none; its results of the tile before have left shared memory
            if (!half_all(1 + part, mbar_wait(&bar_acc_full[acc], acc_ph, abort_flag, status, 4))) break;
            tc_fence_after();
            const unsigned t = tmem + lane_base + (unsigned)(acc * MAX_BN);
            float v[16];
            if (c_lo < c_hi) tmem_ld16(t + c_lo * 16, v);
#pragma unroll 1
            for (int c = c_lo; c < c_hi; c++) {
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; i++) swap[(up * 8 + i) * 32] = up ? v[i] : v[8 + i];
                named_sync(swap_id, 64);
                // the gate warp finishes the first 8 of the 16 rows of x, the up warp the others
                float g[8], u[8], den[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float got = swap[(!up * 8 + i) * 32];
                    g[i] = up ? got : v[i];
                    u[i] = up ? v[8 + i] : got;
                }
                named_sync(swap_id, 64);                   // both have read before either writes again
                if (c + 1 < c_hi) tmem_ld16(t + (c + 1) * 16, v);
                // a division checks for what its short form cannot do, one after the other: what leads to it is done for all 8 before
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (EPI == EPI_CLAMPED) {
                        g[i] = fminf(g[i], act_limit);
                        u[i] = fminf(fmaxf(u[i], -act_limit), act_limit) + 1.f;
                    }
                    den[i] = 1.f + expf(EPI == EPI_CLAMPED ? -act_alpha * g[i] : -g[i]);
                }
                bf16* o = reinterpret_cast<bf16*>(results + (c * 16 + up * 8) * PAIR_STAGE_ROW) + group * 32 + lane;
#pragma unroll
                for (int i = 0; i < 8; i++) o[i * (PAIR_STAGE_ROW / 2)] = __float2bfloat16_rn(g[i] / den[i] * u[i]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_addr(&bar_acc_empty[acc]));
            named_sync(1 + part, 128);
            const int r_hi = min(c_hi * 16, M - t0);
            for (int i = in_part + max(c_lo * 16, t_own - t0) * 8; i < r_hi * 8; i += 128) {
                const int r = i >> 3, f = f0 + (i & 7) * 8;
                const uint4 w = *reinterpret_cast<const uint4*>(results + r * PAIR_STAGE_ROW + (i & 7) * 16);
                bf16* o = y + (int64_t)(t0 + r) * ldy + f;
                if (f + 8 <= N) {
                    *reinterpret_cast<uint4*>(o) = w;
                } else {
                    const bf16* e = reinterpret_cast<const bf16*>(&w);
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (f + j < N) o[j] = e[j];
                }
            }
            acc ^= 1;
            if (acc == 0) acc_ph ^= 1u;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                        // nothing of the pair's is under way in either CTA any more
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
}

// ---- host side -----------------------------------------------------------------

// Accumulator width: a tile's time does not shrink with its width (see the top of the
// file), so the widest one with the fewest waves of tiles wins.
int pick_bn(int M, int N) {
    const int sms = sm_count();
    const int m_tiles = (M + BM - 1) / BM;
    long long best = -1;
    int best_bn = MAX_BN;
    for (int bn = MAX_BN; bn >= 64; bn -= 16) {
        const long long tiles = (long long)m_tiles * ((N + bn - 1) / bn);
        const long long waves = (tiles + sms - 1) / sms;
        if (best < 0 || waves < best) { best = waves; best_bn = bn; }
    }
    return best_bn;
}

template <int EPI>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, void* y, int64_t ldy, int M, int N, int K, int bn, int* status,
           cudaStream_t stream) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc5_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) {
            snprintf(g_kllm_err, sizeof(g_kllm_err), "gemm (tcgen05): %d bytes of shared memory refused: %s", SMEM_BYTES,
                     cudaGetErrorString(e));
            return (int)e;
        }
        attr_set = true;
    }
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + bn - 1) / bn);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    int stages = (SMEM_BYTES - 1024) / (A_BYTES + bn * 128);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    kllm_launch((gemm_tc5_kernel<EPI>), dim3(grid), dim3(THREADS), SMEM_BYTES, stream, ma, mb, y, ldy, M, N, K, bn, stages, status);
    KLLM_LAUNCH_STATUS();
}

// Rows of x in a tile of a pair, and the product's time in units of a wave's row of x: the least waves x (bn + 100).  A wave of
// K = 2048 takes 4.0 us + 0.040 us a row (64 rows 6.6 us, 128 8.5, 256 14.2): issue and hand-over of a k block beside
// its products.
struct PairPlan {
    int bn;
    long long cost;
};
PairPlan pair_plan(int M, int N) {
    const long long pairs = sm_count() / 2, f_tiles = (N + PAIR_F - 1) / PAIR_F;
    PairPlan best{MAX_BN, -1};
    for (int bn = M < MAX_BN ? (M + 15) / 16 * 16 : MAX_BN; bn >= 16; bn -= 16) {
        const long long tiles = f_tiles * ((M + bn - 1) / bn), cost = (tiles + pairs - 1) / pairs * (bn + 100);
        if (best.cost < 0 || cost < best.cost) best = PairPlan{bn, cost};
    }
    return best;
}

template <int EPI>
int launch_pair(const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& mu, void* y, int64_t ldy, int M, int N, int K, int bn,
                float act_limit, float act_alpha, int* status, cudaStream_t stream) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM);
        if (e != cudaSuccess) {
            snprintf(g_kllm_err, sizeof(g_kllm_err), "gemm (tcgen05): %d bytes of shared memory refused: %s", PAIR_SMEM,
                     cudaGetErrorString(e));
            return (int)e;
        }
        attr_set = true;
    }
    const long long tiles = (long long)((M + bn - 1) / bn) * ((N + PAIR_F - 1) / PAIR_F), pairs = sm_count() / 2;
    const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
    int stages = (PAIR_SMEM - 1024 - PAIR_OUT_BYTES) / (A_BYTES + bn * 64);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    kllm_launch((gemm_pair_kernel<EPI>), dim3(grid), dim3(PAIR_THREADS), PAIR_SMEM, stream, mx, mw, mu, (bf16*)y, ldy, M, N, K, bn, stages,
                act_limit, act_alpha, status);
    KLLM_LAUNCH_STATUS();
}

}  // namespace

// What a gated product of M rows and N columns runs as: rows of x in a tile, waves of tiles.
extern "C" int kllm_gemm_tcgen05_pair_plan(int M, int N, int* bn, int* waves) {
    *bn = *waves = 0;
    if (M <= 0 || N <= 0) return 0;
    const PairPlan p = pair_plan(M, N);
    *bn = p.bn;
    *waves = (int)(p.cost / (p.bn + 100));
    return 0;
}

// 1 if the kernel takes these sizes and addresses, else 0 (the caller then uses the
// library product and separate elementwise kernels).
extern "C" int kllm_gemm_tcgen05_fits(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* w_up, int M,
                                      int N, int K, const void* y, int64_t ldy, int epilogue) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (epilogue < 0 || epilogue > 5) return 0;
    if ((K & 7) || (ldx & 7) || (ldw & 7)) return 0;                      // TMA: 16-byte rows
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)w_up & 15) || ((uintptr_t)y & 15)) return 0;
    const bool bf16_out = is_bf16(epilogue);
    if (bf16_out ? (ldy & 7) : (ldy & 3)) return 0;                        // 16-byte vector stores
    if (is_gated(epilogue) && !w_up) return 0;
    return 1;
}

// bn: accumulator width of a tile, 0 = chosen here, else a multiple of 16 from 64 (for the
// gated epilogues, whose accumulators are as wide as a tile has rows of x, from 16) to 256.  act_limit, act_alpha: of epilogue 4.  status: device int that a wait which ran out sets
// (1: producer, 2: accumulator, 3: stage, 4: epilogue).
extern "C" int kllm_gemm_tcgen05(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* w_up, int M, int N,
                                 int K, void* y, int64_t ldy, int epilogue, int bn, float act_limit, float act_alpha, int* status,
                                 void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!kllm_gemm_tcgen05_fits(x, ldx, w, ldw, w_up, M, N, K, y, ldy, epilogue))
        KLLM_FAIL("gemm (tcgen05): sizes %d x %d x %d, strides %lld/%lld/%lld or an address not taken (k and strides "
                  "multiples of 8, 16-byte aligned addresses)", M, N, K, (long long)ldx, (long long)ldw, (long long)ldy);
    if (epilogue == EPI_CLAMPED && !(act_limit > 0.f)) KLLM_FAIL("gemm (tcgen05): the clamped epilogue needs a positive limit");
    if (is_gated(epilogue)) {
        if (bn == 0) bn = pair_plan(M, N).bn;
        if (bn < 16 || bn > MAX_BN || bn % 16) KLLM_FAIL("gemm (tcgen05): accumulator width %d, a multiple of 16 from 16 to %d", bn, MAX_BN);
        CUtensorMap mx, mw, mu;
        int r = tensor_map(&mx, x, ldx, M, K, bn / 2);
        if (!r) r = tensor_map(&mw, w, ldw, N, K, PAIR_F / 2);
        if (!r) r = tensor_map(&mu, w_up, ldw, N, K, PAIR_F / 2);
        if (r) return r;
        return epilogue == EPI_CLAMPED
                   ? launch_pair<EPI_CLAMPED>(mx, mw, mu, y, ldy, M, N, K, bn, act_limit, act_alpha, status, (cudaStream_t)stream)
                   : launch_pair<EPI_SWIGLU>(mx, mw, mu, y, ldy, M, N, K, bn, 0.f, 0.f, status, (cudaStream_t)stream);
    }
    if (bn == 0) bn = pick_bn(M, N);
    if (bn < 64 || bn > MAX_BN || bn % 16) KLLM_FAIL("gemm (tcgen05): accumulator width %d, a multiple of 16 from 64 to %d", bn, MAX_BN);
    CUtensorMap ma, mb;
    int r = tensor_map(&ma, x, ldx, M, K, BM);
    if (!r) r = tensor_map(&mb, w, ldw, N, K, bn);
    if (r) return r;
    cudaStream_t s = (cudaStream_t)stream;
    switch (epilogue) {
        case EPI_BF16: return launch<EPI_BF16>(ma, mb, y, ldy, M, N, K, bn, status, s);
        case EPI_F32: return launch<EPI_F32>(ma, mb, y, ldy, M, N, K, bn, status, s);
        case EPI_ADD_F32: return launch<EPI_ADD_F32>(ma, mb, y, ldy, M, N, K, bn, status, s);
        default: return launch<EPI_RELU2>(ma, mb, y, ldy, M, N, K, bn, status, s);
    }
}
