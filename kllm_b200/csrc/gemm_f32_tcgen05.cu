// y = x . W^T of float32 matrices on the fifth-generation tensor cores, at float32 accuracy.
//
//   x [M, K] float32 (K contiguous), W [N, K] float32 (a projection's weight as the checkpoint
//   stores it), y float32: stored, added into, or silu(x Wg^T) * (x Wu^T).
//
// The reference runs these products through cublasSgemm (backend/model.cu:496-503); on the
// CUDA cores they are bound by the FMA rate (the library reached 50 TFLOP/s at 1003 rows of
// TinyLlama's sizes).  Here every float32 number is the sum of three bfloat16 numbers,
//     v = v0 + v1 + v2,  v0 = bf16(v), v1 = bf16(v - v0), v2 = bf16(v - v0 - v1)
// (8 + 8 + 8 bits of mantissa), and
//     x w = x0 w0 + (x0 w1 + x1 w0) + (x0 w2 + x1 w1 + x2 w0) + terms below 2^-24 |x w|,
// six tcgen05 products with float32 accumulators.  An accumulator only ever holds one k block
// (32 values of k, the small terms first): it is then added, by the rounding add of the CUDA
// cores, to a sum in registers, so that the tensor core's own accumulation, which cuts digits
// off, cannot drift over a long K.
//
// Two kernels.  `split_kernel` writes the three parts of a matrix as three bfloat16 planes; `gemm_f32_tc5_kernel` multiplies
// planes.  W is taken in pieces of rows whose planes (6 bytes a number, PLANE_LIMIT at most) have two buffers that take turns: a
// piece is split while the piece before it is being multiplied, beside the product's CTA on every SM (the product is bound by
// the tensor cores and leaves HBM idle).  A kernel that split inside the product, in registers, was measured at 392 us for
// 1003 x 11264 x 2048 (the splitting warps' loads were exposed, and every tile of x split the same weights again).
//
// The product: persistent pairs of CTAs (clusters of two, cta_group::2), tiles of 256 rows of W (gated: 128 gate and 128 up rows,
// interleaved by 16 in the planes, so that a column's two values lie 16 lanes apart) x bn rows of x, bn a multiple of 16 up to 256
// that follows the number of rows: 1003 rows against 8 tiles of W run as 72 tiles of 112 rows, one wave of the 74 pairs.  A CTA
// holds 128 rows of W and half of the tile's rows of x: 8 KB of operands an instruction of 128 cycles where a CTA alone needs 12.
// Ten warps a CTA:
//   warp 0     one thread loads the planes of a k block by TMA (64-byte rows, 64-byte swizzle; 48 KB a stage at bn = 256, four
//              stages) and announces them on the leader's barriers,
//   warp 1     of the leader: one thread issues the 12 tcgen05.mma (2 k steps x 6 terms) of a block into one of two accumulators,
//   warps 2-9  fetch each finished accumulator (tcgen05.ld) and add it to their sums: a thread owns one column of the result for
//              half of the tile's rows, and stores them at the end of the tile, 32 neighbouring columns a warp.
// The k range is cut into splits of whole blocks (make_plan) that are summed by themselves and then added in split order: that is part of
// the result, and a long K rounds less this way.  Where whole-K tiles leave pairs idle (few rows, narrow matrices) a split is a
// unit of work of its own that leaves its sums in a workspace, and a third kernel adds them; else (sums_stay) a unit has all of K and
// its threads put the sums of the splits before aside in tensor memory.
//
// The numbers are split after a multiplication by 2^24, an accumulator is multiplied by 2^-48 where it is added to the sum: bfloat16 ends at 2^-133 as float32 does
// at 2^-149, so that without it numbers below 2^-110 would lose digits.  With it every float32 below 2^104 is split exactly.
// Larger ones, accumulators above 2^80 and infinities do not give a number this way (an infinity's parts are infinities and
// NaN): a sum that is not finite is taken again, as plain float32 multiply-adds of the operands (plain_dot), so that
// large numbers keep their value and infinities come out where arithmetic gives them.
#include "common.cuh"

KLLM_EXPORT_LAST_ERROR(gemm_f32_tcgen05)

#include "tc5_common.cuh"

namespace {

constexpr int BM = 128;                         // rows of W a CTA holds; a pair's tile has twice as many
constexpr int BN = 256;                         // most rows of x in a tile; accumulators lie this many columns apart
constexpr int BK = 32;                          // a row of a plane is 64 bytes
constexpr int THREADS = 320;
constexpr int FETCH_WARPS = 8;
constexpr int MAX_STAGES = 8;
constexpr int A_PLANE = BM * 64;
constexpr int SMEM_BYTES = 1024 + 4 * 3 * (A_PLANE + BN / 2 * 64);
constexpr int TMEM_COLS = 512;
// Bytes of the planes of one piece of W: with x's planes and the result they stay in the 126 MB of L2.
constexpr long long PLANE_LIMIT = 72LL << 20;

enum Epilogue { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_PARTIAL = 3 };

// K-major operand in the 64-byte swizzled layout: 8-row groups 512 bytes apart, layout type 4
__device__ __forceinline__ uint64_t make_desc64(unsigned addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

constexpr float SCALE = 16777216.f, UNSCALE = 1.f / (SCALE * SCALE);       // 2^24, 2^-48: multiplied exactly

// two numbers, scaled, into their three bfloat16 parts
__device__ __forceinline__ void split2(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    a *= SCALE;
    b *= SCALE;
    p0 = pack_bf16(a, b);
    const float ra = a - __uint_as_float(p0 << 16), rb = b - __uint_as_float(p0 & 0xffff0000u);
    p1 = pack_bf16(ra, rb);
    p2 = pack_bf16(ra - __uint_as_float(p1 << 16), rb - __uint_as_float(p1 & 0xffff0000u));
}

// planes [3][plane_rows][kp] of the rows of src [rows, K] at ld.  With src2 (gated) the two matrices' rows take turns by 16:
// row r of src is plane row 32 (r / 16) + r % 16, row r of src2 is 16 behind it.  Memory bound: 4 bytes read and 6 written
// a number.  BESIDE: launched behind a product that does not read these planes, to run beside it (one CTA on every
// SM beside the product's, more as that one's end): it waits for the kernel before it at its end instead of its beginning, so that what follows it follows that one too.
template <bool BESIDE>
__global__ void __launch_bounds__(256, 6)          // 40 registers: the product's CTA leaves 46 a thread of these
split_kernel(const float* __restrict__ src, const float* __restrict__ src2, int64_t ld, int rows, int K,
             bf16* __restrict__ planes, int64_t plane_rows, int kp) {
    if (!BESIDE) {
        griddep_launch();
        griddep_wait();
    }
    const int pieces = kp / 8;
    const int64_t plane = plane_rows * kp, total = (int64_t)rows * (src2 ? 2 : 1) * pieces;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < total; i0 += 2 * step) {
        float4 u[2], v[2];                                  // two pieces of eight numbers at a time, their loads ahead of the rest
        bf16* o[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int64_t i = min(i0 + e * step, total - 1);
            int64_t r = i / pieces;
            const int k = (int)(i - r * pieces) * 8;
            int64_t to = r;
            const float* from = src;
            if (src2) {
                if (r >= rows) { from = src2; r -= rows; }
                to = (r >> 4) * 32 + (r & 15) + (from == src2 ? 16 : 0);
            }
            const float* p = from + r * ld + k;
            u[e] = __ldg(reinterpret_cast<const float4*>(p));                           // K is a multiple of 4
            v[e] = k + 4 < K ? __ldg(reinterpret_cast<const float4*>(p + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
            o[e] = planes + to * kp + k;
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            if (i0 + e * step >= total) break;
            uint4 q0, q1, q2;
            split2(u[e].x, u[e].y, q0.x, q1.x, q2.x);
            split2(u[e].z, u[e].w, q0.y, q1.y, q2.y);
            split2(v[e].x, v[e].y, q0.z, q1.z, q2.z);
            split2(v[e].z, v[e].w, q0.w, q1.w, q2.w);
            *reinterpret_cast<uint4*>(o[e]) = q0;
            *reinterpret_cast<uint4*>(o[e] + plane) = q1;
            *reinterpret_cast<uint4*>(o[e] + 2 * plane) = q2;
        }
    }
    if (BESIDE) {
        griddep_launch();
        griddep_wait();
    }
}

__device__ __forceinline__ bool is_nan(float v) { return v != v; }
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// x . w as float32 multiply-adds by the 32 lanes of a warp (the same arguments in all of them), for the few elements whose
// six products did not add up to a number (an operand that is not finite or too large, an overflow).  Ends at a NaN,
// which stays one.  A row of 2560 sums over 2048 of k takes 0.3 ms this way; a lane that sums alone took 4.
__device__ __noinline__ float plain_dot(const float* __restrict__ x, const float* __restrict__ w, int K) {
    const int lane = threadIdx.x & 31;
    float s = 0.f;
    for (int k0 = 4 * lane; k0 - 4 * lane < K; k0 += 512) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = k0 + 128 * q;
            if (k < K) {                                                                // K is a multiple of 4
                const float4 u = *reinterpret_cast<const float4*>(x + k), v = *reinterpret_cast<const float4*>(w + k);
                t = fmaf(u.w, v.w, fmaf(u.z, v.z, fmaf(u.y, v.y, fmaf(u.x, v.x, t))));
            }
        }
        s += t;
        if (__any_sync(0xffffffffu, is_nan(s))) break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

struct Args {
    const float *x, *w, *w_up;              // the operands themselves (w: of the piece)
    int64_t ldx, ldw;
    float* y;
    int64_t ldy, split_stride;              // split_stride: elements between the workspace's splits
    int M, N, K, bn, stages;                // N: columns of the result (EPI_PARTIAL: of the workspace)
    int units_of_k, blocks_per_unit, blocks_per_split;      // units a tile's K is cut into; k blocks
    int x_rows, w_rows;                     // rows of a plane of x and of W
    int* status;
};

// ASIDE: a unit has several splits, bn is at most 128
template <int EPI, bool ASIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_f32_tc5_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Args a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_acc_full[2], bar_acc_empty[2];
    __shared__ unsigned s_tmem;
    __shared__ int s_abort;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int bn = a.bn, stages = a.stages;
    const unsigned b_plane = (unsigned)bn * 32, stage_bytes = 3 * (A_PLANE + b_plane);           // bn / 2 rows of 64 bytes
    const int t_tiles = (a.M + bn - 1) / bn, tiles = t_tiles * ((a.w_rows + 2 * BM - 1) / (2 * BM));
    const int units = tiles * a.units_of_k, pairs = gridDim.x >> 1, first = blockIdx.x >> 1;
    const int kblocks = (a.K + BK - 1) / BK;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&bar_acc_full[i], 1); mbar_init(&bar_acc_empty[i], 2 * FETCH_WARPS); }
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
    griddep_wait();
    griddep_launch();                       // not before the wait: what starts now may write planes that the kernels before this one read

    if (warp == 0) {
        // ---- producer: this CTA's rows of W's planes and of x's ----
        int s = 0, issued = 0;
        unsigned ph = 0;
        bool ok = true;
        const unsigned full0 = leader_addr(&bar_full[0]);             // the leader's barriers, 8 bytes apart
        for (int unit = first; ok && unit < units; unit += pairs) {
            const int split = unit / tiles, tile = unit - split * tiles;
            const int t0 = tile % t_tiles * bn + (int)rank * (bn / 2), w0 = (tile / t_tiles * 2 + (int)rank) * BM;
            const int kb0 = split * a.blocks_per_unit, kb1 = min(kblocks, kb0 + a.blocks_per_unit);
            for (int kb = kb0; kb < kb1; kb++) {
                ok = mbar_wait_warp(&bar_empty[s], ph ^ 1u, abort_flag, a.status, 1);
                if (!ok) break;
                if (elect_one()) {
                    const unsigned pa = base + s * stage_bytes, pb = pa + 3 * A_PLANE, bar = full0 + 8u * s;
                    if (rank == 0) mbar_expect_tx(&bar_full[s], 2 * stage_bytes);
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        tma_load_2d_pair(pa + p * A_PLANE, &map_w, kb * BK, p * a.w_rows + w0, bar);
                        tma_load_2d_pair(pb + p * b_plane, &map_x, kb * BK, p * a.x_rows + t0, bar);
                    }
                }
                __syncwarp();
                issued++;
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
        }
        if (ok && !*abort_flag) {
            // the other CTA's products arrive at these barriers: stay until the last has
            for (int j = 0; ok && j < stages; j++) {
                ok = mbar_wait_warp(&bar_empty[s], ph ^ 1u, abort_flag, a.status, 1);
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
        } else if (rank == 0) {
            // copies still in flight must land before the shared memory goes away (the leader waits for both CTAs', the other
            // one is held by the cluster's barrier)
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
            const uint32_t idesc = make_idesc(2 * BM, bn);
            int s = 0, acc = 0;
            unsigned ph = 0, acc_ph = 0;
            bool ok = true;
            for (int unit = first; ok && unit < units; unit += pairs) {
                const int split = unit / tiles;
                const int kb0 = split * a.blocks_per_unit, kb1 = min(kblocks, kb0 + a.blocks_per_unit);
                for (int kb = kb0; kb < kb1; kb++) {
                    ok = mbar_wait_warp(&bar_acc_empty[acc], acc_ph ^ 1u, abort_flag, a.status, 2) &&
                         mbar_wait_warp(&bar_full[s], ph, abort_flag, a.status, 3);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const unsigned d = tmem + (unsigned)(acc * BN);
                        const unsigned pa = base + s * stage_bytes, pb = pa + 3 * A_PLANE;
                        constexpr int TW[6] = {2, 0, 1, 1, 0, 0}, TX[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                        for (int t = 0; t < 6; t++)
#pragma unroll
                            for (int kk = 0; kk < BK / 16; kk++)
                                umma_pair(d, make_desc64(pa + TW[t] * A_PLANE + kk * 32), make_desc64(pb + TX[t] * b_plane + kk * 32),
                                          idesc, kk > 0 || t > 0);
                        umma_commit_pair(&bar_empty[s]);
                        umma_commit_pair(&bar_acc_full[acc]);
                    }
                    __syncwarp();
                    if (++s == stages) { s = 0; ph ^= 1u; }
                    acc ^= 1;
                    if (acc == 0) acc_ph ^= 1u;
                }
            }
        }
    } else {
        // ---- sums and epilogue ----
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const unsigned lane_base = (unsigned)(quarter * 32) << 16;
        const int chunks = (bn + 31) / 32, c_lo = half == 0 ? 0 : (chunks + 1) / 2, mine = half == 0 ? (chunks + 1) / 2 : chunks / 2;
        const bool upper = lane >= 16;
        constexpr int CHUNKS = ASIDE ? 2 : 4;                            // most that a warp has
        int acc = 0;
        unsigned acc_ph = 0;
        bool ok = true;
        for (int unit = first; ok && unit < units; unit += pairs) {
            const int split = unit / tiles, tile = unit - split * tiles;
            const int t0 = tile % t_tiles * bn + c_lo * 32, w0 = (tile / t_tiles * 2 + (int)rank) * BM + quarter * 32;
            const int t_hi = min(tile % t_tiles * bn + bn, a.M);     // rows of x from t0 on that are this tile's
            const int kb0 = split * a.blocks_per_unit, kb1 = min(kblocks, kb0 + a.blocks_per_unit);
            float sum[CHUNKS][32];
            int kb = kb0;
            do {                                                    // one split (ASIDE), or all there is
                const int end = ASIDE ? min(kb1, kb + a.blocks_per_split) : kb1;
#pragma unroll
                for (int c = 0; c < CHUNKS; c++)
#pragma unroll
                    for (int j = 0; j < 32; j++) sum[c][j] = 0.f;
                for (; kb < end; kb++) {
                    ok = mbar_wait(&bar_acc_full[acc], acc_ph, abort_flag, a.status, 4);
                    if (!ok) break;
                    tc_fence_after();
                    const unsigned t = tmem + lane_base + (unsigned)(acc * BN + c_lo * 32);
#pragma unroll
                    for (int c = 0; c < CHUNKS; c++) {
                        if (c >= mine) break;
                        float v[32];
                        tmem_ld32(t + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++) sum[c][j] = fmaf(v[j], UNSCALE, sum[c][j]);      // one rounding, as the add
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(leader_addr(&bar_acc_empty[acc]));
                    acc ^= 1;
                    if (acc == 0) acc_ph ^= 1u;
                }
                ok = __all_sync(0xffffffffu, ok);                   // the warp leaves together or stays for what follows
                if (ASIDE && ok) {
                    unsigned kept = tmem + (unsigned)(BN / 2);      // columns that accumulators of up to 128 leave free
                    asm volatile("" : "+r"(kept));                  // not worth a register in the loop above
                    kept += lane_base + (unsigned)(c_lo * 32);
#pragma unroll
                    for (int c = 0; c < CHUNKS; c++) {
                        if (c >= mine) break;
                        if (kb > a.blocks_per_split) {
                            float v[32];
                            tmem_ld32(kept + c * 32, v);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 32; j++) sum[c][j] = v[j] + sum[c][j];
                        }
                        if (kb < kb1) tmem_st32(kept + c * 32, sum[c]);
                    }
                    tmem_st_wait();
                }
            } while (ASIDE && ok && kb < kb1);
            if (!ok) break;
            // this lane's column; gated: the lower lanes finish the even rows of x, the upper ones the odd rows of the same columns
            const int col = EPI == EPI_SWIGLU ? w0 / 2 + (lane & 15) : w0 + lane;
            const bool live = col < a.N;
            float* y = a.y + (EPI == EPI_PARTIAL ? split * a.split_stride : 0) + (live ? col : 0);
            constexpr int PER = EPI == EPI_SWIGLU ? 16 : 32;        // values a lane stores of a chunk
#pragma unroll
            for (int c = 0; c < CHUNKS; c++) {
                if (c >= mine) break;
                float* s = sum[c];
                auto row = [&](int j) { return t0 + c * 32 + (EPI == EPI_SWIGLU ? 2 * j + (int)upper : j); };
                float zero[4] = {};                                 // 0 times every sum: NaN where one is not finite
#pragma unroll
                for (int j = 0; j < 32; j++) zero[j & 3] = fmaf(s[j], 0.f, zero[j & 3]);
                const bool look = EPI != EPI_PARTIAL &&
                                  __any_sync(0xffffffffu, is_nan((zero[0] + zero[1]) + (zero[2] + zero[3])));
                unsigned odd = 0;                                   // values that are taken again below
                if constexpr (EPI == EPI_SWIGLU) {
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const float got = __shfl_xor_sync(0xffffffffu, upper ? s[2 * j] : s[2 * j + 1], 16);
                        const float g = upper ? got : s[2 * j], u = upper ? s[2 * j + 1] : got;
                        if (look && !(finite(g) && finite(u))) odd |= 1u << j;
                        s[j] = silu_mul(g, u);
                    }
                } else if (look) {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (!finite(s[j])) {
                            odd |= 1u << j;
                            if (EPI == EPI_ADD) s[j] = 0.f;
                        }
                }
                if (EPI == EPI_ADD) {
#pragma unroll
                    for (int q = 0; q < 32; q += 16) {              // loads ahead of the stores
                        float h[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) h[j] = live && row(q + j) < t_hi ? y[(int64_t)row(q + j) * a.ldy] : 0.f;
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (live && row(q + j) < t_hi) y[(int64_t)row(q + j) * a.ldy] = h[j] + s[q + j];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < PER; j++)
                        if (live && row(j) < t_hi) y[(int64_t)row(j) * a.ldy] = s[j];
                }
                if (EPI != EPI_PARTIAL && look) {
                    __syncwarp();
                    if (!live) odd = 0;
                    for (unsigned cols = __ballot_sync(0xffffffffu, odd != 0); cols != 0; cols &= cols - 1) {
                        const int of = __ffs(cols) - 1, at = __shfl_sync(0xffffffffu, col, of), odd_row = of >= 16;
                        for (unsigned left = __shfl_sync(0xffffffffu, odd, of); left != 0; left &= left - 1) {
                            const int j = __ffs(left) - 1;
                            const int r = t0 + c * 32 + (EPI == EPI_SWIGLU ? 2 * j + odd_row : j);
                            if (r >= t_hi) break;                   // rows behind the tile's, in order
                            const float* xr = a.x + (int64_t)r * a.ldx;
                            float* e = a.y + (int64_t)r * a.ldy + at;
                            // a row of NaN, the common case, needs no second look
                            if (is_nan(*xr)) {
                                if (EPI == EPI_ADD && lane == of) *e = *xr;
                                continue;
                            }
                            float v = plain_dot(xr, a.w + (int64_t)at * a.ldw, a.K);
                            if (EPI == EPI_SWIGLU) v = silu_mul(v, plain_dot(xr, a.w_up + (int64_t)at * a.ldw, a.K));
                            if (lane == of) *e = EPI == EPI_ADD ? *e + v : v;
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                                 // nothing of the pair's is under way in either CTA any more
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
}

// The splits' sums, in split order, into the result: stored, added, or (gated: rows of gate and up sums that take turns by 16)
// silu(gate) * up.  Bound by the workspace's bytes, which lie in L2.
template <int EPI>
__global__ void reduce_splits_kernel(float* __restrict__ y, int64_t ldy, const float* __restrict__ ws, int64_t split_stride,
                                     int M, int N, int splits, const Args a) {
    griddep_launch();
    griddep_wait();
    const int n4 = N / 4, ldw = EPI == EPI_SWIGLU ? (N + 15) / 16 * 32 : N, lane = threadIdx.x & 31;
    const int64_t total = (int64_t)M * n4;
    // whole warps walk the elements: a sum that is not finite is taken again by all lanes
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < total; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane, r = i / n4;
        const int c = (int)(i - r * n4) * 4;
        const bool mine = i < total;
        auto sum = [&](const float* p) {
            float4 v = *reinterpret_cast<const float4*>(p);
            for (int s = 1; s < splits; s++) {
                const float4 u = *reinterpret_cast<const float4*>(p + s * split_stride);
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            return v;
        };
        auto again = [&](float4& v, const float* w) {
            float* e = &v.x;
            const bool look = mine && !(finite(v.x) && finite(v.y) && finite(v.z) && finite(v.w)) && !is_nan(a.x[r * a.ldx]);
            if (!__any_sync(0xffffffffu, look)) return;
#pragma unroll
            for (int j = 0; j < 4; j++)
                for (unsigned odd = __ballot_sync(0xffffffffu, look && !finite(e[j])); odd != 0; odd &= odd - 1) {
                    const int of = __ffs(odd) - 1;
                    const float d = plain_dot(a.x + __shfl_sync(0xffffffffu, r, of) * a.ldx,
                                                    w + (__shfl_sync(0xffffffffu, c, of) + j) * a.ldw, a.K);
                    if (lane == of) e[j] = d;
                }
        };
        const float* part = ws + r * ldw + (EPI == EPI_SWIGLU ? (c >> 4) * 32 + (c & 15) : c);
        float4 v = mine ? sum(part) : make_float4(0.f, 0.f, 0.f, 0.f);
        again(v, a.w);
        float4 u = v;
        if (EPI == EPI_SWIGLU) {
            if (mine) u = sum(part + 16);
            again(u, a.w_up);
        }
        if (!mine) continue;
        float4* o = reinterpret_cast<float4*>(y + r * ldy + c);
        if (EPI == EPI_ADD) {
            const float4 h = *o;
            v.x += h.x; v.y += h.y; v.z += h.z; v.w += h.w;
        } else if (EPI == EPI_SWIGLU) {
            v.x = silu_mul(v.x, u.x); v.y = silu_mul(v.y, u.y); v.z = silu_mul(v.z, u.z); v.w = silu_mul(v.w, u.w);
        }
        *o = v;
    }
}

// ---- host side -----------------------------------------------------------------

int planes_map(CUtensorMap* out, const bf16* planes, int64_t rows, int K, int kp, int box_rows) {
    EncodeTiledFn fn = encoder();
    if (!fn) KLLM_FAIL("gemm float32 (tcgen05): the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)kp * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)planes, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) KLLM_FAIL("gemm float32 (tcgen05): tensor map for %lld x %d planes refused: %d", (long long)rows, K, (int)r);
    return 0;
}

template <int EPI, bool ASIDE>
int launch_kernel(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, cudaStream_t s) {
    static bool attr_set = false;
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc5_kernel<EPI, ASIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) {
            snprintf(g_kllm_err, sizeof(g_kllm_err), "gemm float32 (tcgen05): %d bytes of shared memory refused: %s", SMEM_BYTES,
                     cudaGetErrorString(e));
            return (int)e;
        }
        attr_set = true;
    }
    const long long units = (long long)((a.M + a.bn - 1) / a.bn) * ((a.w_rows + 2 * BM - 1) / (2 * BM)) * a.units_of_k, pairs = sm_count() / 2;
    const int grid = 2 * (int)(units < pairs ? units : pairs);
    kllm_launch((gemm_f32_tc5_kernel<EPI, ASIDE>), dim3(grid), dim3(THREADS), SMEM_BYTES, s, mw, mx, a);
    KLLM_LAUNCH_STATUS();
}

template <int EPI>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, cudaStream_t s) {
    return a.blocks_per_split < a.blocks_per_unit ? launch_kernel<EPI, true>(mw, mx, a, s) : launch_kernel<EPI, false>(mw, mx, a, s);
}

// beside: behind a product, to run on the SMs that it occupies
int launch_split(bool beside, const float* src, const float* src2, int64_t ld, int rows, int K, bf16* planes, int64_t plane_rows, int kp,
                 cudaStream_t s) {
    const int64_t work = (int64_t)rows * (src2 ? 2 : 1) * (kp / 8);
    const int64_t blocks = (work + 511) / 512, most = 8LL * sm_count();
    const dim3 grid((unsigned)(blocks < most ? blocks : most));
    if (beside) kllm_launch((split_kernel<true>), grid, dim3(256), 0, s, src, src2, ld, rows, K, planes, plane_rows, kp);
    else kllm_launch((split_kernel<false>), grid, dim3(256), 0, s, src, src2, ld, rows, K, planes, plane_rows, kp);
    KLLM_LAUNCH_STATUS();
}

template <int EPI>
int launch_reduce(float* y, int64_t ldy, const float* ws, int64_t split_stride, int M, int N, int splits, const Args& a, cudaStream_t s) {
    const int64_t blocks = ((int64_t)M * (N / 4) + 255) / 256, most = 8LL * sm_count();
    kllm_launch((reduce_splits_kernel<EPI>), dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, s, y, ldy, ws, split_stride,
                M, N, splits, a);
    KLLM_LAUNCH_STATUS();
}

// How a product is cut: W in pieces of `piece` output columns (whole tiles, the last piece takes the rest), a piece's K
// in `splits` ranges, which one unit sums with the earlier ones put aside (sums_stay) or each a unit of its own.
struct Plan {
    int piece, splits, kp;
    bool sums_stay;
    int64_t x_bytes, w_bytes, ws_bytes;
};
int64_t up256(int64_t b) { return (b + 255) / 256 * 256; }

// Rows of x in a tile: an instruction's time goes with them (from about 96 on), so the least waves x rows wins, the wider tile
// at a tie.  w_tiles: tiles of W, each `splits` units of work.
int pick_bn(int M, int w_tiles, int splits) {
    const long long pairs = sm_count() / 2;
    long long best = -1;
    int best_bn = BN;
    for (int bn = BN; bn >= 16; bn -= 16) {
        const long long units = (long long)w_tiles * splits * ((M + bn - 1) / bn), waves = (units + pairs - 1) / pairs;
        const long long cost = waves * (bn > 96 ? bn : 96);
        if (best < 0 || cost < best) { best = cost; best_bn = bn; }
    }
    return best_bn;
}

// Whether tiles of whole K, their rows of x chosen to fit, do better than a unit a split with the splits' workspace and the kernel behind:
// they keep the pairs busy for most of the time, their splits' sums fit beside the accumulators, and they take no more than 1.1
// times as long, by a k block's 0.22 + 0.0036 bn us (5632 x 2048, whole K: 700 rows in tiles of 80 0.53, 1003 of 112 0.61, 2048 of 240
// 1.1), 1.5 for a split's sums to the workspace, and 2.4 and 5 MB a us for the kernel behind.  5632 x 2048, 700 rows: 112 us whole,
// 93 by splits; 2048 x 2560, 845 rows: 51 and 59.
bool whole_k_pays(int M, int w_tiles, int kblocks, int splits) {
    const int pairs = sm_count() / 2, bn = pick_bn(M, w_tiles, 1), bn_split = pick_bn(M, w_tiles, splits);
    auto waves = [&](int rows, int units) { return ((long long)w_tiles * units * ((M + rows - 1) / rows) + pairs - 1) / pairs; };
    auto block = [](int rows) { return 0.22 + 0.0036 * (rows > 64 ? rows : 64); };
    if (bn > BN / 2 || 10.0 * w_tiles * M < 6.0 * pairs * waves(bn, 1) * (bn > 96 ? bn : 96)) return false;
    const double whole = waves(bn, 1) * kblocks * block(bn);
    const double split = waves(bn_split, splits) * ((kblocks + splits - 1) / splits * block(bn_split) + 1.5) + 2.4 +
                         8e-6 * splits * (double)M * w_tiles * (2 * BM) / 5;
    return whole <= 1.1 * split;
}

// The splits decide in which order a result is added up, so their number does not follow the way the kernel is built: the count is that
// of tiles of 128 rows of x, one for every SM at a time.  Least is a sum of k blocks (0.8 us of such a tile) in which a tile costs its
// blocks and 3, a launch 3, and sums are written and read at 4 MB a block's time.
Plan make_plan(int M, int N, int K, int epilogue) {
    Plan p;
    const bool gated = epilogue == EPI_SWIGLU;
    const int nout = gated ? BN / 2 : BN, sms = sm_count(), kblocks = (K + BK - 1) / BK;
    p.kp = (K + 7) / 8 * 8;
    const long long m_tiles = (M + BM - 1) / BM, n_tiles = (N + nout - 1) / nout;
    long long most = PLANE_LIMIT / (6LL * p.kp * BN);
    if (most < 1) most = 1;
    if (most > n_tiles) most = n_tiles;
    double best = -1;
    p.piece = N;
    p.splits = 1;
    for (long long c = most; c >= 1; c--) {
        const long long full = n_tiles / c, rest = n_tiles - full * c;
        for (int s = 1; s <= 16; s++) {
            const int per = (kblocks + s - 1) / s;
            if (s > 1 && (per < 6 || (kblocks + per - 1) / per != s)) continue;
            auto cost = [&](long long tiles) {
                const double sums = s > 1 ? 3.0 + 8.0 * s * (double)M * tiles * BN / 4e6 : 0.0;
                return (double)((m_tiles * tiles * s + sms - 1) / sms) * (per + 3) + 3.0 + sums;
            };
            const double all = full * cost(c) + (rest ? cost(rest) : 0.0);
            if (best < 0 || all < best) { best = all; p.piece = c == n_tiles ? N : (int)c * nout; p.splits = s; }
        }
    }
    const int64_t cols = gated ? (p.piece + 15) / 16 * 32 : p.piece;
    p.x_bytes = up256(6LL * M * p.kp);
    p.w_bytes = up256(6LL * cols * p.kp);
    p.sums_stay = p.splits > 1 && p.piece == N && whole_k_pays(M, (int)n_tiles, kblocks, p.splits);
    p.ws_bytes = p.splits > 1 && !p.sums_stay ? up256(4LL * p.splits * M * cols) : 0;
    return p;
}

}  // namespace

// Bytes of workspace that the product of these sizes wants (256-byte aligned, its own until it has run).
extern "C" int kllm_gemm_f32_tcgen05_workspace(int M, int N, int K, int epilogue, int64_t* bytes) {
    if (M <= 0 || N <= 0 || K <= 0) { *bytes = 0; return 0; }
    const Plan p = make_plan(M, N, K, epilogue);
    *bytes = p.x_bytes + (p.piece < N ? 2 : 1) * p.w_bytes + p.ws_bytes;
    return 0;
}

// How the product of these sizes is cut: output columns of a piece of W (the last piece takes the rest), ranges of k.
extern "C" int kllm_gemm_f32_tcgen05_plan(int M, int N, int K, int epilogue, int* piece, int* splits) {
    if (M <= 0 || N <= 0 || K <= 0) { *piece = *splits = 0; return 0; }
    const Plan p = make_plan(M, N, K, epilogue);
    *piece = p.piece;
    *splits = p.splits;
    return 0;
}

// 1 if the kernel takes these sizes and addresses, else 0.
extern "C" int kllm_gemm_f32_tcgen05_fits(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* w_up, int M,
                                          int N, int K, const void* y, int64_t ldy, int epilogue) {
    if (M <= 0 || N <= 0 || K <= 0 || epilogue < 0 || epilogue > 2) return 0;
    if ((K & 3) || (N & 3) || (ldx & 3) || (ldw & 3) || (ldy & 3)) return 0;           // 16-byte loads and stores
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)w_up & 15) || ((uintptr_t)y & 15)) return 0;
    if (ldx < K || ldw < K || ldy < N) return 0;
    if (epilogue == EPI_SWIGLU && !w_up) return 0;
    if (M > (1 << 28) || N > (1 << 28)) return 0;                                       // plane rows are 32-bit coordinates
    const long long tiles = ((long long)(M + BM - 1) / BM) * ((N + BN / 2 - 1) / (BN / 2));
    return tiles * 16 < (1LL << 31) ? 1 : 0;
}

// epilogue 0: y = x W^T, 1: y += x W^T, 2: y = silu(x W^T) * (x W_up^T).  ws: kllm_gemm_f32_tcgen05_workspace bytes.
// status: device int that a wait which ran out sets (1: stage free, 2: accumulator free, 3: stage full, 4: accumulator full).
extern "C" int kllm_gemm_f32_tcgen05(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* w_up, int M, int N,
                                     int K, void* y, int64_t ldy, int epilogue, void* ws, int* status, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!kllm_gemm_f32_tcgen05_fits(x, ldx, w, ldw, w_up, M, N, K, y, ldy, epilogue) || ((uintptr_t)ws & 255) || !ws)
        KLLM_FAIL("gemm float32 (tcgen05): sizes %d x %d x %d, strides %lld/%lld/%lld or an address not taken (sizes and "
                  "strides multiples of 4, 16-byte aligned addresses)", M, N, K, (long long)ldx, (long long)ldw, (long long)ldy);
    const Plan p = make_plan(M, N, K, epilogue);
    const bool gated = epilogue == EPI_SWIGLU;
    const int kblocks = (K + BK - 1) / BK, pieces = (N + p.piece - 1) / p.piece;
    bf16* px = (bf16*)ws;
    bf16* pw[2] = {(bf16*)((char*)ws + p.x_bytes), (bf16*)((char*)ws + p.x_bytes + (pieces > 1 ? p.w_bytes : 0))};
    float* part = (float*)((char*)pw[1] + p.w_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    int r = launch_split(false, (const float*)x, nullptr, ldx, M, K, px, M, p.kp, s);
    if (r) return r;
    Args a;
    const bool whole = p.splits == 1 || p.sums_stay;
    a.M = M; a.K = K; a.blocks_per_split = (kblocks + p.splits - 1) / p.splits; a.status = status;
    a.units_of_k = whole ? 1 : p.splits;
    a.blocks_per_unit = whole ? kblocks : a.blocks_per_split;
    a.x_rows = M; a.x = (const float*)x; a.ldx = ldx; a.ldw = ldw;
    // The last piece, the shortest, comes first: its splitting is the one that no product hides.
    for (int i = 0; i < pieces; i++) {
        const int n0 = (i == 0 ? pieces - 1 : i - 1) * p.piece, cols = N - n0 < p.piece ? N - n0 : p.piece;
        float* yp = (float*)y + n0;
        bf16* planes = pw[i & 1];
        a.w_rows = gated ? (cols + 15) / 16 * 32 : cols;
        a.w = (const float*)w + n0 * ldw; a.w_up = gated ? (const float*)w_up + n0 * ldw : nullptr;
        // Beside the product before, which started when its own planes were ready, that is when the product that read this
        // buffer was over; behind split sums' last kernel as usual.
        r = launch_split(i > 0 && whole, a.w, a.w_up, ldw, cols, K, planes, a.w_rows, p.kp, s);
        if (r) return r;
        a.bn = pick_bn(M, (a.w_rows + 2 * BM - 1) / (2 * BM), a.units_of_k);
        a.stages = (SMEM_BYTES - 1024) / (3 * (A_PLANE + a.bn * 32));
        if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
        CUtensorMap mw, mx;
        r = planes_map(&mw, planes, 3LL * a.w_rows, K, p.kp, BM);
        if (!r) r = planes_map(&mx, px, 3LL * M, K, p.kp, a.bn / 2);
        if (r) return r;
        if (whole) {
            a.N = cols; a.y = yp; a.ldy = ldy; a.split_stride = 0;
            r = epilogue == EPI_STORE ? launch<EPI_STORE>(mw, mx, a, s) : epilogue == EPI_ADD ? launch<EPI_ADD>(mw, mx, a, s)
                                                                                             : launch<EPI_SWIGLU>(mw, mx, a, s);
        } else {
            a.N = a.w_rows; a.y = part; a.ldy = a.w_rows; a.split_stride = (int64_t)M * a.w_rows;
            r = launch<EPI_PARTIAL>(mw, mx, a, s);
            if (r) return r;
            r = epilogue == EPI_STORE ? launch_reduce<EPI_STORE>(yp, ldy, part, a.split_stride, M, cols, p.splits, a, s)
                : epilogue == EPI_ADD ? launch_reduce<EPI_ADD>(yp, ldy, part, a.split_stride, M, cols, p.splits, a, s)
                                      : launch_reduce<EPI_SWIGLU>(yp, ldy, part, a.split_stride, M, cols, p.splits, a, s);
        }
        if (r) return r;
    }
    return 0;
}
