// Causal grouped-query attention of float32 portions over the paged cache on the tensor cores, at float32 accuracy.
//
// The CUDA cores reach a quarter of their rate on this (csrc/attention_simt.cu: 257 us for 1003 tokens, 32 heads of 64 on
// 4 kv heads, 17 TFLOP/s).  Here every number of Q, K, V and of the probabilities is the sum of three bfloat16 numbers,
//     v = v0 + v1 + v2,  v0 = bf16(v), v1 = bf16(v - v0), v2 = bf16(v - v0 - v1),
// and a product of two is the six products whose parts matter at 24 bits (x2 y0 + x0 y2 + x1 y1 + x1 y0 + x0 y1, then x0 y0); x1 y2,
// x2 y1 and x2 y2, below 2^-24 of it, are left out.
// The five small ones and the large one have accumulators of their own that hold one score, or one key tile of one output, and
// are then added by the rounding adds of the CUDA cores: what the tensor cores cut off in their accumulation cannot drift over a
// long context.
//
// mma.sync and not tcgen05: the probabilities' parts go from the scores' registers straight into the second product's operand
// registers, and 64 rows x 64 keys x 64 dims in twelve products is too little work a tile to pay for trips through tensor memory.
// A CTA of four warps has a tile of up to 64 rows, a row being one (query token, head), 16 rows a warp.  Key tiles of KT keys come
// as float32 by asynchronous copies while the tile before is being multiplied, all threads split them into three bfloat16 planes
// (16-byte pieces, exclusive-or swizzled), and the warps read the planes with ldmatrix.  Two CTAs an SM at head size 64 (104 KB
// each), one at 128.  Measured: 1003 tokens, 32 heads of 64 on 4 kv heads 121 us a layer (the CUDA cores 257), the tensor cores'
// pipe busy for 38 % of it, DRAM for 1 %: two CTAs of four warps are all that 222 registers and 104 KB leave an SM, and they
// split every key tile between two meetings of the CTA.  Relative error of the outputs about half the multiply-add kernel's.
//
// Masks, sinks, slopes, window and kept keys as in attention_simt.cu, expf and one division at the end too.  V is split after a
// multiplication by 2^24, which the division takes back, so that small values keep their digits.  An operand that is not finite,
// or too large for the parts, makes a score or an output that is not finite; a CTA that finds one computes its rows again by
// plain multiply-adds, visible key by visible key (plain_rows), where infinities and NaN come out as arithmetic gives them.
#include "common.cuh"

KLLM_EXPORT_LAST_ERROR(attention_f32_mma)

namespace {

constexpr int ROWS = 64, THREADS = 128, LINE = 64;      // LINE: granule of the key line, as in attention_simt.cu
constexpr float VSCALE = 16777216.f, VUNSCALE = 1.f / VSCALE;
constexpr int key_tile(int hd) { return 4096 / hd; }    // 64 or 32 keys
constexpr size_t smem_bytes(int hd) { return (size_t)3 * ROWS * hd * 2 + (size_t)2 * key_tile(hd) * hd * (3 * 2 + 4); }

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// two numbers into their three bfloat16 parts
__device__ __forceinline__ void split2(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    p0 = pack2(a, b);
    const float ra = a - __uint_as_float(p0 << 16), rb = b - __uint_as_float(p0 & 0xffff0000u);
    p1 = pack2(ra, rb);
    p2 = pack2(ra - __uint_as_float(p1 << 16), rb - __uint_as_float(p1 & 0xffff0000u));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// the six products of a step of 16: the small ones into `lo`, the large one into `hi`
__device__ __forceinline__ void mma6(float (&lo)[4], float (&hi)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int t) {
    mma_bf16(lo, a[2], b[0][2 * t], b[0][2 * t + 1]);
    mma_bf16(hi, a[0], b[0][2 * t], b[0][2 * t + 1]);
    mma_bf16(lo, a[0], b[2][2 * t], b[2][2 * t + 1]);
    mma_bf16(lo, a[1], b[1][2 * t], b[1][2 * t + 1]);
    mma_bf16(lo, a[1], b[0][2 * t], b[0][2 * t + 1]);
    mma_bf16(lo, a[0], b[1][2 * t], b[1][2 * t + 1]);
}
// 16-byte piece c of row r of a plane of rows of HD bfloat16
template <int HD>
__device__ __forceinline__ unsigned piece(int r, int c) { return (unsigned)(r * HD * 2 + ((c ^ (r & 7)) << 4)); }

// eight numbers, times `scale`, into piece c of row r of three planes that lie `plane` bytes apart
template <int HD>
__device__ __forceinline__ void put_parts(unsigned char* planes, int plane, int r, int c, float4 u, float4 v, float scale) {
    uint4 p0, p1, p2;
    split2(u.x * scale, u.y * scale, p0.x, p1.x, p2.x);
    split2(u.z * scale, u.w * scale, p0.y, p1.y, p2.y);
    split2(v.x * scale, v.y * scale, p0.z, p1.z, p2.z);
    split2(v.z * scale, v.w * scale, p0.w, p1.w, p2.w);
    unsigned char* p = planes + piece<HD>(r, c);
    *reinterpret_cast<uint4*>(p) = p0;
    *reinterpret_cast<uint4*>(p + plane) = p1;
    *reinterpret_cast<uint4*>(p + 2 * plane) = p2;
}

struct Args {
    float* out;                 // [tokens, n_heads * HD]
    const float* q;
    int64_t q_stride;
    const float *kcache, *vcache;       // [pages, n_kv, page_size, HD]
    const int *q_start, *start_pos, *block_table;
    int max_blocks, n_requests, n_heads, n_kv, page_size, window, qt, segment, keep;
    float scale;
    const float *slopes, *sinks;
};

struct Tile {                   // what a CTA has: rows (token tok0 + r / gs, head g * gs + r % gs), r < R, of request s
    int s, g, gs, R, tok0, p0;
};

// The tile's rows by multiply-adds, one warp a row, its visible keys one after the other.
template <int HD>
__device__ __noinline__ void plain_rows(const Args& a, const Tile& t) {
    constexpr int D = HD / 32;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < t.R; r += THREADS / 32) {
        const int tok = t.tok0 + r / t.gs, h = t.g * t.gs + r % t.gs, p = t.p0 + r / t.gs;
        float q[D], o[D];
#pragma unroll
        for (int i = 0; i < D; i++) {
            q[i] = a.q[(int64_t)tok * a.q_stride + (int64_t)h * HD + lane + 32 * i];
            o[i] = 0.f;
        }
        int lo = a.window > 0 && p + 1 > a.window ? p + 1 - a.window : 0;
        if (a.segment > 0) lo = max(lo, p - p % a.segment);
        float m = a.sinks ? a.sinks[h] : -INFINITY, l = a.sinks ? 1.f : 0.f;
        const float slope = a.slopes ? a.slopes[h] : 0.f;
        for (int k = min(a.keep, lo) > 0 ? 0 : lo; k <= p; k++) {
            if (k >= a.keep && k < lo) k = lo;
            const int lp = k / a.page_size;
            const int64_t at = (((int64_t)a.block_table[(int64_t)t.s * a.max_blocks + lp] * a.n_kv + t.g) * a.page_size + (k - lp * a.page_size)) * HD;
            float sc = 0.f;
#pragma unroll
            for (int i = 0; i < D; i++) sc = fmaf(q[i], a.kcache[at + lane + 32 * i], sc);
            sc = warp_sum(sc) * a.scale + slope * (float)(k - p);
            const float m_new = fmaxf(m, sc);
            // while the scores seen are all -inf the maximum is no base: such a key weighs 0, and one whose score is NaN stays NaN
            // (fmaxf passes it over)
            const float alpha = m_new == -INFINITY ? 1.f : expf(m - m_new), w = expf(sc - (m_new == -INFINITY ? 0.f : m_new));
            l = l * alpha + w;
            m = m_new;
#pragma unroll
            for (int i = 0; i < D; i++) o[i] = o[i] * alpha + w * a.vcache[at + lane + 32 * i];
        }
#pragma unroll
        for (int i = 0; i < D; i++) a.out[((int64_t)tok * a.n_heads + h) * HD + lane + 32 * i] = o[i] / l;
    }
}

template <int HD>
__global__ void __launch_bounds__(THREADS, HD == 64 ? 2 : 1)
attn_f32_mma_kernel(const Args a) {
    constexpr int KT = key_tile(HD), KS = HD / 16, NP = KT / 16;     // k steps of the first product, 16-key groups of a tile
    constexpr int C8 = HD / 8;                                       // 8-number pieces of a row
    constexpr int Q_PLANE = ROWS * HD * 2, K_PLANE = KT * HD * 2;
    constexpr bool HOLD_Q = HD == 64;                                // Q's parts stay in registers (48 of them)
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* Qp = smem;
    unsigned char* Kp = Qp + 3 * Q_PLANE;
    unsigned char* Vp = Kp + 3 * K_PLANE;
    float* Kf = reinterpret_cast<float*>(Vp + 3 * K_PLANE);
    float* Vf = Kf + KT * HD;
    griddep_wait();
    griddep_launch();

    // which request and which of its tiles this CTA has: the longest key ranges first, every kv head's share of a tile beside
    // each other
    Tile t;
    t.g = blockIdx.x % a.n_kv;
    int tile = (gridDim.x - 1 - blockIdx.x) / a.n_kv, n_new = 0;
    bool found = false;
    for (t.s = 0; t.s < a.n_requests; t.s++) {
        n_new = a.q_start[t.s + 1] - a.q_start[t.s];
        const int nt = (n_new + a.qt - 1) / a.qt;
        if (tile < nt) { found = true; break; }
        tile -= nt;
    }
    if (!found) return;
    const int q0 = tile * a.qt, nq = min(a.qt, n_new - q0);
    t.gs = a.n_heads / a.n_kv;
    t.R = nq * t.gs;
    t.tok0 = a.q_start[t.s] + q0;
    t.p0 = a.start_pos[t.s] + q0;
    int lo_all = (a.window > 0 && t.p0 + 1 > a.window) ? t.p0 + 1 - a.window : 0;
    if (a.segment > 0) lo_all = max(lo_all, t.p0 - t.p0 % a.segment);
    const KeyLine line(lo_all, t.p0 + nq, a.keep, LINE);
    const int total = line.total();
    const int* table = a.block_table + (int64_t)t.s * a.max_blocks;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane & 3;

    auto copy_tile = [&](int v0) {
        const int key0 = line.key(v0), lim = line.limit(v0);
        constexpr int TPK = THREADS / KT;                            // threads of a key
        const int k = tid / TPK, kp = key0 + k;
        const bool ok = kp < lim;
        int64_t at = 0;
        if (ok) {
            const int lp = kp / a.page_size;
            at = (((int64_t)table[lp] * a.n_kv + t.g) * a.page_size + (kp - lp * a.page_size)) * HD;
        }
        const int bytes = ok ? 16 : 0;                               // 0: the 16 bytes are filled with zeros
        const unsigned dk = (unsigned)__cvta_generic_to_shared(Kf + k * HD), dv = (unsigned)__cvta_generic_to_shared(Vf + k * HD);
#pragma unroll
        for (int c = tid % TPK; c < HD / 4; c += TPK) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dk + c * 16), "l"(a.kcache + at + 4 * c), "r"(bytes));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dv + c * 16), "l"(a.vcache + at + 4 * c), "r"(bytes));
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    copy_tile(0);
    for (int e = tid; e < ROWS * C8; e += THREADS) {
        const int r = e / C8, c = e - r * C8;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
        if (r < t.R) {
            const float* p = a.q + (int64_t)(t.tok0 + r / t.gs) * a.q_stride + (int64_t)(t.g * t.gs + r % t.gs) * HD + 8 * c;
            u = __ldg(reinterpret_cast<const float4*>(p));
            v = __ldg(reinterpret_cast<const float4*>(p + 4));
        }
        put_parts<HD>(Qp, Q_PLANE, r, c, u, v, 1.f);
    }
    __syncthreads();

    // this thread's two rows of its warp's sixteen
    const int row0 = warp * 16 + (lane >> 2);
    float m[2], l[2], slope[2];
    int pos[2], wlo[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int r = row0 + 8 * i;
        const bool live = r < t.R;
        m[i] = a.sinks && live ? a.sinks[t.g * t.gs + r % t.gs] : -INFINITY;
        l[i] = a.sinks && live ? 1.f : 0.f;
        pos[i] = live ? t.p0 + r / t.gs : -1;                        // -1: no key is visible to a row that does not exist
        slope[i] = a.slopes && live ? a.slopes[t.g * t.gs + r % t.gs] : 0.f;
        wlo[i] = a.window > 0 ? pos[i] + 1 - a.window : 0;
        if (a.segment > 0 && live) wlo[i] = max(wlo[i], pos[i] - pos[i] % a.segment);
    }
    const int last_row = min(t.R, warp * 16 + 16) - 1;
    const int max_pos = warp * 16 < t.R ? t.p0 + last_row / t.gs : -1;         // no row of this warp sees a key behind it
    // ldmatrix addresses: lanes 0-15 the rows, 16-31 the same rows 8 numbers further (Q); V by keys likewise; K: lanes 8-15 and
    // 24-31 the same keys 8 numbers further
    const unsigned q_base = (unsigned)__cvta_generic_to_shared(Qp), k_base = (unsigned)__cvta_generic_to_shared(Kp),
                   v_base = (unsigned)__cvta_generic_to_shared(Vp);
    auto load_q = [&](uint32_t (&f)[3][4], int ks) {
#pragma unroll
        for (int p = 0; p < 3; p++) ldsm4(f[p], q_base + p * Q_PLANE + piece<HD>(warp * 16 + (lane & 15), 2 * ks + (lane >> 4)));
    };
    uint32_t qf[HOLD_Q ? KS : 1][3][4];
    if (HOLD_Q) {
#pragma unroll
        for (int ks = 0; ks < KS; ks++) load_q(qf[HOLD_Q ? ks : 0], ks);
    }
    float o[C8][4];
#pragma unroll
    for (int d = 0; d < C8; d++)
#pragma unroll
        for (int j = 0; j < 4; j++) o[d][j] = 0.f;
    float zero = 0.f;                                                // 0 times every score: NaN once one was not finite

    for (int v0 = 0; v0 < total; v0 += KT) {
        const int key0 = line.key(v0), lim = line.limit(v0);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                             // the tile has arrived, the planes are no longer read
        for (int e = tid; e < KT * C8; e += THREADS) {
            const int r = e / C8, c = e - r * C8;
            const float4* k = reinterpret_cast<const float4*>(Kf + r * HD + 8 * c);
            const float4* v = reinterpret_cast<const float4*>(Vf + r * HD + 8 * c);
            put_parts<HD>(Kp, K_PLANE, r, c, k[0], k[1], 1.f);
            put_parts<HD>(Vp, K_PLANE, r, c, v[0], v[1], VSCALE);
        }
        __syncthreads();
        if (v0 + KT < total) copy_tile(v0 + KT);
        const int groups = min(NP, (min(lim, max_pos + 1) - key0 + 15) / 16);  // 16-key groups that this warp's rows see any of
        if (groups <= 0) continue;

        float s[NP][2][4];
#pragma unroll
        for (int n = 0; n < NP; n++) {
            if (n >= groups) {
#pragma unroll
                for (int j = 0; j < 8; j++) s[n][j >> 2][j & 3] = 0.f;
                continue;
            }
            float small[2][4] = {};
#pragma unroll
            for (int j = 0; j < 8; j++) s[n][j >> 2][j & 3] = 0.f;
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                uint32_t kf[3][4];
#pragma unroll
                for (int p = 0; p < 3; p++)
                    ldsm4(kf[p], k_base + p * K_PLANE + piece<HD>(16 * n + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)));
                if (!HOLD_Q) load_q(qf[0], ks);
#pragma unroll
                for (int h = 0; h < 2; h++) mma6(small[h], s[n][h], qf[HOLD_Q ? ks : 0], kf, h);
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                s[n][j >> 2][j & 3] += small[j >> 2][j & 3];
                zero = fmaf(s[n][j >> 2][j & 3], 0.f, zero);
            }
        }
        // ---- the running softmax of the thread's two rows ----
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float mx = -INFINITY;
#pragma unroll
            for (int n = 0; n < NP; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int kp = key0 + 16 * n + 8 * (j >> 1) + 2 * quad + (j & 1);
                    float& x = s[n][j >> 1][2 * i + (j & 1)];
                    const bool vis = kp < lim && kp <= pos[i] && (kp >= wlo[i] || kp < a.keep);
                    x = vis ? x * a.scale + slope[i] * (float)(kp - pos[i]) : -INFINITY;
                    mx = fmaxf(mx, x);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m[i], mx);
            const float base = m_new == -INFINITY ? 0.f : m_new;    // nothing seen yet: every exponential below is 0
            alpha[i] = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < NP; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float& x = s[n][j >> 1][2 * i + (j & 1)];
                    x = expf(x - base);
                    sum += x;
                }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[i] = l[i] * alpha[i] + sum;
            m[i] = m_new;
        }
        // ---- probabilities x values ----
        uint32_t pf[NP][3][4];
#pragma unroll
        for (int n = 0; n < NP; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                split2(s[n][h][0], s[n][h][1], pf[n][0][2 * h], pf[n][1][2 * h], pf[n][2][2 * h]);
                split2(s[n][h][2], s[n][h][3], pf[n][0][2 * h + 1], pf[n][1][2 * h + 1], pf[n][2][2 * h + 1]);
            }
#pragma unroll
        for (int d = 0; d < C8; d += 2) {
            float hi[2][4] = {}, small[2][4] = {};
#pragma unroll
            for (int n = 0; n < NP; n++) {
                if (n >= groups) break;
                uint32_t vf[3][4];
#pragma unroll
                for (int p = 0; p < 3; p++) ldsm4_t(vf[p], v_base + p * K_PLANE + piece<HD>(16 * n + (lane & 15), d + (lane >> 4)));
#pragma unroll
                for (int h = 0; h < 2; h++) mma6(small[h], hi[h], pf[n], vf, h);
            }
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int j = 0; j < 4; j++) o[d + h][j] = fmaf(o[d + h][j], alpha[j >> 1], hi[h][j] + small[h][j]);
        }
    }

    // ---- the end: one division, unless something was not finite ----
#pragma unroll
    for (int d = 0; d < C8; d++)
#pragma unroll
        for (int j = 0; j < 4; j++) zero = fmaf(o[d][j], 0.f, zero);
    if (__syncthreads_or(zero != zero)) {
        plain_rows<HD>(a, t);
        return;
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int r = row0 + 8 * i;
        if (r >= t.R) continue;
        const float inv = 1.f / l[i];
        float* out = a.out + ((int64_t)(t.tok0 + r / t.gs) * a.n_heads + t.g * t.gs + r % t.gs) * HD;
#pragma unroll
        for (int d = 0; d < C8; d++)
            *reinterpret_cast<float2*>(out + 8 * d + 2 * quad) =
                make_float2(o[d][2 * i] * inv * VUNSCALE, o[d][2 * i + 1] * inv * VUNSCALE);
    }
}

template <int HD>
int launch(const Args& a, int max_tiles, cudaStream_t s) {
    auto kern = attn_f32_mma_kernel<HD>;
    static bool raised = false;
    if (!raised) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(HD));
        if (e != cudaSuccess) {
            snprintf(g_kllm_err, sizeof(g_kllm_err), "attention (float32, mma): shared memory limit: %s", cudaGetErrorString(e));
            return (int)e;
        }
        raised = true;
    }
    kllm_launch(kern, dim3(max_tiles * a.n_kv), dim3(THREADS), smem_bytes(HD), s, a);
    KLLM_LAUNCH_STATUS();
}

}  // namespace

// 1 if the kernel takes these sizes and addresses, else 0 (csrc/attention_simt.cu takes them then).
extern "C" int kllm_attention_f32_mma_fits(const void* out, const void* q, int64_t q_stride, const void* kcache, const void* vcache,
                                           int n_heads, int n_kv, int hd) {
    if ((hd != 64 && hd != 128) || n_kv <= 0 || n_heads <= 0 || n_heads % n_kv || n_heads / n_kv > ROWS || (q_stride & 3)) return 0;
    return (((uintptr_t)out | (uintptr_t)q | (uintptr_t)kcache | (uintptr_t)vcache) & 15) ? 0 : 1;
}

// Arguments as in kllm_attention_simt with chunk 0, in float32 with values as wide as keys and as many heads of them.
extern "C" int kllm_attention_f32_mma(void* out, const void* q, int64_t q_stride, const void* kcache, const void* vcache,
                                      const int* q_start, const int* start_pos, const int* block_table, int max_blocks, int n_requests,
                                      int max_tiles, int n_heads, int n_kv, int hd, int page_size, int window, float scale, int qt,
                                      const float* slopes, const float* sinks, int segment, int keep, void* stream) {
    if (n_requests <= 0 || max_tiles <= 0) return 0;
    if (!kllm_attention_f32_mma_fits(out, q, q_stride, kcache, vcache, n_heads, n_kv, hd))
        KLLM_FAIL("attention (float32, mma): %d heads of %d on %d kv heads, or an address, not taken", n_heads, hd, n_kv);
    if (qt < 1 || qt * (n_heads / n_kv) > ROWS || page_size <= 0 || segment < 0 || keep < 0 || (keep > 0 && (window <= 0 || segment > 0)))
        KLLM_FAIL("attention (float32, mma): %d tokens a tile, page size %d, segment %d, %d kept keys beside a window of %d", qt, page_size,
                  segment, keep, window);
    Args a;
    a.out = (float*)out; a.q = (const float*)q; a.q_stride = q_stride; a.kcache = (const float*)kcache; a.vcache = (const float*)vcache;
    a.q_start = q_start; a.start_pos = start_pos; a.block_table = block_table; a.max_blocks = max_blocks; a.n_requests = n_requests;
    a.n_heads = n_heads; a.n_kv = n_kv; a.page_size = page_size; a.window = window; a.qt = qt; a.segment = segment; a.keep = keep;
    a.scale = scale; a.slopes = slopes; a.sinks = sinks;
    return hd == 64 ? launch<64>(a, max_tiles, (cudaStream_t)stream) : launch<128>(a, max_tiles, (cudaStream_t)stream);
}
