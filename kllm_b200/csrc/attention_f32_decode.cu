// Attention of single float32 tokens (decode) over the paged cache, with the rotary encoding, the cache write and the merge of the
// key ranges inside: one kernel where the general route (csrc/rope.cu, csrc/attention_simt.cu) takes three.
//
// A decoding token has few rows (the GS heads of a kv head) and long contexts: the kernel is its cache reads.  A CTA of four warps
// has one (token, kv head) and a range of `chunk` keys; a warp takes batches of keys (four a lane group), every lane 16 bytes of a
// key and of a value, straight into registers, the next batch's on their way while this one's are used and the first one's before
// griddepcontrol.wait (the cached keys do not depend on the kernel before; the token's own key and value, which do, are taken from
// its projections).  HD / 4 lanes share a key: a lane multiplies its four dims of the key with those of all GS queries, the GS sums
// meet in halving exchanges that leave one head's score in each lane, and the weights go back to all lanes by shuffles.  Every
// lane group keeps its own running maximum, sum and output; they are added in group order at the end.  A context of several
// ranges: partial results through L2, added in range order by the CTA that ends last (an atomic counter finds it).
// Formulas as in attention_simt.cu, float32 throughout; the order of every sum depends on the token's position and the window alone.
// Measured: a decode step of 8 tokens at 2048 keys, TinyLlama's 22 layers, 1764 us, with the three kernels 1870; alone, out of L2, 24 us,
// DRAM busy for 17 %: 213 registers at eight heads a kv head leave an SM two CTAs.
#include "common.cuh"

KLLM_EXPORT_LAST_ERROR(attention_f32_decode)

namespace {

constexpr int THREADS = 128, WARPS = 4, UNROLL = 4;

struct Args {
    float* out;                                 // [tokens, n_heads * HD]
    float *part_o, *part_ml;                    // [tokens, n_heads, splits, HD] and [.., 2]: several ranges
    unsigned* counters;                         // [tokens * n_kv], zero, left zero
    const float *q, *k, *v;                     // this step's projections, unrotated
    int64_t q_stride, k_stride, v_stride;
    const float* cos_sin;                       // [positions, HD]: cos, then sin
    float *kcache, *vcache;                     // [pages, n_kv, page_size, HD]
    const int *positions, *block_table;         // token t is request t
    int max_blocks, n_heads, n_kv, page_size, window, chunk, splits;
    float scale;
};

__device__ __forceinline__ float4 shfl4(float4 v, int o) {
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o),
                       __shfl_xor_sync(0xffffffffu, v.z, o), __shfl_xor_sync(0xffffffffu, v.w, o));
}

template <int HD, int GS>
__global__ void __launch_bounds__(THREADS)
attn_f32_decode_kernel(const Args a) {
    constexpr int LPK = HD / 4, KPW = 32 / LPK, GROUPS = WARPS * KPW;       // lanes of a key, keys a load, lane groups of the CTA
    constexpr int BATCH = UNROLL * KPW, OWN = LPK / GS;                     // keys of a batch; lanes that hold one head's score
    static_assert(GS <= LPK && UNROLL == 4, "a lane holds one head's score; four keys a batch");
    __shared__ __align__(16) float so[GROUPS][GS][HD];
    __shared__ float sm[GROUPS][GS], sl[GROUPS][GS];
    __shared__ int s_last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LPK, li = lane % LPK;
    const int t = blockIdx.x / a.n_kv, g = blockIdx.x % a.n_kv, split = blockIdx.y;
    const int pos = a.positions[t];
    const int first = a.window > 0 && pos + 1 > a.window ? pos + 1 - a.window : 0;      // the first visible key
    const int total = pos + 1 - first, lo = split * a.chunk, hi = min(total, lo + a.chunk);
    if (lo >= total) return;
    const int* table = a.block_table + (int64_t)t * a.max_blocks;
    auto place = [&](int kp) {
        const int lp = kp / a.page_size;
        return (((int64_t)table[lp] * a.n_kv + g) * a.page_size + (kp - lp * a.page_size)) * HD + 4 * li;
    };
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [&](float4 (&kb)[UNROLL], float4 (&vb)[UNROLL], int from) {
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const int v = from + u * KPW + sub;
            kb[u] = vb[u] = zero4;
            if (v < hi && first + v != pos) {
                const int64_t at = place(first + v);
                kb[u] = __ldcg(reinterpret_cast<const float4*>(a.kcache + at));
                vb[u] = __ldcg(reinterpret_cast<const float4*>(a.vcache + at));
            }
        }
    };
    float4 k0[UNROLL], v0[UNROLL], k1[UNROLL], v1[UNROLL];
    int at = lo + warp * BATCH;
    load(k0, v0, at);
    const float4 c4 = __ldg(reinterpret_cast<const float4*>(a.cos_sin + (int64_t)pos * HD + 4 * (li % (LPK / 2))));
    float4 s4 = __ldg(reinterpret_cast<const float4*>(a.cos_sin + (int64_t)pos * HD + HD / 2 + 4 * (li % (LPK / 2))));
    if (li < LPK / 2) s4 = make_float4(-s4.x, -s4.y, -s4.z, -s4.w);
    // dims j and j + HD / 2 lie in lanes LPK / 2 apart: a c - b s and b c + a s
    auto rotate = [&](float4 v) {
        const float4 p = shfl4(v, LPK / 2);
        return make_float4(v.x * c4.x + p.x * s4.x, v.y * c4.y + p.y * s4.y, v.z * c4.z + p.z * s4.z, v.w * c4.w + p.w * s4.w);
    };
    griddep_wait();
    griddep_launch();
    float4 q[GS], o[GS];
#pragma unroll
    for (int h = 0; h < GS; h++) {
        q[h] = __ldcg(reinterpret_cast<const float4*>(a.q + (int64_t)t * a.q_stride + (int64_t)(g * GS + h) * HD + 4 * li));
        o[h] = zero4;
    }
    float4 kn = __ldcg(reinterpret_cast<const float4*>(a.k + (int64_t)t * a.k_stride + (int64_t)g * HD + 4 * li));
    const float4 vn = __ldcg(reinterpret_cast<const float4*>(a.v + (int64_t)t * a.v_stride + (int64_t)g * HD + 4 * li));
#pragma unroll
    for (int h = 0; h < GS; h++) q[h] = rotate(q[h]);
    kn = rotate(kn);
    if (hi == total && warp == 0 && sub == 0) {
        const int64_t own = place(pos);
        *reinterpret_cast<float4*>(a.kcache + own) = kn;
        *reinterpret_cast<float4*>(a.vcache + own) = vn;
    }

    float m = -INFINITY, l = 0.f;                          // of head li / OWN, over this lane group's keys
    auto use = [&](float4 (&kb)[UNROLL], float4 (&vb)[UNROLL], int from) {
        float sc[UNROLL], mx = -INFINITY;
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const int v = from + u * KPW + sub;
            if (v < hi && first + v == pos) { kb[u] = kn; vb[u] = vn; }
            float d[GS];
#pragma unroll
            for (int h = 0; h < GS; h++) d[h] = (q[h].x * kb[u].x + q[h].y * kb[u].y) + (q[h].z * kb[u].z + q[h].w * kb[u].w);
#pragma unroll
            for (int off = LPK / 2, n = GS / 2; off >= 1; off >>= 1, n >>= 1) {
                if (n >= 1) {
                    const bool upper = (li & off) != 0;
#pragma unroll
                    for (int j = 0; j < n; j++) {
                        const float send = upper ? d[j] : d[j + n], keep = upper ? d[j + n] : d[j];
                        d[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                    }
                } else {
                    d[0] += __shfl_xor_sync(0xffffffffu, d[0], off);
                }
            }
            sc[u] = v < hi ? d[0] * a.scale : -INFINITY;
            mx = fmaxf(mx, sc[u]);
        }
        // 0 while nothing had been seen.  A maximum of -inf is no base: its keys weigh 0, and a score that is NaN, which fmaxf passes
        // over, stays NaN.
        const float m_new = fmaxf(m, mx), base = m_new == -INFINITY ? 0.f : m_new, alpha = m_new == -INFINITY ? 1.f : expf(m - m_new);
        float p[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) p[u] = expf(sc[u] - base);
        l = l * alpha + ((p[0] + p[1]) + (p[2] + p[3]));
        m = m_new;
#pragma unroll
        for (int h = 0; h < GS; h++) {
            const int from_lane = sub * LPK + h * OWN;
            const float al = __shfl_sync(0xffffffffu, alpha, from_lane);
            float w[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; u++) w[u] = __shfl_sync(0xffffffffu, p[u], from_lane);
            // the batch's values first, then one addition to what was there: as many instructions, a chain of roundings a quarter as long
            auto four = [&](float a0, float a1, float a2, float a3) { return fmaf(w[3], a3, fmaf(w[2], a2, fmaf(w[1], a1, w[0] * a0))); };
            o[h].x = fmaf(o[h].x, al, four(vb[0].x, vb[1].x, vb[2].x, vb[3].x));
            o[h].y = fmaf(o[h].y, al, four(vb[0].y, vb[1].y, vb[2].y, vb[3].y));
            o[h].z = fmaf(o[h].z, al, four(vb[0].z, vb[1].z, vb[2].z, vb[3].z));
            o[h].w = fmaf(o[h].w, al, four(vb[0].w, vb[1].w, vb[2].w, vb[3].w));
        }
    };
    while (at < hi) {                                      // the same for all lanes of a warp
        const int next = at + WARPS * BATCH;
        load(k1, v1, next);
        use(k0, v0, at);
        if (next >= hi) break;
        at = next + WARPS * BATCH;
        load(k0, v0, at);
        use(k1, v1, next);
    }
    // ---- the lane groups' results, added in group order ----
    const int group = warp * KPW + sub;
#pragma unroll
    for (int h = 0; h < GS; h++) *reinterpret_cast<float4*>(&so[group][h][4 * li]) = o[h];
    if (li % OWN == 0) { sm[group][li / OWN] = m; sl[group][li / OWN] = l; }
    __syncthreads();
    const int ns = (total + a.chunk - 1) / a.chunk;
    for (int e = threadIdx.x; e < GS * LPK; e += THREADS) {
        const int h = e / LPK, c = 4 * (e % LPK);
        float M = -INFINITY;
#pragma unroll
        for (int i = 0; i < GROUPS; i++) M = fmaxf(M, sm[i][h]);
        float L = 0.f;
        float4 r = zero4;
#pragma unroll
        for (int i = 0; i < GROUPS; i++) {
            const float w = sl[i][h] == 0.f ? 0.f : expf(sm[i][h] - M);            // 0: a group without a key, or with weights of 0 alone
            const float4 x = *reinterpret_cast<const float4*>(&so[i][h][c]);
            L += sl[i][h] * w;
            r.x += x.x * w; r.y += x.y * w; r.z += x.z * w; r.w += x.w * w;
        }
        const int64_t row = (int64_t)t * a.n_heads + g * GS + h;
        if (ns == 1) {
            const float inv = 1.f / L;
            *reinterpret_cast<float4*>(a.out + row * HD + c) = make_float4(r.x * inv, r.y * inv, r.z * inv, r.w * inv);
        } else {
            __stcg(reinterpret_cast<float4*>(a.part_o + (row * a.splits + split) * HD + c), r);
            if (c == 0) __stcg(reinterpret_cast<float2*>(a.part_ml + (row * a.splits + split) * 2), make_float2(M, L));
        }
    }
    if (ns == 1) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned before = atomicAdd(a.counters + blockIdx.x, 1u);
        s_last = before == (unsigned)ns - 1;
        if (s_last) a.counters[blockIdx.x] = 0;            // ready for the next launch
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    for (int e = threadIdx.x; e < GS * LPK; e += THREADS) {
        const int h = e / LPK, c = 4 * (e % LPK);
        const int64_t row = (int64_t)t * a.n_heads + g * GS + h;
        const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + row * a.splits;
        const float* po = a.part_o + row * a.splits * HD + c;
        float M = -INFINITY, L = 0.f;
        for (int j = 0; j < ns; j++) M = fmaxf(M, __ldcg(ml + j).x);
        float4 r = zero4;
#pragma unroll 4
        for (int j = 0; j < ns; j++) {
            const float2 x = __ldcg(ml + j);
            const float4 y = __ldcg(reinterpret_cast<const float4*>(po + (int64_t)j * HD));
            const float w = expf(x.x - M);
            L += x.y * w;
            r.x += y.x * w; r.y += y.y * w; r.z += y.z * w; r.w += y.w * w;
        }
        const float inv = 1.f / L;
        *reinterpret_cast<float4*>(a.out + row * HD + c) = make_float4(r.x * inv, r.y * inv, r.z * inv, r.w * inv);
    }
}

}  // namespace

// 1 if the kernel takes heads of this size in groups of this width, else 0.
extern "C" int kllm_attention_f32_decode_fits(int n_heads, int n_kv, int hd) {
    const int gs = n_kv > 0 && n_heads % n_kv == 0 ? n_heads / n_kv : 0;
    return (hd == 64 || hd == 128) && (gs == 1 || gs == 2 || gs == 4 || gs == 8 || gs == 16) ? 1 : 0;
}

// One token a request.  q [n, n_heads * hd], k and v [n, n_kv * hd]: this step's projections, unrotated, rows at strides (elements);
// cos_sin [positions, hd]; counters [n * n_kv], zero, left zero.  The keys a token sees (all, or the last `window`) are cut into
// ranges of `chunk`, at most `splits` of them, whose partial results go through part_o [n, n_heads, splits, hd] and part_ml [.., 2].
extern "C" int kllm_attention_f32_decode(void* out, void* part_o, void* part_ml, void* counters, const void* q, int64_t q_stride,
                                         const void* k, int64_t k_stride, const void* v, int64_t v_stride, const float* cos_sin,
                                         void* kcache, void* vcache, const int* positions, const int* block_table, int max_blocks, int n,
                                         int n_heads, int n_kv, int hd, int page_size, int window, float scale, int chunk, int splits,
                                         void* stream) {
    if (n <= 0) return 0;
    if (!kllm_attention_f32_decode_fits(n_heads, n_kv, hd)) KLLM_FAIL("attention decode (float32): %d heads of %d on %d kv heads", n_heads, hd, n_kv);
    if (!q || !k || !v || !cos_sin || page_size <= 0 || window < 0 || chunk <= 0 || splits < 1 || splits > 65535 ||
        (splits > 1 && (!part_o || !part_ml || !counters)))
        KLLM_FAIL("attention decode (float32): operands or ranges missing (page size %d, window %d, %d ranges of %d)", page_size, window, splits, chunk);
    if ((((uintptr_t)out | (uintptr_t)part_o | (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)cos_sin | (uintptr_t)kcache |
          (uintptr_t)vcache) & 15) || ((uintptr_t)part_ml & 7) || ((q_stride | k_stride | v_stride) & 3))
        KLLM_FAIL("attention decode (float32): operands must be 16-byte aligned, strides multiples of 4");
    Args a{(float*)out, (float*)part_o, (float*)part_ml, (unsigned*)counters, (const float*)q, (const float*)k, (const float*)v, q_stride,
           k_stride, v_stride, cos_sin, (float*)kcache, (float*)vcache, positions, block_table, max_blocks, n_heads, n_kv, page_size, window,
           chunk, splits, scale};
    const int gs = n_heads / n_kv;
    const dim3 grid(n * n_kv, splits);
#define KLLM_DEC(HD_, GS_) if (hd == HD_ && gs == GS_) kllm_launch((attn_f32_decode_kernel<HD_, GS_>), grid, dim3(THREADS), 0, (cudaStream_t)stream, a)
    KLLM_DEC(64, 1); KLLM_DEC(64, 2); KLLM_DEC(64, 4); KLLM_DEC(64, 8); KLLM_DEC(64, 16);
    KLLM_DEC(128, 1); KLLM_DEC(128, 2); KLLM_DEC(128, 4); KLLM_DEC(128, 8); KLLM_DEC(128, 16);
#undef KLLM_DEC
    KLLM_LAUNCH_STATUS();
}
