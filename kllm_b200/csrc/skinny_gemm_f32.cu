// Y[n, N] = X[n, K] . W[N, K]^T in true float32 for up to 8 rows n (decode steps of the
// 32-bit path): the weights are streamed from HBM exactly once and meet the activations
// in FMA instructions on the CUDA cores; no tensor cores, no reduced-precision mode.
// The reference runs these products through cublasSgemm (backend/model.cu:496-503,
// :1090-1115); at a few rows the library picks matrix-vector kernels by the row count,
// which stream at a fraction of the memory's speed and sum in an order that depends on
// the batch.  Here every output element is summed in an order that depends on K alone.
// Prologues and epilogues as in skinny_gemm.cu:
//
//   prologue  X_PLAIN     X is a float32 matrix [n, K]
//             X_NORM      X = rmsnorm(x) * gain of float32 rows x (optionally gathered by
//                         `rows`), computed by every CTA for itself (backend/model.cu:101-122)
//   epilogue  STORE       Y as float32
//             ADD         Y is added into a float32 matrix (the residual stream)
//             SWIGLU      W holds a gate and an up matrix [F, K] each; the output is
//                         silu(gate row) * (up row) as float32 [n, F]
//                         (backend/model.cu:477-483, :1112-1114)
//
// Layout of the work: a CTA of 16 warps, one per SM, walks tiles of eight weight rows (SWIGLU: four gate rows and their
// four up rows).  A warp owns a contiguous sixteenth of K for every tile of its CTA: it brings that part of X (8 rows) into
// shared memory for itself, and nothing waits for another warp until the CTA's tiles are through.  The norm's scale is a
// factor of a whole row, so it multiplies the finished sums; the sums of squares are taken beside the products.  Within
// a warp eight lanes share a weight row (128 bytes a load) and a lane has two of the tile's rows, so a batch of four steps
// of 32 elements is eight 16-byte loads a lane; two register buffers take turns, 64 KB an SM in flight in each.  The products
// are two-wide (fma.rn.f32x2 on neighbouring k: weights and X both lie in memory as such pairs).  A tile ends in three
// exchanges between the eight lanes (14 shuffles) and a store of the warp's 64 partial sums; the warps' are added in pairs
// (sum_warps), for up to MAX_SLOTS tiles at a time.  Every order is fixed by K alone.
//
// Measured in a decode step of 8 rows of TinyLlama's sizes (B200; us beside what the kernel before hides): gate and up 23.4
// (32.0 in the form that met in shared memory at every tile, with eight parts of K and four rows a warp), down 15.5, O 7.2
// (22.7 together), QKV 12.6 (13.8).
#include "common.cuh"

KLLM_EXPORT_LAST_ERROR(skinny_gemm_f32)

namespace {

constexpr int THREADS = 512, WARPS = 16, ROWS = 8;              // ROWS: rows of X
constexpr int TILE = 8, PARTS = TILE * ROWS;                    // weight rows of a tile; partial sums a warp leaves of one
constexpr int STEP = 32, UNROLL = 4;                            // elements of k a step takes, steps a register buffer holds
constexpr int MAX_SLOTS = 16;                                   // tiles whose partial sums are kept until they are added up
constexpr size_t SMEM_MOST = 227 * 1024;
enum { X_PLAIN = 0, X_NORM = 1 };
enum { STORE = 0, ADD = 1, SWIGLU = 2 };

struct Args {
    const float* w;       // [N, K] at w_stride; SWIGLU: the gate matrix [F, K]
    const float* w_up;    // SWIGLU: the up matrix
    int64_t w_stride;
    int N, K, n;
    const float* x;       // rows of width K at x_stride
    int64_t x_stride;
    const float* gain;    // X_NORM: [K]
    const int* rows;      // X_NORM: optional gather of rows
    float eps;
    float* y;             // [n, N] at y_stride
    int64_t y_stride;
#ifdef KLLM_BIAS
    const float* bias;    // ADD: optional [N], joins the sum; SWIGLU: optional [N], to the gate rows' sums
    const float* bias_up; // SWIGLU: optional [N], to the up rows' sums
    int act;              // SWIGLU: 0 silu, 1 the gelu with tanh, 2 clamped (limit, alpha); STORE: 3 the square of relu
    float limit, alpha;   // act 2: g' = min(g, limit), u' = clamp(u, -limit, limit): g' sigmoid(alpha g') (u' + 1)
#endif
};

// four neighbouring weights as two pairs
__device__ __forceinline__ ulonglong2 ldg_stream(const float* p) {
    ulonglong2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0,%1}, [%2];\n" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(unsigned long long v) {
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// The warps' values, `stride` floats apart, added in pairs: 0 and 1, 2 and 3, ..., then the pairs'.  One after the other they rounded 8 to
// 9 % more over the sums of this file's sizes than the 8 parts of K of an earlier form; in pairs it is less than that.  (Warp w and
// w + 8 first, which keeps eight sums at a time, cost the stream of weights its registers: a decode step of 8 tokens 1827 us, 1768 this way.)
__device__ __forceinline__ float sum_warps(const float* p, int stride) {
    float half[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float* q = p + h * 8 * stride;
        half[h] = ((q[0] + q[stride]) + (q[2 * stride] + q[3 * stride])) + ((q[4 * stride] + q[5 * stride]) + (q[6 * stride] + q[7 * stride]));
    }
    return half[0] + half[1];
}

// EXACT: every warp's part of K is a whole number of batches.
template <int PRO, int EPI, bool EXACT>
__global__ void __launch_bounds__(THREADS, 1)
skinny_f32_kernel(const Args a, const int slots) {
    extern __shared__ __align__(16) float xs[];            // [ROWS][K], then the partial sums [slots][WARPS][TILE][ROWS]
    __shared__ float ss_part[WARPS][ROWS];
    const int K = a.K, N = a.N, n = a.n;
    float* red = xs + (size_t)ROWS * K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane >> 3, kl = lane & 7;
    constexpr int OUT_PER_TILE = EPI == SWIGLU ? TILE / 2 : TILE;    // output columns of a tile
    const int n_tiles = (N + OUT_PER_TILE - 1) / OUT_PER_TILE;
    const int steps = K / STEP, per_warp = (steps + WARPS - 1) / WARPS;
    const int my_steps = max(0, min(per_warp, steps - warp * per_warp));
    const int nb = (per_warp + UNROLL - 1) / UNROLL;                 // batches per tile, the same for all warps
    const int k0 = warp * per_warp * STEP;                           // this warp's part of K: k0 .. k0 + my_steps * STEP

    // two register buffers: [step][0] a row of the tile's first four, [step][1] of its other four (SWIGLU: the up row)
    ulonglong2 buf0[UNROLL][2], buf1[UNROLL][2];
    auto load_batch = [&](ulonglong2 (&buf)[UNROLL][2], int tile, int b) {
        const float *p0, *p1;                                        // rows past the end repeat the last one
        if (EPI == SWIGLU) {
            const int64_t r = min(tile * 4 + sub, N - 1);
            p0 = a.w + r * a.w_stride;
            p1 = a.w_up + r * a.w_stride;
        } else {
            p0 = a.w + (int64_t)min(tile * 8 + sub, N - 1) * a.w_stride;
            p1 = a.w + (int64_t)min(tile * 8 + 4 + sub, N - 1) * a.w_stride;
        }
        const int off = k0 + b * UNROLL * STEP + 4 * kl;
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
            if (EXACT || b * UNROLL + u < my_steps) {
                buf[u][0] = ldg_stream(p0 + off + u * STEP);
                buf[u][1] = ldg_stream(p1 + off + u * STEP);
            }
    };
    int cur_tile = blockIdx.x, cur_b = 0, slot = 0;        // the batch that sits in the buffer used next
    load_batch(buf0, cur_tile, 0);                         // weights do not depend on X: on their way first
    griddep_wait();
    griddep_launch();

    // ---- this warp's part of X into shared memory, rows past n are zero ----
    {
        const int len = my_steps * STEP;
        if (PRO == X_NORM) {
            float ss[ROWS];
#pragma unroll
            for (int c = 0; c < ROWS; c++) ss[c] = 0.f;
            for (int i = 4 * lane; i < len; i += 128) {
                float4 v[ROWS];
#pragma unroll
                for (int c = 0; c < ROWS; c++)
                    v[c] = c < n ? __ldcg(reinterpret_cast<const float4*>(a.x + (int64_t)(a.rows ? a.rows[c] : c) * a.x_stride + k0 + i))
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 g = __ldg(reinterpret_cast<const float4*>(a.gain + k0 + i));
#pragma unroll
                for (int c = 0; c < ROWS; c++) {
                    ss[c] += (v[c].x * v[c].x + v[c].y * v[c].y) + (v[c].z * v[c].z + v[c].w * v[c].w);
                    *reinterpret_cast<float4*>(xs + (size_t)c * K + k0 + i) =
                        make_float4(v[c].x * g.x, v[c].y * g.y, v[c].z * g.z, v[c].w * g.w);
                }
            }
            // eight sums over 32 lanes: halved three times, then two plain exchanges; lanes 4 r .. 4 r + 3 hold row r's
#pragma unroll
            for (int o = 16, h = ROWS / 2; o >= 4; o >>= 1, h >>= 1) {
                const bool upper = (lane & o) != 0;
#pragma unroll
                for (int j = 0; j < h; j++) {
                    const float send = upper ? ss[j] : ss[j + h], keep = upper ? ss[j + h] : ss[j];
                    ss[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 2);
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
            if ((lane & 3) == 0) ss_part[warp][lane >> 2] = ss[0];
        } else {
#pragma unroll
            for (int c = 0; c < ROWS; c++) {
                float* dst = xs + (size_t)c * K + k0;
                if (c < n) {
                    const float* src = a.x + (int64_t)c * a.x_stride + k0;
                    for (int i = 4 * lane; i < len; i += 128) cp_async16(dst + i, src + i);
                } else {
                    for (int i = 4 * lane; i < len; i += 128) *reinterpret_cast<float4*>(dst + i) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        }
        __syncwarp();
    }

    // ---- tiles ----
    unsigned long long acc[2][ROWS];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int c = 0; c < ROWS; c++) acc[r][c] = 0;
    float scale = 1.f;                                     // the norm's, of row threadIdx.x % ROWS
    bool have_scale = PRO != X_NORM;

    // The partial sums of `held` tiles, the last of them last_tile, added up and stored.
    auto finish = [&](int last_tile, int held) {
        __syncthreads();
        const int c = threadIdx.x % ROWS;
        if (!have_scale) {
            scale = rsqrtf(sum_warps(&ss_part[0][c], ROWS) / (float)K + a.eps);
            have_scale = true;
        }
        constexpr int OUTS = EPI == SWIGLU ? PARTS / 2 : PARTS;
        for (int e = threadIdx.x; e < held * OUTS; e += THREADS) {
            const int sl = e / OUTS, rc = e - sl * OUTS, tile = last_tile - (held - 1 - sl) * (int)gridDim.x;
            const float* part = red + (size_t)sl * WARPS * PARTS + rc;
            float v = sum_warps(part, PARTS), up = EPI == SWIGLU ? sum_warps(part + PARTS / 2, PARTS) : 0.f;
            const int col = tile * OUT_PER_TILE + rc / ROWS;
            if (c >= n || col >= N) continue;
            float* dst = a.y + (int64_t)c * a.y_stride + col;
            if (PRO == X_NORM) { v *= scale; up *= scale; }
#ifdef KLLM_BIAS
            if (EPI != STORE && a.bias) v += a.bias[col];
            if (EPI == SWIGLU && a.bias_up) up += a.bias_up[col];
            if (EPI == STORE && a.act == 3) {
                v = fmaxf(v, 0.f);
                v *= v;
            }
            if (EPI == SWIGLU && a.act == 2) {
                v = fminf(v, a.limit);
                up = fminf(fmaxf(up, -a.limit), a.limit);
                *dst = v / (1.f + expf(-a.alpha * v)) * (up + 1.f);
            } else if (EPI == SWIGLU && a.act == 1)
                *dst = 0.5f * v * (1.f + tanhf(0.79788456080286536f * (v + 0.044715f * v * v * v))) * up;
            else
#endif
            if (EPI == SWIGLU) *dst = (v / (1.f + expf(-v))) * up;
            else if (EPI == ADD) *dst += v;
            else *dst = v;
        }
    };

    // multiply the batch (cur_tile, cur_b) held in `cur` while the following batch loads into `nxt`
    auto phase = [&](ulonglong2 (&cur)[UNROLL][2], ulonglong2 (&nxt)[UNROLL][2]) {
        int nxt_tile = cur_tile, nxt_b = cur_b + 1;
        if (nxt_b == nb) { nxt_b = 0; nxt_tile += gridDim.x; }
        if (nxt_tile < n_tiles) load_batch(nxt, nxt_tile, nxt_b);
        const float* xk = xs + k0 + cur_b * UNROLL * STEP + 4 * kl;
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
            if (EXACT || cur_b * UNROLL + u < my_steps) {
#pragma unroll
                for (int c = 0; c < ROWS; c++) {
                    const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(xk + (size_t)c * K + u * STEP);
                    fma2(acc[0][c], cur[u][0].x, xv.x);
                    fma2(acc[1][c], cur[u][1].x, xv.x);
                    fma2(acc[0][c], cur[u][0].y, xv.y);
                    fma2(acc[1][c], cur[u][1].y, xv.y);
                }
            }
        if (cur_b == nb - 1) {
            // 16 sums over the 8 lanes of a row: each exchange halves what a lane holds
            float v[2 * ROWS];
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int c = 0; c < ROWS; c++) { v[r * ROWS + c] = sum2(acc[r][c]); acc[r][c] = 0; }
#pragma unroll
            for (int o = 4, h = ROWS; o >= 1; o >>= 1, h >>= 1) {
                const bool upper = (kl & o) != 0;
#pragma unroll
                for (int j = 0; j < h; j++) {
                    const float send = upper ? v[j] : v[j + h], keep = upper ? v[j + h] : v[j];
                    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            // lane kl: row kl >> 2 of the two, tokens 2 (kl & 3) and the next
            *reinterpret_cast<float2*>(red + ((size_t)slot * WARPS + warp) * PARTS + ((kl >> 2) * 4 + sub) * ROWS + 2 * (kl & 3)) =
                make_float2(v[0], v[1]);
            if (++slot == slots || nxt_tile >= n_tiles) {
                finish(cur_tile, slot);
                slot = 0;
                if (nxt_tile < n_tiles) __syncthreads();
            }
        }
        cur_tile = nxt_tile;
        cur_b = nxt_b;
    };
    while (cur_tile < n_tiles) {
        phase(buf0, buf1);
        if (cur_tile >= n_tiles) break;
        phase(buf1, buf0);
    }
}

template <int PRO, int EPI, bool EXACT>
int launch_exact(const Args& a, cudaStream_t s) {
    static size_t attr_smem = 0;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int out_per_tile = EPI == SWIGLU ? TILE / 2 : TILE;
    const int n_tiles = (a.N + out_per_tile - 1) / out_per_tile;
    const int grid = max(1, min(n_tiles, max(1, sms)));
    // as many tiles between two summings as shared memory holds beside X, spread evenly
    const size_t x_bytes = (size_t)ROWS * a.K * 4, slot_bytes = (size_t)WARPS * PARTS * 4;
    const int most = (int)min((size_t)MAX_SLOTS, (SMEM_MOST - 1024 - x_bytes) / slot_bytes);
    const int per_cta = (n_tiles + grid - 1) / grid, rounds = (per_cta + most - 1) / most;
    const int slots = (per_cta + rounds - 1) / rounds;
    const size_t smem = x_bytes + slots * slot_bytes;
    auto kern = skinny_f32_kernel<PRO, EPI, EXACT>;
    if (smem > attr_smem) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            snprintf(g_kllm_err, sizeof(g_kllm_err), "skinny_gemm_f32: %zu bytes of shared memory refused: %s", smem,
                     cudaGetErrorString(e));
            return (int)e;
        }
        attr_smem = smem;
    }
    kllm_launch_dep(n_tiles <= 3 * grid, (kern), dim3(grid), dim3(THREADS), smem, s, a, slots);
    KLLM_LAUNCH_STATUS();
}

template <int PRO, int EPI>
int launch(const Args& a, cudaStream_t s) {
    return a.K % (WARPS * STEP * UNROLL) == 0 ? launch_exact<PRO, EPI, true>(a, s) : launch_exact<PRO, EPI, false>(a, s);
}

}  // namespace

// 1 if (n, K) can run here: up to 8 rows, K a multiple of 128 whose 8 rows fit shared memory.
extern "C" int kllm_skinny_gemm_f32_fits(int n, int K) {
    return (n >= 1 && n <= ROWS && K >= 128 && K % 128 == 0 && (size_t)ROWS * K * 4 <= 220 * 1024) ? 1 : 0;
}

// prologue 0: x float32 [n, K] at x_stride.  prologue 1: rows of x (row r is rows[r] when rows is
// given) normalised with gain [K] and eps.  epilogue 0: y written; 1: y += result; 2: w = gate
// [N, K], w_up = up [N, K], y = silu(gate) * up.  w_stride: elements from one weight row to the
// next (more than K when the call multiplies a slice of the columns of a wider matrix).
// bias, bias_up, act, limit, alpha: see Args; refused by a library compiled without KLLM_BIAS (as in skinny_gemm.cu).
extern "C" int kllm_skinny_gemm_f32(const float* w, const float* w_up, int64_t w_stride, int N, int K, int n,
                                    const float* x, int64_t x_stride, const float* gain, const int* rows, float eps,
                                    float* y, int64_t y_stride, int prologue, int epilogue, const float* bias,
                                    const float* bias_up, int act, float limit, float alpha, void* stream) {
    if (n <= 0 || N <= 0) return 0;
    if (!kllm_skinny_gemm_f32_fits(n, K))
        KLLM_FAIL("skinny_gemm_f32: %d rows of width %d not supported (1..8 rows, width a multiple of 128 that fits "
                  "shared memory)", n, K);
    if (!w || !x || !y || ((uintptr_t)w & 15) || ((uintptr_t)x & 15) || (w_stride % 4) || (x_stride % 4) || w_stride < K)
        KLLM_FAIL("skinny_gemm_f32: operands must be 16-byte aligned with row strides that are multiples of 4");
    if (prologue == X_NORM && (!gain || ((uintptr_t)gain & 15))) KLLM_FAIL("skinny_gemm_f32: the norm needs a 16-byte aligned gain");
    if (epilogue == SWIGLU && (!w_up || ((uintptr_t)w_up & 15))) KLLM_FAIL("skinny_gemm_f32: SWIGLU needs the up matrix");
    Args a;
    a.w = w; a.w_up = w_up; a.w_stride = w_stride; a.N = N; a.K = K; a.n = n; a.x = x; a.x_stride = x_stride;
    a.gain = gain; a.rows = rows; a.eps = eps; a.y = y; a.y_stride = y_stride;
#ifdef KLLM_BIAS
    if (act < 0 || act > 3 || (act && epilogue != (act == 3 ? STORE : SWIGLU)) || (act == 2 && !(limit > 0.f)))
        KLLM_FAIL("skinny_gemm_f32: activation %d does not go with epilogue %d", act, epilogue);
    a.bias = bias; a.bias_up = bias_up; a.act = act; a.limit = limit; a.alpha = alpha;
#else
    if (bias || bias_up || act) KLLM_FAIL("skinny_gemm_f32: this library was built without biases and activations");
#endif
    cudaStream_t s = (cudaStream_t)stream;
#define KLLM_F32_CASE(P, E) if (prologue == P && epilogue == E) return launch<P, E>(a, s)
    KLLM_F32_CASE(X_PLAIN, STORE); KLLM_F32_CASE(X_PLAIN, ADD); KLLM_F32_CASE(X_PLAIN, SWIGLU);
    KLLM_F32_CASE(X_NORM, STORE); KLLM_F32_CASE(X_NORM, ADD); KLLM_F32_CASE(X_NORM, SWIGLU);
#undef KLLM_F32_CASE
    KLLM_FAIL("skinny_gemm_f32: unknown prologue %d or epilogue %d", prologue, epilogue);
}
