// The launches of all layers of a prompt's step, made from one call: n > 16 tokens through L layers of
//   x += Wo attn(rope(Wqkv norm(x)));  x += Wdown(silu(Wgate norm(x)) * (Wup norm(x)))
// in bfloat16 with a float32 residual stream (the layer of the reference, backend/model.cu:1067-1124).
//
// No kernel of its own: the launchers of the other libraries and the library product are called in the order in
// which the parts call them one by one (parts/block.py), with the same arguments, so the results are the same bits.
// What it saves is the host's time between two launches.  Made from Python the 246 launches of a step of 22 layers
// took 5.7 ms, and a step of a few hundred tokens is 1 to 3 ms of GPU work.
#include "common.cuh"

#include <cublas_v2.h>
#include <dlfcn.h>

KLLM_EXPORT_LAST_ERROR(prompt_layers)

namespace {

// the other libraries' entry points, in the order in which the caller hands them over
struct Entries {
    int (*norm)(void*, const void*, void*, const void*, const int*, int, int, float, int, int, void*);
    int (*rope)(void*, int64_t, const void*, int64_t, const void*, int64_t, const float*, const int*, const int*, const int*, int,
                void*, void*, int, int, int, int, int, int, int, void*);
    int (*decode)(void*, void*, void*, const void*, int64_t, const void*, const void*, const int*, const int*, const int*, int, int,
                  int, int, int, int, int, float, int, const float*, int, const float*, int, void*);
    int (*prefill)(void*, const void*, int64_t, const void*, const void*, const int*, const int*, const int*, int, int, int, int,
                   int, int, int, int, float, int*, void*);
    int (*silu)(void*, int64_t, const void*, int64_t, const void*, int64_t, int, int, int, int, void*);
};

typedef cublasStatus_t (*GemmEx)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void*, const void*,
                                 cudaDataType, int, const void*, cudaDataType, int, const void*, void*, cudaDataType, int,
                                 cublasComputeType_t, cublasGemmAlgo_t);

// the product of the library that this process has loaded already (with torch); null: none
GemmEx library_product() {
    static GemmEx fn = [] {
        void* lib = dlopen("libcublas.so.12", RTLD_NOW | RTLD_NOLOAD);
        return lib ? (GemmEx)dlsym(lib, "cublasGemmEx") : nullptr;
    }();
    return fn;
}

// y [n, N] (+)= x [n, K] . w [N, K]^T; out: CUDA_R_16BF (stored) or CUDA_R_32F
bool product(cublasHandle_t blas, const void* w, int N, int K, const void* x, int n, void* y, cudaDataType out, bool add) {
    const float one = 1.f, beta = add ? 1.f : 0.f;
    return library_product()(blas, CUBLAS_OP_T, CUBLAS_OP_N, N, n, K, &one, w, CUDA_R_16BF, K, x, CUDA_R_16BF, K, &beta, y, out, N,
                             CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT) == CUBLAS_STATUS_SUCCESS;
}

}  // namespace

// 1 if the library product can be called from here.
extern "C" int kllm_prompt_layers_ready() { return library_product() != nullptr ? 1 : 0; }

// layers: host array of n_layers x 9 addresses (w_qkv [(H + 2G) hd, d], w_o [d, H hd], w_gate_up [2F, d], w_down [d, F],
// gain1, gain2 float32 [d], key pages, value pages, cos / sin table float32 [positions, hd]).  entries: the addresses of `Entries`.  blas: a handle of the library
// product that is set to the stream.  A layer has two halves, the first up to the norm in front of the feed-forward (left
// in xn), the second the down product (from act): the halves first .. last - 1 of the layers' 2 n_layers are run.  x [n, d] float32; positions, token_req [n]; table [requests, max_blocks]; the first
// `singles` requests bring one token each and run as decoding tokens in num_splits ranges (part_o, part_ml: their
// scratch), the requests behind them as portions.  xn [n, d], qkv [n, (H + 2G) hd], attn [n, H hd], act [n, F] bfloat16;
// gate_up: float32 [n, 2F], for the gate and up products and the activation behind every first half; null: the caller
// makes act from xn between two calls.  failed: the number of the entry that refused (5: the library product), whose
// library holds the message.
extern "C" int kllm_prompt_layers(int first, int last, const void* layers, int n_layers, const void* entries, void* blas, int n, int d, int H, int G,
                                  int hd, int F, float eps, float scale, float* x, const int* positions,
                                  const int* token_req, const int* table, int max_blocks, int n_requests, const int* q_start,
                                  const int* start_pos, int singles, int num_splits, int page_size, void* xn, void* qkv,
                                  void* attn, void* part_o, void* part_ml, void* act, void* gate_up, int* status, int* failed,
                                  void* stream) {
    if (first < 0 || first >= last || last > 2 * n_layers || n < 1 || d < 1 || H < 1 || G < 1 || hd < 1 || F < 1 || !layers || !entries || !blas || !x || !xn || !qkv ||
        !attn || !act || !failed || singles < 0 || singles >= n_requests)
        KLLM_FAIL("prompt_layers: an argument is missing or out of range");
    if (!library_product()) KLLM_FAIL("prompt_layers: the product library is not loaded in this process");
    const Entries& e = *(const Entries*)entries;
    cublasHandle_t b = (cublasHandle_t)blas;
    const int qd = H * hd, kd = G * hd, w = qd + 2 * kd;
    bf16* q = (bf16*)qkv;
    auto refuse = [&](int which, int rc) { *failed = which; return rc; };
    int rc;
    for (int half = first; half < last; half++) {
        void* const* p = (void* const*)layers + 9 * (half / 2);
        if (half & 1) {
            if (!product(b, p[3], d, F, act, n, x, CUDA_R_32F, true)) return refuse(5, -1);
            continue;
        }
        if ((rc = e.norm(x, nullptr, xn, p[4], nullptr, n, d, eps, KLLM_BF16, KLLM_BF16, stream))) return refuse(0, rc);
        if (!product(b, p[0], w, d, xn, n, q, CUDA_R_16BF, false)) return refuse(5, -1);
        if ((rc = e.rope(q, w, q + qd, w, q + qd + kd, w, (const float*)p[8], positions, token_req, table, max_blocks, p[6], p[7], n, H, G, hd, hd,
                         page_size, KLLM_BF16, stream)))
            return refuse(1, rc);
        if (singles > 0 && (rc = e.decode(attn, part_o, part_ml, q, w, p[6], p[7], positions, nullptr, table, max_blocks, singles, H, G,
                                          hd, page_size, 0, scale, num_splits, nullptr, 0, nullptr, 0, stream)))
            return refuse(2, rc);
        if ((rc = e.prefill(attn, q, w, p[6], p[7], q_start + singles, start_pos + singles, table + (int64_t)singles * max_blocks,
                            max_blocks, n, n_requests - singles, H, G, hd, page_size, 0, scale, status, stream)))
            return refuse(3, rc);
        if (!product(b, p[1], d, qd, attn, n, x, CUDA_R_32F, true)) return refuse(5, -1);
        if ((rc = e.norm(x, nullptr, xn, p[5], nullptr, n, d, eps, KLLM_BF16, KLLM_BF16, stream))) return refuse(0, rc);
        if (!gate_up) continue;
        if (!product(b, p[2], 2 * F, d, xn, n, gate_up, CUDA_R_32F, false)) return refuse(5, -1);
        if ((rc = e.silu(act, F, gate_up, 2 * (int64_t)F, (float*)gate_up + F, 2 * (int64_t)F, n, F, KLLM_BF16, KLLM_F32, stream)))
            return refuse(4, rc);
    }
    return 0;
}
