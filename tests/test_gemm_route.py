"""Which gated products run on the tcgen05 kernel and which through the library, on the host."""
import pytest

from kllm_b200 import kernels

# K, N, rows, us of the kernel, us of the library's two launches (B200, weights from memory)
MEASURED = [
    (2048, 5632, 24, 13.0, 12.5), (2048, 5632, 128, 14.0, 12.7), (2048, 5632, 400, 20.5, 23.5), (2048, 5632, 845, 32.5, 40.3),
    (2048, 2048, 128, 10.4, 8.2), (2048, 8192, 96, 15.7, 18.1), (4096, 14336, 96, 44.5, 52.3), (4096, 14336, 128, 46.0, 53.7),
    (4096, 11008, 450, 70.3, 80.3), (4096, 4096, 64, 17.3, 15.9), (1024, 2816, 128, 7.9, 7.3), (1024, 2816, 2048, 20.1, 31.8),
    (768, 3072, 4096, 32.2, 63.9), (512, 2048, 4096, 20.3, 37.4), (8192, 28672, 300, 261.5, 362.8), (14336, 4096, 224, 59.5, 52.5),
    (5120, 13824, 128, 54.8, 62.4),
]


@pytest.mark.parametrize("K,N,n,here,library", MEASURED)
def test_the_faster_route_is_taken(monkeypatch, K, N, n, here, library):
    """Sizes at which the routes differ by 4 % and more; the same rows and columns go either way by K alone."""
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    monkeypatch.setattr(kernels, "USE_TCGEN05", True)
    for epilogue in ("swiglu", "clamped"):
        assert kernels.gemm_pays(n, N, epilogue, K=K) == (here < library)


def test_nothing_to_do_and_no_tensor_cores(monkeypatch):
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    monkeypatch.setattr(kernels, "USE_TCGEN05", True)
    assert not kernels.gemm_pays(0, 4096, "swiglu") and not kernels.gemm_pays(64, 0, "swiglu")
    assert kernels.gemm_pays(2048, 5632, "swiglu", K=2048)
    monkeypatch.setattr(kernels, "USE_TCGEN05", False)
    assert not kernels.gemm_pays(2048, 5632, "swiglu", K=2048)


@pytest.mark.gpu
def test_the_rule_counts_the_tiles_that_the_kernel_runs():
    import ctypes
    from kllm_b200.csrc.build import load_library
    out = (ctypes.c_int * 2)()
    for n in (1, 16, 17, 64, 200, 256, 257, 845, 2048, 8192):
        for N in (8, 128, 1000, 2816, 5632, 14336, 28672):
            load_library("gemm_tcgen05").kllm_gemm_tcgen05_pair_plan(n, N, ctypes.addressof(out), ctypes.addressof(out) + 4)
            assert tuple(out) == kernels.pair_plan(n, N, kernels.sm_count() // 2), (n, N)
