"""The float32 product on the tensor cores (csrc/gemm_f32_tcgen05.cu) against float64, at the edges of its tiles (128
rows, 256 columns, k blocks of 32), with and without splits of K, in one piece of W and in several."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SIZES = [  # rows, columns, k
    (1, 4, 4), (33, 256, 32), (127, 252, 36), (128, 260, 60), (129, 512, 100), (300, 1028, 2052), (33, 2560, 2048),
    (257, 4100, 160),
    (131, 11264, 1100),
]

# rows, columns, k, epilogue: columns of a piece of W whose parts stay in L2, and ranges of k.  A shorter last piece, pieces
# with ranges of k, and the columns' offset in the result of each epilogue.
CUTS = [
    (131, 11264, 1100, "swiglu", 5632, 1), (1003, 5632, 2048, "swiglu", 2304, 1), (64, 5632, 2048, "swiglu", 3072, 6),
    (128, 32000, 2048, "f32", 5632, 6), (128, 32000, 2048, "add", 5632, 6), (700, 12004, 2048, "f32", 6144, 1),
    (700, 12004, 2048, "add", 6144, 1),
]


def _bound(K):
    # An element's error over sqrt(mean square of the results): the dropped terms are below 2^-24 of every product, an
    # accumulator of 12 products cuts less than 12 x 2^-23 of what it holds, and K / 32 rounded adds follow: a random walk
    # of sqrt(K / 32) x 2^-24 times the sums' size.  Five standard deviations and more for the largest of the results.
    return 5 * 2.0 ** -23 * (12.0 ** 0.5 + (K / 32.0) ** 0.5)


def _product(rows, cols, k, epilogue):
    from kllm_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + cols + k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    wide = rnd(rows, k + 8)
    x, w = wide[:, 4:4 + k], rnd(cols, k) * 0.05                 # a view: rows at a stride, 16 bytes off
    want = x.double() @ w.double().T
    scale = want.square().mean().sqrt()
    if epilogue == "swiglu":
        up = rnd(cols, k) * 0.05
        y = kernels.gemm_f32(x, w, weight_up=up, epilogue="swiglu")
        u = x.double() @ up.double().T
        # an error e in gate or up moves the result by at most 1.1 |u| e and |silu(g)| e; expf adds a few ulp of it
        slack = _bound(k) * scale * (1.1 * u.abs() + want.abs() + 1e-30) + 8 * 2.0 ** -24 * (want * u).abs()
        want = torch.nn.functional.silu(want) * u
    elif epilogue == "add":
        y = rnd(rows, cols)
        want = want + y.double()
        kernels.gemm_f32(x, w, epilogue="add", out=y)
        slack = _bound(k) * scale + 2.0 ** -23 * want.abs()
    else:
        y = kernels.gemm_f32(x, w)
        slack = torch.full_like(want, float(_bound(k) * scale))
    bad = (y.double() - want).abs() - slack
    assert bad.max() <= 0, f"{int((bad > 0).sum())} of {bad.numel()} beyond the bound, worst by {float(bad.max())}"
    assert int(kernels.status_word(y.device).item()) == 0


@pytest.mark.parametrize("epilogue", ["f32", "add", "swiglu"])
@pytest.mark.parametrize("rows,cols,k", SIZES)
def test_float32_product(rows, cols, k, epilogue):
    _product(rows, cols, k, epilogue)


@pytest.mark.parametrize("rows,cols,k,epilogue,piece,splits", CUTS)
def test_float32_product_in_pieces(rows, cols, k, epilogue, piece, splits):
    from kllm_b200.csrc.build import load_library
    cut = (ctypes.c_int * 2)()
    load_library("gemm_f32_tcgen05").kllm_gemm_f32_tcgen05_plan(rows, cols, k, ("f32", "add", "swiglu").index(epilogue),
                                                                ctypes.addressof(cut), ctypes.addressof(cut) + 4)
    assert tuple(cut) == (piece, splits)
    _product(rows, cols, k, epilogue)


def test_sums_of_one_sign_do_not_drift():
    """Every product positive and a long k: what the tensor core's accumulation cuts off stays within one block of k."""
    from kllm_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(11)
    x, w = (torch.rand(n, 16384, generator=g, device="cuda") for n in (64, 256))
    want = x.double() @ w.double().T
    # every block of 32 is short by less than 12 x 2^-23 of itself; the 512 rounded adds are a walk of 0.29 x 2^-23 a step
    # at the sum's full size, sqrt(512 / 3) steps' worth over a growing sum: five deviations are 19 x 2^-23
    assert ((kernels.gemm_f32(x, w).double() - want).abs() / want).max() <= (12 + 19) * 2.0 ** -23


def test_large_and_non_finite_numbers():
    """Finite numbers up to the largest float32 are exact; an infinity or NaN leaves the other rows alone, and the infinity
    stays one where it meets a number that is not zero."""
    from kllm_b200 import kernels
    x = torch.zeros(40, 64, device="cuda")
    x[0], x[1], x[2, 5], x[3, 6] = 3.4028234e38, -3.4e38, float("inf"), float("nan")
    x[4], x[5] = 1.1754944e-38, 1.0 + 2.0 ** -23
    y = kernels.gemm_f32(x, torch.eye(64, device="cuda"))
    assert y[2, 5] == float("inf") and torch.isnan(y[2, :5]).all() and torch.isnan(y[2, 6:]).all() and torch.isnan(y[3]).all()
    keep = [0, 1, 4, 5] + list(range(6, 40))
    assert torch.equal(y[keep], x[keep])


@pytest.mark.parametrize("rows,cols,k", [(40, 260, 64), (64, 2560, 2048)])
@pytest.mark.parametrize("scale", [2.0 ** -125, 2.0 ** -113, 2.0 ** -107, 2.0 ** 70, 2.0 ** 98])
def test_full_mantissas_of_any_size(rows, cols, k, scale):
    """Operands of every size with full mantissas, their partners such that the results are of ordinary size."""
    from kllm_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(int(k + cols))
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").clamp(-8, 8)
    x, w = rnd(rows, k) * scale, rnd(cols, k)
    partner = min(1.0 / scale, 2.0 ** 100)                    # below 2^104, where numbers are split
    for a, b in ((x, w), (x, w * partner), (rnd(rows, k) * partner, rnd(cols, k) * scale)):
        want = a.double() @ b.double().T
        rms = want.square().mean().sqrt()
        # results that are subnormal are rounded to multiples of 2^-149 (the sums of several ranges of k one by one)
        assert ((kernels.gemm_f32(a, b).double() - want).abs().max() - 16 * 2.0 ** -149) <= _bound(k) * rms


@pytest.mark.parametrize("epilogue", ["f32", "add", "swiglu"])
@pytest.mark.parametrize("rows,cols,k", [(40, 260, 64), (64, 2560, 2048), (300, 1028, 52)])
def test_infinities(rows, cols, k, epilogue):
    """Operands with infinities and products that overflow against float64 rounded to float32, and every other row and
    column the same bits as without them.  64 x 2560 x 2048 sums in several ranges of k, the others in one."""
    from kllm_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, up, h = rnd(rows, k), rnd(cols, k), rnd(cols, k), rnd(rows, cols)
    call = lambda x, w, up: (kernels.gemm_f32(x, w, weight_up=up, epilogue="swiglu") if epilogue == "swiglu" else
                             kernels.gemm_f32(x, w, epilogue="add", out=h.clone()) if epilogue == "add" else kernels.gemm_f32(x, w))
    plain = call(x, w, up)
    inf = float("inf")
    xi, wi, ui = x.clone(), w.clone(), up.clone()
    xi[3, 7], xi[5, 0], xi[5, k - 1], xi[rows - 1, 30] = inf, -inf, inf, -inf
    xi[9] = 0.0
    xi[9, 11] = 1.2345678e30
    wi[4, 9], wi[cols - 1, 2], ui[6, 3] = inf, -inf, inf
    wi[17, 11], ui[17, 11] = -1.2345678e30, 1.7654321e30
    got = call(xi, wi, ui)
    wide = xi.double() @ wi.double().T
    if epilogue == "swiglu":
        # the activation in float32, as the kernels take it: exp(-g) overflows from g = -88.7 on, and 0 times an infinite
        # up is NaN where float64 still has a tiny number
        gate = wide.float()
        wide = (gate / (1 + torch.exp(-gate))) * (xi.double() @ ui.double().T).float()
    elif epilogue == "add":
        wide = wide + h.double()
    want = wide.float()
    hit_r, hit_c = [3, 5, 9, rows - 1], [4, 6, 17, cols - 1]
    touched = torch.zeros(rows, cols, dtype=torch.bool, device="cuda")
    touched[hit_r] = True
    touched[:, hit_c] = True
    assert torch.equal(got[~touched], plain[~touched])
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(want)), kind.__name__


@pytest.mark.parametrize("stay,part,cols,k,epilogue,splits", [(500, 400, 2560, 2048, "f32", 3), (700, 600, 2048, 2048, "add", 3),
                                                              (250, 190, 2816, 1024, "swiglu", 3), (870, 800, 516, 1500, "swiglu", 4)])
def test_splits_are_added_in_one_order_whoever_adds_them(stay, part, cols, k, epilogue, splits):
    """With ``stay`` rows a pair sums all of K, the splits before put aside in tensor memory; with ``part`` rows every split is
    a unit of work and a kernel behind adds them: rows that both have come out the same to the bit, and as near to 64 bits as
    sums of K / splits are."""
    from kllm_b200 import kernels
    from kllm_b200.csrc.build import load_library
    lib, epi, up = load_library("gemm_f32_tcgen05"), ("f32", "add", "swiglu").index(epilogue), lambda b: -(-b // 256) * 256
    kp, w_rows = -(-k // 8) * 8, -(-cols // 16) * 32 if epilogue == "swiglu" else cols
    for rows, sums in ((stay, 0), (part, up(4 * splits * part * w_rows))):
        cut, size = (ctypes.c_int * 2)(), ctypes.c_int64(0)
        lib.kllm_gemm_f32_tcgen05_plan(rows, cols, k, epi, ctypes.addressof(cut), ctypes.addressof(cut) + 4)
        lib.kllm_gemm_f32_tcgen05_workspace(rows, cols, k, epi, ctypes.byref(size))
        assert tuple(cut) == (cols, splits) and size.value == up(6 * rows * kp) + up(6 * w_rows * kp) + sums
    g = torch.Generator(device="cuda").manual_seed(stay + k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, w2, y = rnd(stay, k), rnd(cols, k) * 0.05, rnd(cols, k) * 0.05, rnd(stay, cols)
    got = []
    for rows in (stay, part):
        out = y[:rows].clone()
        kernels.gemm_f32(x[:rows], w, weight_up=w2 if epilogue == "swiglu" else None, epilogue=epilogue, out=out)
        got.append(out)
    assert torch.equal(got[0][:part], got[1])
    _product(stay, cols, k, epilogue)


def test_route():
    """Which float32 products run here, and that the general product takes the route and agrees with float64."""
    from kllm_b200 import kernels
    w = torch.randn(2048, 1024, device="cuda")
    for rows, taken in ((32, False), (33, True), (200, True)):
        x = torch.randn(rows, 1024, device="cuda")
        assert kernels.gemm_f32_fits(x, w) is taken
        y = kernels.linear(x, w)
        want = x.double() @ w.double().T
        assert (y.double() - want).norm() <= 2e-6 * want.norm()
    x = torch.randn(64, 1024, device="cuda")
    assert not kernels.gemm_f32_fits(x[:, 1:1001], w[:, 1:1001])        # not 16-byte aligned
    assert not kernels.gemm_f32_fits(x.t().contiguous().t(), w)         # k not contiguous
    assert not kernels.gemm_f32_fits(x[:, :1022], w[:, :1022])
    assert not kernels.gemm_f32_fits(x, w[:512])                        # too small to pay
    assert not kernels.gemm_f32_fits(torch.empty(0, 1024, device="cuda"), w)


def test_what_the_library_does_stays_with_it():
    """An ``out`` of another shape is resized, as below the route's sizes; a product whose gradient is wanted has one."""
    from kllm_b200 import kernels
    x, w = torch.randn(64, 1024, device="cuda"), torch.randn(2048, 1024, device="cuda")
    want = x.double() @ w.double().T
    for shape in ((0,), (3, 3)):
        out = torch.empty(shape, device="cuda")
        y = kernels.linear(x, w, out=out)
        assert y is out and y.shape == (64, 2048) and (y.double() - want).norm() <= 2e-6 * want.norm()
    v = w.clone().requires_grad_()
    y = kernels.linear(x, v)
    assert y.requires_grad
    y.sum().backward()
    assert (v.grad - x.sum(dim=0)).abs().max() <= 1e-4 * x.sum(dim=0).abs().max()
    with torch.no_grad():
        assert kernels.gemm_f32_fits(x, v) and not kernels.linear(x, v).requires_grad
