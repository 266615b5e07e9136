"""How the attention kernels are cut and chosen, and the barrier on which the tensor-memory attention kernel announces its products into the output, by its own account of
which products complete a phase and which phases are waited for (csrc/attention_tcgen05_ptmem.cu).  A wait by parity
passes at once while the phase before it is open, so it is sound only for the phase behind the one waited for
last; no order between arrivals on different barriers is taken for granted here."""
import ctypes

import pytest


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 33])
def test_every_phase_is_awaited_in_turn(hd, ntiles):
    from kllm_b200.csrc.build import load_library
    lib = load_library("attention_tcgen05_ptmem", {"KLLM_HD": hd})
    announced, awaited = (ctypes.c_int * ntiles)(), (ctypes.c_int * (ntiles + 1))()
    n = lib.kllm_attention_tcgen05_ptmem_output_phases( ntiles, ctypes.addressof(announced), ctypes.addressof(awaited))
    phases = [j for j in range(ntiles) if announced[j]]         # phase p is the product of tile phases[p]
    assert list(awaited[:n]) == list(range(len(phases)))
    assert phases[awaited[n - 1]] == ntiles - 1                 # the last wait is for the last product



def test_which_form_a_step_takes(monkeypatch):
    """Long chains and a second wave do not go to the form of one CTA an SM at head size 128, and one wave goes to the form
    with two score buffers at 64, also where the chains are short."""
    from kllm_b200 import kernels
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    form = kernels.tcgen05_choice
    assert form(128, 4, 8, 600, 1, 2600) == "tmem" and form(128, 4, 8, 600, 1, 600) == "smem"
    assert form(128, 4, 8, 300, 1, 8300) == "smem" and form(128, 4, 8, 850, 1, 850) == "tmem"
    assert form(64, 8, 4, 700, 1, 700) == "smem" and form(64, 8, 4, 2048, 1, 2048) == "smem"
    assert form(64, 8, 4, 2400, 24, 100) == "tmem" and form(64, 8, 4, 8192, 1, 8192) == "tmem"


# tokens, kv heads, context, head size: ranges.  Times of the ranges beside it, in kernels.decode_splits.
SPLITS = [
    (1, 4, 256, 64, 1), (1, 4, 512, 64, 8), (8, 4, 300, 64, 5), (16, 4, 300, 64, 1), (16, 4, 400, 64, 4), (24, 4, 512, 64, 1),
    (1, 8, 200, 128, 1), (1, 8, 300, 128, 5), (8, 8, 300, 128, 1), (8, 8, 512, 128, 4), (16, 8, 512, 128, 1),
    (1, 8, 100, 256, 1), (1, 8, 256, 256, 1), (1, 8, 300, 256, 5), (8, 8, 512, 256, 1),
    (64, 8, 1280, 128, 1), (24, 32, 1500, 128, 1), (64, 4, 2000, 64, 2), (16, 32, 2000, 64, 1), (24, 32, 2000, 64, 2),
    (24, 8, 2000, 256, 2), (32, 8, 2000, 256, 1), (8, 4, 2048, 64, 8), (1, 8, 8000, 128, 16),
]


@pytest.mark.parametrize("n,kv,ctx,hd,ranges", SPLITS)
def test_ranges_of_a_context(monkeypatch, n, kv, ctx, hd, ranges):
    """Few pairs cut contexts that outlast the merge, many do not; long contexts are cut where that fills the last wave."""
    from kllm_b200 import kernels
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    assert kernels.decode_splits(n, kv, ctx, hd) == ranges
