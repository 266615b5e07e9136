"""The barrier on which the tensor-memory attention kernel announces its products into the output, by its own account of
which products complete a phase and which phases are waited for (csrc/attention_tcgen05_ptmem.cu).  A wait by parity
passes at once while the phase before it is open, so it is sound only for the phase behind the one waited for
last; no order between arrivals on different barriers is taken for granted here."""
import ctypes

import pytest


@pytest.mark.parametrize("hd,buffers", [(64, 1), (64, 2), (128, 1)])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 33])
def test_every_phase_is_awaited_in_turn(hd, buffers, ntiles):
    from kllm_b200.csrc.build import load_library
    lib = load_library("attention_tcgen05_ptmem", {"KLLM_HD": hd})
    announced, awaited = (ctypes.c_int * ntiles)(), (ctypes.c_int * (ntiles + 1))()
    n = lib.kllm_attention_tcgen05_ptmem_output_phases(buffers, ntiles, ctypes.addressof(announced), ctypes.addressof(awaited))
    phases = [j for j in range(ntiles) if announced[j]]         # phase p is the product of tile phases[p]
    assert list(awaited[:n]) == list(range(len(phases)))
    assert phases[awaited[n - 1]] == ntiles - 1                 # the last wait is for the last product

