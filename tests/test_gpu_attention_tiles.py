"""The tcgen05 attention that keeps its probabilities in tensor memory at the edges of its tiles (64 keys; cases at the
edges of 128 too), with windows, pages that split a tile, and many tiles of one chain."""
import pytest

from test_gpu_kernels import attention_case, close

pytestmark = pytest.mark.gpu

# cached and new tokens of the requests
EDGES = [([0], [1]), ([0, 63, 64], [64, 1, 1]), ([127, 0, 128], [1, 128, 2]), ([129, 0], [3, 129]), ([191, 65], [2, 200])]


@pytest.mark.parametrize("hd,H,G", [(64, 8, 2), (128, 4, 4), (128, 8, 1)])
@pytest.mark.parametrize("window", [None, 70, 129])
@pytest.mark.parametrize("start,new", EDGES)
def test_tile_edges(hd, H, G, window, start, new):
    lengths = [a + b for a, b in zip(start, new)]
    for page in (16, 64):
        got, want = attention_case("bfloat16", H, G, hd, page, lengths, new, window, seed=hd + len(new), kernel="tcgen05_tmem")
        close(got, want, "bfloat16")


@pytest.mark.parametrize("hd,H,G,tokens", [(64, 32, 4, 700), (64, 32, 32, 2600), (128, 32, 8, 900)])
def test_long_chains_agree_with_the_other_form(hd, H, G, tokens):
    """Launches of one and of several waves against the form that passes the probabilities through shared memory.  At head
    size 64 both sum in the same order; at 128 the bound leaves two bfloat16 roundings of an output and a little more."""
    import torch
    from kllm_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.bfloat16)
    pages = -(-tokens // 64)
    q, k, v = rnd(tokens, H * hd) * 2, rnd(pages, G, 64, hd), rnd(pages, G, 64, hd)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).int().cuda().view(1, pages)
    start = torch.tensor([0, tokens], dtype=torch.int32, device="cuda")
    outs = []
    for form in ("smem", "tmem", "tmem"):
        out = torch.empty_like(q)
        kernels.attention_prefill_tcgen05(out, q, k, v, start, start[:1], table, 1, H, G, hd, 0, hd ** -0.5, probabilities=form)
        outs.append(out.float())
    assert int(kernels.status_word(q.device).item()) == 0
    assert torch.equal(outs[1], outs[2])
    if hd == 64:
        assert torch.equal(outs[0], outs[1])
    else:
        assert (outs[0] - outs[1]).norm() <= 2.0 ** -7 * outs[0].norm()


def test_form_of_steps_of_one_cta_an_sm():
    from kllm_b200 import kernels
    assert kernels.tcgen05_form(128, 4, 8, 700, 1, 700) == "smem"
    assert kernels.tcgen05_form(128, 4, 8, 1050, 2, 1600) == "tmem"
