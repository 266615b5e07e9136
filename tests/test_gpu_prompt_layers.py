"""A step with portions launched from native code (csrc/prompt_layers.cu) against the same step launched part by
part: the same kernels and library products with the same arguments in the same order, so the caches and logits agree to
the bit."""
import random

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CONFIGS = {  # hidden, heads, kv heads, head size, feed-forward
    "d64": (256, 8, 2, 64, 704), "d128": (512, 4, 4, 128, 1024), "wide group": (640, 20, 1, 64, 192),
}
# requests' tokens in the step: single tokens first, then portions; the first portion continues a prompt
STEPS = [[17], [1, 16], [1, 1, 1, 40, 9, 1], [200, 3], [1] * 6 + [130]]


def _config(name):
    d, h, g, hd, f = CONFIGS[name]
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": 3, "hidden_size": d, "num_attention_heads": h,
            "num_key_value_heads": g, "head_dim": hd, "intermediate_size": f, "vocab_size": 512, "rope_theta": 10000.0,
            "rms_norm_eps": 1e-5, "max_position_embeddings": 1024}


def _run(name, step, native):
    from kllm_b200 import Engine, Options, StepEntry
    rng = random.Random(len(step))
    engine = Engine(None, Options(max_seq=512, block_size=16, num_blocks=300, max_batch=8, max_step_tokens=512, dtype="bfloat16"),
                    config=_config(name), random_seed=3)
    assert engine.model.prompt_layers is not None
    runs = []
    if native:
        inner = engine.model.prompt_layers
        inner_run = inner.run
        inner.run = lambda *a: (runs.append(1), inner_run(*a))
    else:
        engine.model.prompt_layers = None
    requests = [engine.cache.open() for _ in step]
    for i, r in enumerate(requests):
        engine.step([StepEntry(r, [rng.randrange(512) for _ in range(5 + 37 * i % 90)])])
    del runs[:]
    tokens = [[rng.randrange(512) for _ in range(n)] for n in step]
    logits = engine.step([StepEntry(r, t, [len(t) - 1]) for r, t in zip(requests, tokens)]).clone()
    keys = [k.clone() for k in engine.cache.groups[0].k_store + engine.cache.groups[0].v_store]
    engine.close()
    assert len(runs) == (1 if native else 0)
    return logits, keys


@pytest.mark.parametrize("step", STEPS, ids=lambda s: "+".join(map(str, s)))
@pytest.mark.parametrize("name", list(CONFIGS))
def test_native_launches_agree(name, step):
    a, ka = _run(name, step, False)
    b, kb = _run(name, step, True)
    assert torch.equal(a, b)
    for x, y in zip(ka, kb):
        assert torch.equal(x, y)


@pytest.mark.parametrize("name", ["d64", "d128"])
def test_native_launches_agree_behind_long_contexts(name, monkeypatch):
    """Single tokens whose contexts are cut into ranges (the scratch of partial results and their merge), and a portion
    behind a context of its own."""
    from kllm_b200 import Engine, Options, StepEntry, kernels
    cuts = []
    rule = kernels.decode_splits
    monkeypatch.setattr(kernels, "decode_splits", lambda *a: (cuts.append(rule(*a)), cuts[-1])[1])
    out = []
    for native in (False, True):
        engine = Engine(None, Options(max_seq=1600, block_size=64, num_blocks=120, max_batch=4, max_step_tokens=1500, dtype="bfloat16"),
                        config=dict(_config(name), max_position_embeddings=2048), random_seed=3)
        if not native:
            engine.model.prompt_layers = None
        rng = random.Random(7)
        requests = [engine.cache.open() for _ in range(3)]
        for r, n in zip(requests, (1400, 700, 900)):
            engine.step([StepEntry(r, [rng.randrange(512) for _ in range(n)])])
        del cuts[:]
        logits = engine.step([StepEntry(r, [rng.randrange(512) for _ in range(n)], [n - 1]) for r, n in zip(requests, (1, 1, 40))])
        out.append([logits.clone()] + [t.clone() for t in engine.cache.groups[0].k_store + engine.cache.groups[0].v_store])
        assert cuts and min(cuts) > 1
        engine.close()
    for x, y in zip(*out):
        assert torch.equal(x, y)


def test_steps_that_stay_with_the_parts():
    """Decode steps and steps of few tokens do not go that way, nor a step that is watched layer by layer."""
    from kllm_b200 import Engine, Options, StepEntry
    engine = Engine(None, Options(max_seq=128, block_size=16, num_blocks=80, max_batch=4, dtype="bfloat16", max_step_tokens=128),
                    config=_config("d64"), random_seed=1)
    taken = []
    inner = engine.model.prompt_layers.run
    engine.model.prompt_layers.run = lambda *a: (taken.append(1), inner(*a))
    r = [engine.cache.open() for _ in range(3)]
    engine.step([StepEntry(r[0], [1] * 16, [15])])
    engine.step([StepEntry(x, [2], [0]) for x in r])
    engine.model.tap = lambda i, x: None
    engine.step([StepEntry(r[1], [1] * 30, [29])])
    engine.model.tap = None
    assert not taken
    engine.step([StepEntry(r[2], [1] * 30, [29])])
    assert taken
    engine.close()


def test_wide_step_takes_the_gated_product():
    """Where gate, up and activation are one kernel it runs between the halves of every layer."""
    from kllm_b200 import Engine, Options, StepEntry, kernels
    cfg = dict(_config("d64"), intermediate_size=9472, max_position_embeddings=4096)
    assert kernels.gemm_pays(512, 9472, "swiglu")
    out = []
    for native in (False, True):
        engine = Engine(None, Options(max_seq=600, block_size=16, num_blocks=160, max_batch=3, max_step_tokens=600, dtype="bfloat16"),
                        config=cfg, random_seed=5)
        if not native:
            engine.model.prompt_layers = None
        r = [engine.cache.open() for _ in range(2)]
        engine.step([StepEntry(r[0], [3] * 20)])
        before = kernels.launches
        out.append((engine.step([StepEntry(r[0], [7], [0]), StepEntry(r[1], [i % 512 for i in range(511)], [100, 510])]).clone(),
                    kernels.launches - before))
        engine.close()
    (a, la), (b, lb) = out
    assert torch.equal(a, b)
    assert la == lb                                   # the same kernels


def test_settings_of_the_products_are_obeyed(monkeypatch):
    """The direct calls of the library know nothing of torch's settings: with any that is not the default the parts run."""
    from kllm_b200 import Engine, Options, StepEntry, kernels
    engine = Engine(None, Options(max_seq=128, block_size=16, num_blocks=80, max_batch=8, dtype="bfloat16", max_step_tokens=128),
                    config=_config("d64"), random_seed=1)
    taken = []
    inner = engine.model.prompt_layers.run
    engine.model.prompt_layers.run = lambda *a: (taken.append(1), inner(*a))

    def step():
        del taken[:]
        r = engine.cache.open()
        logits = engine.step([StepEntry(r, list(range(30)), [29])]).clone()
        engine.cache.close(r)
        return logits, bool(taken)
    want, native = step()
    assert native
    m = torch.backends.cuda.matmul
    with monkeypatch.context() as mp:
        mp.setattr(m, "allow_bf16_reduced_precision_reduction", False)
        got, native = step()
        assert not native and (got - want).abs().max() <= 1e-2 * want.abs().max()
    before = torch.backends.cuda.preferred_blas_library()
    try:
        torch.backends.cuda.preferred_blas_library("cublaslt")
        got, native = step()
        assert not native and (got - want).abs().max() <= 1e-2 * want.abs().max()
    finally:
        torch.backends.cuda.preferred_blas_library(before)
    with monkeypatch.context() as mp:
        mp.setattr(m, "allow_tf32", True)
        with pytest.raises(kernels.KernelError, match="TF32"):
            step()
    assert step()[1]
    engine.close()


def test_tables_and_weights_are_those_of_the_call(monkeypatch):
    """What the parts hold when the step runs counts, not what they held when the model was bound: a layer's own table of
    angles is used, and from a weight on that the native launches do not take (rows at a stride) the parts run."""
    from kllm_b200 import Engine, Options, StepEntry, kernels
    engine = Engine(None, Options(max_seq=128, block_size=16, num_blocks=80, max_batch=8, dtype="bfloat16", max_step_tokens=128),
                    config=_config("d64"), random_seed=1)
    layers, model = engine.model.prompt_layers, engine.model
    took = []                                                    # layers launched natively, of three
    inner = kernels.prompt_layers
    monkeypatch.setattr(kernels, "prompt_layers", lambda *a: (took.append(inner(*a)), took[-1])[1])

    def step(native):
        model.prompt_layers = layers if native else None
        r = engine.cache.open()
        logits = engine.step([StepEntry(r, list(range(30)), [29])]).clone()
        engine.cache.close(r)
        return logits
    before = step(True)
    position = model.blocks[1].mixer.position
    position.cos_sin = position.cos_sin.roll(7, dims=0)          # another rotation in one layer
    a, b = step(True), step(False)
    assert torch.equal(a, b) and not torch.equal(a, before) and took == [3, 3]
    for i in (2, 1, 0):
        del took[:]
        mlp = model.blocks[i].feed_forward
        wide = torch.zeros(mlp.w_down.shape[0], mlp.w_down.shape[1] + 8, dtype=mlp.w_down.dtype, device="cuda")
        wide[:, :mlp.w_down.shape[1]] = mlp.w_down
        mlp.w_down = wide[:, :mlp.w_down.shape[1]]
        assert torch.equal(step(True), step(False)) and took == [i]
    engine.close()
