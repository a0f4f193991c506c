"""The two forms of latent attention in one step: absorbed for decoding and short portions, expanded for long ones."""

from __future__ import annotations

import dataclasses

import pytest
import torch

from forge_engine_b200.config.registry import read_model_config
from forge_engine_b200.engine import ModelRunner, StepEntry
from forge_engine_b200.engine.batch import build_batch
from forge_engine_b200.ops import native
from forge_engine_b200.parts import latent_attention as part

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def latent_runner(seed, heads=3, dim=64, rot=32, vdim=64, rank=64, q_rank=64, width=128, pages=128, requests=8, sink=False):
    raw = {"architecture": "Zofadra", "vocab": 32, "width": width, "norm": {"eps": 1e-5}, "layers": [{"type": "latent_attention", "mixer": {
        "heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": q_rank, "kv_rank": rank,
        "rot": {"base": 1e4, "dims": rot}, "scale": (dim + rot) ** -0.5}}]}
    arch, _, spec = read_model_config(raw)
    layer = spec.layers[0]
    spec = dataclasses.replace(spec, layers=(dataclasses.replace(layer, mixer=dataclasses.replace(layer.mixer, sink=sink)),))
    gen = torch.Generator().manual_seed(seed)
    weights = {name: ((1 + 0.1 * torch.randn(info.shape, generator=gen)) if "norm" in name else
                      torch.randn(info.shape, generator=gen) * (info.shape[-1] ** -0.5 if len(info.shape) > 1 else 1.0)).bfloat16().to(DEV)
               for name, info in arch.expected_tensors(spec).items()}
    return ModelRunner.from_tensors(spec, weights, dtype="bfloat16", device=DEV, page_size=16, num_pages=pages, max_requests=requests, architecture=arch)


def cached(runner, starts, counts, seed):
    """Requests with random cached latents and pages for their new tokens; the step's batch."""
    cache = runner.cache
    for i, (start, count) in enumerate(zip(starts, counts)):
        runner.begin(i)
        if start:
            cache.reserve(i, start)
            cache.advance(i, start)
        cache.reserve(i, start + count)
    store = cache.kv_of_run(0)[0]
    store.copy_(torch.randn(store.shape, generator=torch.Generator().manual_seed(seed)))
    return build_batch([StepEntry(i, [0] * c) for i, c in enumerate(counts)], cache, DEV)


@pytest.mark.parametrize("starts, counts", (([90, 0, 60, 700], [1, 1, 300, 260]), ([60, 90, 700, 8, 0], [300, 1, 260, 5, 1]), ([60, 700, 20], [300, 260, 3])))
def test_rows_go_through_one_form(starts, counts, monkeypatch):
    """Decoding and short entries before, between and after long portions: the products of the absorbed form see
    the short entries' rows alone, those of the expanded one the others', and every row is what the absorbed
    form gives for the whole step (each form lies within 1e-2 of 64 bits: test_expanded_latent_attention)."""
    monkeypatch.setattr(part, "EXPAND_BESIDE", 0.0)
    runner = latent_runner(5)
    x = torch.randn((sum(counts), 128), generator=torch.Generator().manual_seed(1)).bfloat16().to(DEV)
    batch = cached(runner, starts, counts, 2)
    mixer = runner.model.blocks[0].mixer
    rows = {"absorbed": [], "expanded": []}

    def note(name, call):
        return lambda x, *args, **kw: (rows[name].append(x.shape[0]), call(x, *args, **kw))[1]

    monkeypatch.setattr(mixer, "_per_head", note("absorbed", mixer._per_head))
    monkeypatch.setattr(mixer, "up_q", note("absorbed", mixer.up_q))
    monkeypatch.setattr(mixer, "expanded", (mixer.expanded[0], note("expanded", mixer.expanded[1])))
    got = mixer.attend(x, batch, runner.cache.view(0)).double()
    short = sum(c for c in counts if c <= mixer.expand_from)
    assert rows == {"absorbed": [short] * 3, "expanded": [sum(counts) - short]}
    monkeypatch.setattr(part, "EXPAND_STEP", 1 << 30)
    batch.plans.clear(), batch.shared.clear()
    want = mixer.attend(x, batch, runner.cache.view(0)).double()
    runner.check_status()
    for a, b in zip(got.split(counts), want.split(counts)):
        assert float((a - b).norm() / b.norm()) < 2e-2


@pytest.mark.parametrize("sink", (False, True))
@pytest.mark.parametrize("heads, at_once", ((3, 2), (5, 1), (8, 3)))
def test_heads_take_turns(heads, at_once, sink, monkeypatch):
    """Keys and values held for some heads at a time give what they give for all at once, up to the order of the
    sums of the product that expands them (its results are bfloat16 numbers: 2^-8 of them)."""
    starts, counts = [90, 700], [300, 260]
    runner = latent_runner(heads, heads=heads, sink=sink)
    x = torch.randn((sum(counts), 128), generator=torch.Generator().manual_seed(1)).bfloat16().to(DEV)
    batch = cached(runner, starts, counts, 2)
    mixer = runner.model.blocks[0].mixer
    whole = mixer.attend(x, batch, runner.cache.view(0)).double()
    rows, calls = 128 * (4 + 8), []
    monkeypatch.setattr(part, "EXPAND_BYTES", at_once * rows * 512)
    monkeypatch.setattr(native, "attention_prefill_expanded", lambda *a, call=native.attention_prefill_expanded: (calls.append(a[8]), call(*a))[1])
    parts = mixer.attend(x, batch, runner.cache.view(0)).double()
    runner.check_status()
    assert sum(calls) == heads and len(calls) > 1 and max(calls) <= at_once
    assert float((parts - whole).norm() / whole.norm()) < 2.0**-8
