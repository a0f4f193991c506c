"""What latent attention layers decide on the host for a step."""

from __future__ import annotations

import itertools

import pytest
import torch

from forge_engine_b200.config.registry import read_model_config
from forge_engine_b200.parts.base import BuildContext
from forge_engine_b200.parts.latent_attention import LatentAttention


def mixers(layers, heads=2, rank=32, rot=32, q_rank=16, width=32, wide=()):
    """A mixer per (dim, vdim) of ``layers``, with weights on the CPU; layers ``wide`` store their key expansion
    in 32 bits."""
    raw = {"architecture": "Zofadra", "vocab": 32, "width": width, "norm": {"eps": 1e-5}, "layers": [
        {"type": "latent_attention", "mixer": {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": q_rank, "kv_rank": rank,
                                               "rot": {"base": 1e4, "dims": rot}, "scale": (dim + rot) ** -0.5}} for dim, vdim in layers]}
    _, _, spec = read_model_config(raw)
    made = []
    for i, layer in enumerate(spec.layers):
        weights = {name: torch.zeros(info.shape, dtype=torch.float32 if i in wide and name.endswith("uk") else torch.bfloat16)
                   for name, info in LatentAttention.weight_shapes(layer.mixer).items()}
        made.append(LatentAttention(layer.mixer, weights, BuildContext(torch.bfloat16, torch.device("cpu"), None)))
    return made


@pytest.mark.parametrize("sizes, wide", (([(64, 64), (128, 128), (96, 48)], ()), ([(64, 64), (64, 64)], (1,))))
def test_a_layer_is_given_a_plan_it_can_carry_out(sizes, wide):
    """Layers of the same heads, rank and rotated part, of which some cannot expand keys and values (heads too
    wide, values not in thirty-twos, a matrix stored in 32 bits), in every order: a plan expands entries where
    the layer can, and only there."""
    can = [dim + 32 <= 128 and vdim <= 128 and vdim % 32 == 0 and i not in wide for i, (dim, vdim) in enumerate(sizes)]
    for order in itertools.permutations(range(len(sizes))):
        made, plans = mixers([sizes[i] for i in order], wide=[order.index(i) for i in wide]), {}
        for mixer in made:
            mixer.plan_step([(0, 0, 600)], 16, plans)
        for i, mixer in zip(order, made):
            assert (mixer.expanded is not None) == can[i]
            assert (plans[mixer.plan_key][1] is not None) == can[i], order


@pytest.mark.parametrize("window", (None, 1, 40, 200, 1000))
def test_pairs_of_queries_and_keys(window):
    mixer = object.__new__(LatentAttention)
    mixer.window = window
    for start in (0, 1, 39, 40, 41, 500):
        for count in (1, 2, 39, 40, 41, 300):
            want = sum(min(start + i + 1, window or 10**9) for i in range(count))
            assert mixer._pairs([(0, start, count)]) == want, (start, count)


@pytest.mark.parametrize("decoders, portions, expands", ((0, [(0, 600)], True), (0, [(0, 300), (0, 300)], True), (0, [(0, 512)], False),
                                                         (8, [(0, 700)], False), (100, [(0, 430)], False), (48, [(2000, 1000)], True)))
def test_portions_beside_other_entries_are_expanded_where_that_pays_for_both_forms(decoders, portions, expands):
    """32 heads of rank 256: a step without short entries expands above 512 tokens; beside decoding requests
    the portions' attention has to be long enough to pay for the second set of launches."""
    mixer, = mixers([(64, 64)], heads=32, rank=256)
    entries, plans = [(i, 2000, 1) for i in range(decoders)] + [(99, s, n) for s, n in portions], {}
    mixer.plan_step(entries, 16, plans)
    splits, spans = plans[mixer.plan_key]
    assert (spans is not None) == expands and (splits is None) == (expands and not decoders)


@pytest.mark.parametrize("rank, rot, least", ((16, 32, 385), (32, 16, 129), (32, 32, 129), (256, 32, 129)))
def test_portions_are_expanded_from_a_length_that_depends_on_the_rank(rank, rot, least):
    mixer, = mixers([(64, 64)], rank=rank, rot=rot)
    for count, spans in ((least - 1, None), (least, ((60, least),) * 8)):
        plans = {}
        mixer.plan_step([(i, 60, count) for i in range(8)], 16, plans)
        assert plans[mixer.plan_key][1] == spans


@pytest.mark.parametrize("heads", (1, 3, 32, 128))
def test_expanded_keys_and_values_are_held_within_bounds(heads):
    """Whatever the contexts of a step add up to, the keys and values held at a time take at most 1 GiB, or one
    head's; every head has its turn, in stretches that differ by less than one head's share."""
    mixer = object.__new__(LatentAttention)
    mixer.h = heads
    for rows in (128, 4096, 65536, 480 * 1024, 1 << 20, 1 << 22):
        most = mixer._heads_at_once(rows)
        assert 1 <= most <= heads and (most == 1 or most * rows * 512 <= 1 << 30)
        turns = -(-heads // most)
        assert most == -(-heads // turns) and (turns == 1 or rows * 512 * -(-heads // (turns - 1)) > 1 << 30)
