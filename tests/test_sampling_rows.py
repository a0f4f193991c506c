"""The parameters that travel with a launch of the sampling kernel are those that the array form holds."""

from __future__ import annotations

import math
import struct

import pytest
import torch

from forge_engine_b200.sampling.params import SamplingParams
from forge_engine_b200.sampling.sampler import packed_rows


@pytest.mark.parametrize("temperature", (0.0, 1e-50, 0.8, 1, 3.4028234e38, 3.40282356e38, 3.4028235677973366e38, 1e39, 1.7e308))
@pytest.mark.parametrize("top_k", (None, 1, 50, 50.0, 2.5, (1 << 31) - 1))
def test_rows_hold_what_tensors_hold(temperature, top_k):
    params = [SamplingParams(temperature=temperature, top_k=top_k, top_p=0.9, min_p=0.05), SamplingParams(temperature=0.7)]
    seeds, counters = [-3, (1 << 64) + 5], [0, (1 << 63) + 1]
    first = struct.unpack("=" + "3fi2Q" * 2, packed_rows(params, seeds, counters))[:6]
    floats = torch.tensor([temperature, 0.9, 0.05], dtype=torch.float32).tolist()
    assert list(first) == floats + [torch.tensor([top_k or 0], dtype=torch.int32).item(), (1 << 64) - 3, 0]
    assert math.isinf(first[0]) == (temperature > 3.40282356e38)
