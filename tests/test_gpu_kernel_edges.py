"""Kernels at the sizes where their tiles, stretches and choices between forms begin and end, each
against 64-bit arithmetic on the same inputs."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def native():
    from forge_engine_b200.ops import native as module

    module.require_cuda()
    module.lib()
    return module


# -- 32-bit products -------------------------------------------------------------------------------
@pytest.mark.parametrize("xd, wd", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("o, k", [(7, 8), (33, 128), (2049, 136), (2056, 264), (8200, 24), (8193, 40)])
def test_product_of_any_number_of_rows(native, xd, wd, o, k):
    """Row counts at the edges of the forms for few rows and of the tiles, outputs at the edges of their
    column counts, depths of a part and of several stretches of 128 (and one whose rows do not start on 16
    bytes): within the bound of a sum of k products each rounded once, and a row's bits do not depend on how
    many others there are."""
    gen = torch.Generator().manual_seed(o + k)
    w = torch.randn((o, k), generator=gen).to(wd).to(DEV)
    rows = torch.randn((131, k), generator=gen).to(xd).to(DEV)
    bias = torch.randn(o, generator=gen).to(DEV)
    bound = (rows.double().abs() @ w.double().abs().t() + bias.double().abs()) * (k + 1) * 2.0**-24
    want = rows.double() @ w.double().t() + bias.double()
    first = None
    for n in (1, 2, 4, 5, 8, 16, 17, 64, 65, 131):
        got = torch.empty((n, o), device=DEV)
        native.gemm_simt(rows[:n].contiguous(), w, got, bias)
        assert bool(((got.double() - want[:n]).abs() <= bound[:n]).all()), n
        first = got[0].clone() if first is None else first
        assert torch.equal(got[0], first), n
    odd = rows[:, : k - 1].contiguous(), w[:, : k - 1].contiguous()
    for n in (3, 70):
        got = torch.empty((n, o), device=DEV)
        native.gemm_simt(odd[0][:n].contiguous(), odd[1], got)
        assert bool(((got.double() - odd[0][:n].double() @ odd[1].double().t()).abs() <= bound[:n]).all()), n


@pytest.mark.parametrize("n", (1, 6, 40, 90))
def test_batched_product_with_strided_rows(native, n):
    gen = torch.Generator().manual_seed(n)
    batch, o, k = 3, 70, 48
    x = torch.randn((n, batch, k + 8), generator=gen).to(DEV)[:, :, :k]
    w = torch.randn((batch, o, k), generator=gen).to(DEV)
    out = torch.full((n, batch, o + 3), 7.0, device=DEV)
    native.gemm_simt_batched(x, w, out[:, :, :o])
    want = torch.einsum("nbk,bok->nbo", x.double(), w.double())
    bound = torch.einsum("nbk,bok->nbo", x.double().abs(), w.double().abs()) * (k + 1) * 2.0**-24
    assert bool(((out[:, :, :o].double() - want).abs() <= bound).all())
    assert float((out[:, :, o:] - 7.0).abs().max()) == 0.0
