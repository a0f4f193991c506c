"""Kernels at the sizes where their tiles, stretches and choices between forms begin and end, each
against 64-bit arithmetic on the same inputs."""

from __future__ import annotations

import struct

import pytest
import torch

from test_gpu_kernels import dense_attention, paged_layout, status_word, twin_uniform

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


@pytest.mark.parametrize("xd, wd", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("n, o, k", ((33, 2100, 65), (65, 4200, 31), (130, 9000, 33), (500, 1300, 127), (40, 64, 1)))
def test_product_of_rows_off_16_bytes(native, xd, wd, n, o, k):
    """Odd depths in both tile sizes, one operand or both a number at a time."""
    gen = torch.Generator().manual_seed(n + k)
    x, w = torch.randn((n, k), generator=gen).to(xd).to(DEV), torch.randn((o, k), generator=gen).to(wd).to(DEV)
    got = torch.empty((n, o), device=DEV)
    native.gemm_simt(x, w, got)
    bound = (x.double().abs() @ w.double().abs().t()) * (k + 1) * 2.0**-24
    assert bool(((got.double() - x.double() @ w.double().t()).abs() <= bound).all())


@pytest.mark.parametrize("n, o, k", ((1, 100, 1024), (4, 300, 1152), (16, 9000, 2048)))
def test_a_wait_that_runs_out_is_reported(native, n, o, k):
    """Loaders that do not report a stretch of k: the block gives up after a few polls, the status word says so and
    the rows are NaN; the next call is sound again."""
    gen = torch.Generator().manual_seed(o)
    x, w = (torch.randn(shape, generator=gen).to(DEV) for shape in ((n, k), (o, k)))
    good, bad, again = (torch.empty((n, o), device=DEV) for _ in range(3))
    status = status_word()
    native.gemm_simt(x, w, good, status=status)
    assert int(status.item()) == 0
    try:
        native.gemm_simt_set_test_fault(2000, 2)
        native.gemm_simt(x, w, bad, status=status)
        torch.cuda.synchronize()
    finally:
        native.gemm_simt_set_test_fault()
    assert int(status.item()) == 8 and not bool(torch.isfinite(bad).any())
    native.gemm_simt(x, w, again, status=status_word())
    assert torch.equal(again, good)


@pytest.mark.parametrize("xd, wd", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("n, o, k", ((1, 100, 1152), (4, 5000, 2048), (16, 9000, 1152), (4, 40100, 1024)))
def test_a_wait_that_runs_out_in_either_kernel_for_few_rows(native, xd, wd, n, o, k):
    """The kernel of multiply-adds, whose ring these depths go round (operands of mixed types and of 16 bits go there whatever their
    depth), and the one on the tensor cores where one block takes all of k."""
    assert xd != wd or wd != torch.float32 or o < 40000 or native.lib().fe_gemm_split_cuts(n, o, k, 1) == 1
    gen = torch.Generator().manual_seed(o)
    x, w = torch.randn((n, k), generator=gen).to(xd).to(DEV), torch.randn((o, k), generator=gen).to(wd).to(DEV)
    good, bad, again = (torch.empty((n, o), device=DEV) for _ in range(3))
    status = status_word()
    native.gemm_simt(x, w, good, status=status)
    bound = (x.double().abs() @ w.double().abs().t()) * (k + 1) * 2.0**-24
    assert int(status.item()) == 0 and bool(((good.double() - x.double() @ w.double().t()).abs() <= bound).all())
    try:
        native.gemm_simt_set_test_fault(2000, 2)
        native.gemm_simt(x, w, bad, status=status)
        torch.cuda.synchronize()
    finally:
        native.gemm_simt_set_test_fault()
    assert int(status.item()) == 8 and not bool(torch.isfinite(bad).any())
    native.gemm_simt(x, w, again, status=status_word())
    assert torch.equal(again, good)


def test_layers_give_products_their_status_word(native, monkeypatch):
    from forge_engine_b200.parts.linear import Linear

    seen, status = [], status_word()
    monkeypatch.setattr(native, "gemm_simt", lambda *args, status=None, **kw: seen.append(status))
    Linear(torch.randn(8, 16, device=DEV), status=status)(torch.randn(2, 16, device=DEV))
    assert len(seen) == 1 and seen[0] is status


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, rows, k", ((1185, 8, 36), (1186, 3, 37), (1187, 9, 48), (1184, 8, 1), (600, 12, 130), (593, 16, 6400), (593, 16, 6408)))
def test_router_logits_of_many_tokens(native, dtype, n, rows, k):
    """Four tokens a block, with a rest of one to three and widths off eight and off four: the bits of a token a block (few
    tokens go there), and within a chain's bound of 64 bits.  The last width is the first whose four tokens do not fit."""
    gen = torch.Generator().manual_seed(n + k)
    x, w, bias = torch.randn((n, k), generator=gen).to(dtype).to(DEV), torch.randn((rows, k), generator=gen).to(DEV), torch.randn(rows, generator=gen).to(DEV)
    got, alone = torch.empty((n, rows), device=DEV), torch.empty((n, rows), device=DEV)
    native.moe_logits(x, w, got, bias)
    for at in range(0, n, 100):
        native.moe_logits(x[at : at + 100].contiguous(), w, alone[at : at + 100], bias)
    assert torch.equal(got, alone)
    bound = (x.double().abs() @ w.double().abs().t() + bias.double().abs()) * (k + 2) * 2.0**-24
    assert bool(((got.double() - x.double() @ w.double().t() - bias.double()).abs() <= bound).all())


# -- 32-bit attention --------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, page, window", [
    (4, 2, 64, 16, None), (16, 8, 128, 16, None), (6, 1, 40, 4, 50), (20, 1, 16, 8, None), (4, 4, 256, 32, 130), (9, 3, 72, 2, 1)])
def test_attention_of_entries(native, dtype, nq, nkv, d, page, window):
    """Entries of one token (at both sides of a span of 128 positions) beside entries of several (at both
    sides of a tile of 32 rows and of 64 keys), each also alone: the same bits, and the dense result."""
    lengths = [300, 1, 128, 129, 257, 64, 65, 400]
    counts = [1, 1, 1, 1, 33, 64, 2, 17]
    k_cache, v_cache, table, keys, values = paged_layout(lengths, page, nkv, d, dtype, seed=d + nq)
    gen = torch.Generator().manual_seed(5)
    positions = [p for n, c in zip(lengths, counts) for p in range(n - c, n)]
    entry = [e for e, c in enumerate(counts) for _ in range(c)]
    q = torch.randn((len(positions), nq, d), generator=gen).to(dtype)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)
    status = status_word()

    def attend(rows, table, cu_tokens):
        out = torch.empty((len(rows), nq * d), dtype=dtype, device=DEV)
        native.attention_simt(q[rows].reshape(len(rows), nq * d).to(DEV), nq * d, k_cache, v_cache, table, ints([positions[r] for r in rows]),
                              ints([0 if table.shape[0] == 1 else entry[r] for r in rows]), window, d ** -0.5, out, nq, status,
                              entries=(ints(cu_tokens), len(cu_tokens) - 1, max(b - a for a, b in zip(cu_tokens, cu_tokens[1:]))))
        return out

    together = attend(list(range(len(positions))), table, cu)
    assert int(status.item()) == 0
    for e, count in enumerate(counts):
        rows = list(range(cu[e], cu[e + 1]))
        assert torch.equal(attend(rows, table[e : e + 1].contiguous(), [0, count]), together[rows])
        want = dense_attention(q[rows], keys[e], values[e], torch.tensor([positions[r] for r in rows]), d ** -0.5, window)
        mine = together[rows].view(count, nq, d).double().cpu()
        torch.testing.assert_close(mine, want, **(dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, window", [(32, 32, 64, None), (30, 30, 40, 150), (16, 16, 128, 300), (32, 16, 256, None)])
def test_attention_of_portions_that_fill_the_chip(native, dtype, nq, nkv, d, window):
    """A portion of enough row tiles that a block folds all spans of its rows itself, after cached keys and beside a shorter
    one: the bits of the same tokens in pieces small enough that every span has blocks of its own, and the dense result."""
    page, lengths, counts = 16, [900, 300], [840, 33]
    k_cache, v_cache, table, keys, values = paged_layout(lengths, page, nkv, d, dtype, seed=d)
    positions = [p for n, c in zip(lengths, counts) for p in range(n - c, n)]
    entry = [e for e, c in enumerate(counts) for _ in range(c)]
    q = torch.randn((len(positions), nq, d), generator=torch.Generator().manual_seed(5)).to(dtype)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    floats, status = native.lib().fe_attention_simt_tile_scratch, status_word()

    def attend(rows, table, cu):
        out = torch.empty((len(rows), nq * d), dtype=dtype, device=DEV)
        native.attention_simt(q[rows].reshape(len(rows), nq * d).to(DEV), nq * d, k_cache, v_cache, table, ints([positions[r] for r in rows]),
                              ints([0 if table.shape[0] == 1 else entry[r] for r in rows]), window, d ** -0.5, out, nq, status,
                              entries=(ints(cu), len(cu) - 1, max(b - a for a, b in zip(cu, cu[1:]))))
        return out

    assert floats(len(positions), 2, nq, nkv, d, table.shape[1], page) == 0
    together = attend(list(range(len(positions))), table, [0, 840, 873])
    for first, last in ((0, 31), (31, 64), (64, 164), (164, 290), (290, 417), (417, 500), (740, 840), (840, 873)):
        one = table[entry[first] : entry[first] + 1].contiguous()
        assert floats(last - first, 1, nq, nkv, d, one.shape[1], page) > 0
        assert torch.equal(attend(list(range(first, last)), one, [0, last - first]), together[first:last]), first
    assert int(status.item()) == 0
    for e, at in ((0, 0), (1, 840)):
        want = dense_attention(q[at : at + counts[e]], keys[e], values[e], torch.tensor(positions[at : at + counts[e]]), d ** -0.5, window)
        mine = together[at : at + counts[e]].view(counts[e], nq, d).double().cpu()
        torch.testing.assert_close(mine, want, **(dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, window, wide", [(16, 16, 64, None, 0), (32, 8, 40, None, 300), (16, 16, 128, 700, 0), (16, 2, 256, None, 0), (8, 8, 64, 100, 400)])
def test_attention_spans_that_blocks_share(native, dtype, nq, nkv, d, window, wide):
    """More spans than blocks share a row tile of a long portion, windows that leave most spans unseen, and block tables far
    wider than a request's pages: the bits of the same tokens in pieces with blocks for every span, and the dense result."""
    page, lengths, counts = 16, [3000, 60], [190, 60]
    k_cache, v_cache, table, keys, values = paged_layout(lengths, page, nkv, d, dtype, seed=d)
    table = torch.nn.functional.pad(table, (0, wide), value=-1)
    positions = [p for n, c in zip(lengths, counts) for p in range(n - c, n)]
    q = torch.randn((len(positions), nq, d), generator=torch.Generator().manual_seed(5)).to(dtype)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    status = status_word()

    def attend(first, last, entry):
        out = torch.empty((last - first, nq * d), dtype=dtype, device=DEV)
        one = table[entry : entry + 1].contiguous()
        assert native.lib().fe_attention_simt_tile_scratch(last - first, 1, nq, nkv, d, one.shape[1], page) > 0
        native.attention_simt(q[first:last].reshape(last - first, nq * d).to(DEV), nq * d, k_cache, v_cache, one, ints(positions[first:last]),
                              ints([0] * (last - first)), window, d ** -0.5, out, nq, status, entries=(ints([0, last - first]), 1, last - first))
        return out

    for entry, first, last, step in ((0, 0, 190, 19), (1, 190, 250, 2)):
        together = attend(first, last, entry)
        for at in range(first, last, step):
            assert torch.equal(attend(at, at + step, entry), together[at - first : at - first + step]), at
        want = dense_attention(q[first:last], keys[entry], values[entry], torch.tensor(positions[first:last]), d ** -0.5, window)
        mine = together.view(last - first, nq, d).double().cpu()
        torch.testing.assert_close(mine, want, **(dict(atol=2e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)))
    assert int(status.item()) == 0


def test_attention_marks_missing_pages_and_keeps_later_infinities_out(native):
    """A position without a page sets the status bit; an infinite value of a later token of the same tile
    changes no earlier row."""
    k_cache, v_cache, table, keys, values = paged_layout([40], 8, 1, 16, torch.float32, seed=3)
    q = torch.randn((40, 2, 16), generator=torch.Generator().manual_seed(1))
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731

    def attend(table, positions, cu):
        out, status = torch.empty((len(positions), 32), device=DEV), status_word()
        native.attention_simt(q[positions].reshape(len(positions), 32).to(DEV), 32, k_cache, v_cache, table, ints(positions),
                              ints([0] * len(positions)), None, 0.25, out, 2, status, entries=(ints(cu), 1, len(positions)))
        return out, int(status.item())

    clean, status = attend(table, list(range(40)), [0, 40])
    assert status == 0
    v_cache[int(table[0, 39 // 8]), :, 39 % 8] = float("inf")
    loud, status = attend(table, list(range(40)), [0, 40])
    assert status == 0 and torch.equal(loud[:39], clean[:39]) and not bool(torch.isfinite(loud[39]).any())
    holed = table.clone()
    holed[0, 1] = -1
    assert attend(holed, list(range(40)), [0, 40])[1] & 2
    assert attend(holed, [30], [0, 1])[1] & 2
    assert attend(table[:, :2].contiguous(), [39], [0, 1])[1] & 2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, window", [(4, 2, 64, None), (6, 1, 40, 50), (4, 4, 256, 130), (9, 3, 72, 300)])
def test_attention_of_a_portion_cut_in_any_way(native, dtype, nq, nkv, d, window):
    """A prompt in one portion, in two, as single tokens and as tokens without entries: the same bits."""
    length, page = 333, 16
    k_cache, v_cache, table, _, _ = paged_layout([length], page, nkv, d, dtype, seed=d)
    q = torch.randn((length, nq * d), generator=torch.Generator().manual_seed(4)).to(dtype).to(DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    status = status_word()

    def attend(first, last, cu=None):
        out = torch.empty((last - first, nq * d), dtype=dtype, device=DEV)
        rows = table if cu is None else table.expand(len(cu) - 1, -1).contiguous()
        entry = [0] * (last - first) if cu is None else [e for e in range(len(cu) - 1) for _ in range(cu[e + 1] - cu[e])]
        native.attention_simt(q[first:last].contiguous(), nq * d, k_cache, v_cache, rows, ints(list(range(first, last))), ints(entry), window,
                              d ** -0.5, out, nq, status, entries=None if cu is None else
                              (ints(cu), len(cu) - 1, max(b - a for a, b in zip(cu, cu[1:]))))
        return out

    whole = attend(0, length, [0, length])
    assert torch.equal(attend(0, length), whole)
    assert torch.equal(attend(0, length, list(range(length + 1))), whole)
    for cut in (1, 64, 127, 200, length - 1):
        assert torch.equal(torch.cat((attend(0, cut, [0, cut]), attend(cut, length, [0, length - cut]))), whole), cut
        assert torch.equal(attend(0, length, [0, cut, length]), whole), cut
    assert int(status.item()) == 0


def test_attention_keeps_its_partial_results_to_itself(native, monkeypatch):
    """Runs on several streams share no buffer, and many single tokens beside one long block table take a bounded
    one: they go through it in slices, with the same results."""
    nq, nkv, d, page = 4, 2, 64, 16
    lengths = [1 + 37 * i for i in range(40)]
    k_cache, v_cache, table, _, _ = paged_layout(lengths, page, nkv, d, torch.float32, seed=2)
    q = torch.randn((40, nq * d), generator=torch.Generator().manual_seed(3)).to(DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    wide = torch.full((40, 32768), -1, dtype=torch.int32, device=DEV)
    wide[:, : table.shape[1]] = table
    monkeypatch.setattr(native, "_attention_workspace", None)
    status, outs = status_word(), []
    for t in (table, wide):
        sizes = (nq, nkv, d, t.shape[1], page)
        assert native.lib().fe_attention_simt_scratch(40, *sizes) <= 1 << 25
        assert (native.lib().fe_attention_simt_units(40, *sizes) < 40) == (t is wide)
        for entries in (None, (ints(list(range(41))), 40, 1)):
            out, before = torch.empty((40, nq * d), device=DEV), native.LAUNCHES
            native.attention_simt(q, nq * d, k_cache, v_cache, t, ints([n - 1 for n in lengths]), ints(list(range(40))), None, 0.125, out, nq,
                                  status, entries=entries)
            assert native.LAUNCHES - before == 2 * -(-40 // native.lib().fe_attention_simt_units(40, *sizes))
            outs.append(out)
    assert int(status.item()) == 0 and all(torch.equal(out, outs[0]) for out in outs[1:])


# -- gated recurrence ------------------------------------------------------------------------------
@pytest.mark.parametrize("heads, dk, dv, lead", ((2, 64, 64, 4), (1, 128, 128, 4), (1, 160, 100, 4), (2, 12, 260, 8), (1, 168, 36, 1), (3, 6, 8, 4)))
@pytest.mark.parametrize("counts", ([128], [129, 200, 3], [191, 1, 192, 130]))
def test_gated_recurrence_chunks(native, heads, dk, dv, lead, counts):
    """One stretch of 128 channels or columns and more, rows that start on 16 bytes and rows that do not,
    sub-chunks that are whole and that are cut; gates from nearly zero to one, from states that are not zero."""
    gen = torch.Generator().manual_seed(heads * 100 + dk + dv)
    qk, v, n = heads * dk, heads * dv, sum(counts)
    rand = lambda *shape: torch.randn(*shape, generator=gen)  # noqa: E731
    width = (lead + 2 * qk + v + 3) // 4 * 4
    proj = rand(n, width)
    proj[:, lead + qk : lead + 2 * qk] *= 4.0
    proj[5::7, lead + qk : lead + 2 * qk] = -40.0            # gates at their lower bound
    lower, bias, norm = torch.rand(qk, generator=gen) * 0.5, rand(qk), 1 + 0.2 * rand(dv)
    lower[: qk // 2] = 0.0
    state = rand(len(counts) + 1, heads, dk, dv)
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    got_state, out, status = state.to(DEV), torch.empty(n, v, device=DEV), status_word()
    native.gated_recurrence(proj.to(DEV), lead, lead + qk, lead + 2 * qk, bias.to(DEV), lower.to(DEV), norm.to(DEV), 1e-5, got_state,
                            ints(list(range(len(counts)))), ints(cu), out, len(counts), status, max_new=max(counts))
    assert int(status.item()) == 0
    rows = proj.double()
    q = torch.nn.functional.silu(rows[:, lead : lead + qk]).view(n, heads, dk)
    f = (lower.double() + (1 - lower.double()) * torch.sigmoid(rows[:, lead + qk : lead + 2 * qk] + bias.double())).view(n, heads, dk)
    val = rows[:, lead + 2 * qk : lead + 2 * qk + v].view(n, heads, dv)
    for e in range(len(counts)):
        s = state[e].double()
        want = torch.empty(counts[e], heads, dv, dtype=torch.float64)
        for i, t in enumerate(range(cu[e], cu[e + 1])):
            s = f[t][:, :, None] * s + (1 - f[t])[:, :, None] * val[t][:, None, :]
            want[i] = torch.einsum("hdv,hd->hv", s, q[t])
        want = (want * torch.rsqrt((want * want).mean(-1, keepdim=True) + 1e-5) * norm.double()).reshape(counts[e], v)
        assert float((out[cu[e] : cu[e + 1]].cpu().double() - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
        assert float((got_state[e].cpu().double() - s).abs().max()) <= 1e-5 * max(1.0, float(s.abs().max()))
    assert torch.equal(got_state[-1].cpu(), state[-1])       # the row of no entry


@pytest.mark.parametrize("dk", (4, 20, 36, 72, 100, 136))
def test_gated_recurrence_channels_off_sixteen(native, dk):
    """Products between sub-chunks over every remainder of sixteen channels; lanes with one, two and four channels."""
    test_gated_recurrence_chunks(native, 2, dk, 8, 4, [150, 133])


# -- delta rule: chunks ---------------------------------------------------------------------------
@pytest.mark.parametrize("kv_heads, heads, dk, dv", ((1, 2, 64, 64), (2, 2, 72, 40), (1, 1, 128, 128), (1, 2, 160, 36), (1, 1, 176, 64), (1, 1, 152, 100), (2, 4, 6, 10), (1, 1, 13, 5), (1, 1, 65, 129)))
@pytest.mark.parametrize("counts", ([96], [97, 160, 3], [191, 1, 192, 130]))
def test_delta_rule_chunks(native, kv_heads, heads, dk, dv, counts):
    """Heads that fill the fragments' eights and heads that do not (odd ones among them), chunks that are whole
    and that are cut, entries that are walked between them; from states that are not zero."""
    gen = torch.Generator().manual_seed(heads * 100 + dk + dv)
    n, qk = sum(counts), kv_heads * dk
    room = native.lib().fe_delta_rule_scratch
    assert room(n, len(counts), heads, dk, dv, max(counts)) > room(n, len(counts), heads, dk, dv, 1)      # not all of them walked
    rand = lambda *shape: torch.randn(*shape, generator=gen)  # noqa: E731
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    q, k, v = unit(rand(n, kv_heads, dk)) * dk**-0.5, unit(rand(n, kv_heads, dk)), rand(n, heads, dv)
    qkv = torch.cat((q.reshape(n, qk), k.reshape(n, qk), v.reshape(n, -1)), dim=1)
    gates = torch.stack((torch.rand(n, heads, generator=gen), -2.0 * torch.rand(n, heads, generator=gen) ** 4), dim=-1)
    gates[7::31, :, 1] = -60.0                               # the state all but forgotten
    gate, norm, state = rand(n, heads * dv), 1 + 0.2 * rand(dv), rand(len(counts) + 1, heads, dk, dv)
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    got_state, out, status = state.to(DEV), torch.empty(n, heads * dv, device=DEV), status_word()
    native.delta_rule(qkv.to(DEV), gates.to(DEV), gate.to(DEV), norm.to(DEV), 1e-3, got_state, ints(list(range(len(counts)))),
                      ints(cu), out, kv_heads, len(counts), max(counts), status)
    assert int(status.item()) == 0
    group = lambda x: x.double().repeat_interleave(heads // kv_heads, dim=1)  # noqa: E731
    q, k, v, beta, g = group(q), group(k), v.double(), gates[..., 0].double(), gates[..., 1].double().exp()
    for e in range(len(counts)):
        s = state[e].double()
        want = torch.empty(counts[e], heads, dv, dtype=torch.float64)
        for i, t in enumerate(range(cu[e], cu[e + 1])):
            s = g[t][:, None, None] * s
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", s, k[t]))
            s = s + k[t][:, :, None] * u[:, None, :]
            want[i] = torch.einsum("hkv,hk->hv", s, q[t])
        want = (want * torch.rsqrt((want * want).mean(-1, keepdim=True) + 1e-3) * norm.double()).reshape(counts[e], -1)
        want *= torch.nn.functional.silu(gate[cu[e] : cu[e + 1]].double())
        assert float((out[cu[e] : cu[e + 1]].cpu().double() - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
        assert float((got_state[e].cpu().double() - s).abs().max()) <= 1e-5 * max(1.0, float(s.abs().max()))
    assert torch.equal(got_state[-1].cpu(), state[-1])       # the row of no entry


# -- values that are not finite --------------------------------------------------------------------
@pytest.mark.parametrize("loud", (float("inf"), float("nan"), 3.4e38))
@pytest.mark.parametrize("name, dk, dv", (("gated", 64, 64), ("gated", 12, 100), ("gated", 12, 260), ("delta", 64, 64), ("delta", 72, 130),
                                          ("retention", 64, 64), ("retention", 40, 200), ("memory", 64, 64), ("memory", 24, 72)))
def test_a_loud_value_reaches_no_earlier_token(native, name, dk, dv, loud):
    """A value that is infinite, no number, or rounds to infinity as a bfloat16 number, late in a chunk: the rows of the
    tokens before it, and of other heads, are what they are without it, bit for bit."""
    heads, n = 2, 200
    gen = torch.Generator().manual_seed(dk + dv)
    rand = lambda *shape: torch.randn(*shape, generator=gen)  # noqa: E731
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    qk, v = heads * dk, heads * dv
    proj, gate, norm, gates = rand(n, 2 * qk + 2 * v + 2 * heads), rand(n, v), torch.ones(v, device=DEV), torch.rand(n, heads, 2, generator=gen)
    proj[:, : 2 * qk] *= dk**-0.5
    gates[..., 1] *= -0.2

    def run(values):
        p = proj.clone()
        p[:, 2 * qk : 2 * qk + v] = values
        p, state, status = p.to(DEV), torch.zeros(2, heads, dk, dv, device=DEV), status_word()
        out, slots, cu = torch.empty(n, v, device=DEV), ints([0]), ints([0, n])
        if name == "gated":
            native.gated_recurrence(p, 0, qk, 2 * qk, None, torch.zeros(qk, device=DEV), norm[:dv], 1e-5, state, slots, cu, out, 1, status, max_new=n)
        elif name == "delta":
            native.delta_rule(p[:, : 2 * qk + v].contiguous(), gates.to(DEV), gate.to(DEV), norm[:dv], 1e-5, state, slots, cu, out, heads, 1, n, status)
        elif name == "retention":
            native.retention(p, (0, qk, 2 * qk, 2 * qk + v), 1.0, torch.full((heads,), 0.97, device=DEV), None, 0, False, None, 1e-5, state, slots,
                             cu, out, 1, n, status)
        else:
            native.matrix_memory(p, (0, qk, 2 * qk, 2 * qk + v, 2 * qk + 2 * v, 2 * qk + 2 * v + heads), torch.full((heads,), -2.0, device=DEV),
                                 torch.full((heads,), 3.0, device=DEV), 15.0, 1.0, norm, 1e-5, state, torch.zeros(2, heads, dk, device=DEV),
                                 torch.zeros(2, heads, device=DEV), slots, cu, out, 1, n, status)
        assert int(status.item()) == 0
        return out.view(n, heads, dv)

    values = rand(n, v)
    clean = run(values)
    for at in (31, 50, 64, 127, 140):
        spoilt = values.clone()
        spoilt[at, dv // 2] = loud
        got = run(spoilt)
        assert torch.equal(got[:at], clean[:at]) and torch.equal(got[:, 1], clean[:, 1]), at
        assert not torch.equal(got[at, 0], clean[at, 0])


# -- delta rule's inputs ---------------------------------------------------------------------------
@pytest.mark.parametrize("taps, dk, dv", ((2, 64, 64), (3, 32, 20), (4, 128, 128), (4, 40, 64), (4, 6, 10), (5, 64, 64)))
@pytest.mark.parametrize("counts", ([256], [1, 2, 3, 270, 1], [100, 100, 57]))
def test_delta_prepare_of_many_tokens(native, taps, dk, dv, counts):
    """Runs of tokens that begin and end inside entries, entries shorter than the taps between them."""
    gen = torch.Generator().manual_seed(taps * 100 + dk)
    heads, kv, n = 4, 2, sum(counts)
    channels = 2 * kv * dk + heads * dv
    rand = lambda *shape: torch.randn(*shape, generator=gen, dtype=torch.float64)  # noqa: E731
    proj, conv, a_log, dt = rand(n, channels + heads * dv + 2 * heads), rand(channels, taps), rand(heads), rand(heads)
    state = rand(len(counts) + 1, taps - 1, channels)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)
    want, want_state = torch.empty(n, channels, dtype=torch.float64), state.clone()
    for e in range(len(counts)):
        rows = torch.cat([state[e], proj[cu[e] : cu[e + 1], :channels]])
        y = sum(rows[j : j + counts[e]] * conv[:, j] for j in range(taps))
        y = y * torch.sigmoid(y)
        for r in range(2 * kv):
            part = y[:, r * dk : (r + 1) * dk]
            part *= torch.rsqrt((part * part).sum(-1, keepdim=True) + 1e-6) * (dk ** -0.5 if r < kv else 1.0)
        want[cu[e] : cu[e + 1]] = y
        want_state[e] = rows[counts[e] :]
    b, a = proj[:, channels + heads * dv : -heads], proj[:, -heads:]
    want_gates = torch.stack([torch.sigmoid(b), -torch.exp(a_log) * torch.nn.functional.softplus(a + dt)], dim=-1)
    dev = lambda t: t.float().to(DEV).contiguous()  # noqa: E731
    out, gates, got_state = torch.empty(n, channels, device=DEV), torch.empty(n, heads, 2, device=DEV), dev(state)
    native.delta_prepare(dev(proj), channels + heads * dv, channels + heads * dv + heads, dev(conv.T), got_state, ints(list(range(len(counts)))),
                         ints(cu), ints([e for e, c in enumerate(counts) for _ in range(c)]), dev(a_log), dev(dt), kv, dk, heads, dv, out,
                         gates, len(counts))
    for mine, ref in ((out, want), (gates, want_gates), (got_state, want_state)):
        assert float((mine.cpu() - ref).abs().max()) <= 2e-5 * max(1.0, float(ref.abs().max()))


# -- sampling -------------------------------------------------------------------------------------
def drawn(row, temperature, top_k, top_p, u):
    """(index, running sums, target): among equal values top-k keeps the lowest indices and top-p all or none."""
    x = row.double() / temperature
    x = x - x.max()
    keep = torch.ones_like(x, dtype=torch.bool)
    if top_k:
        keep[:] = False
        keep[torch.sort(x, descending=True, stable=True).indices[:top_k]] = True
    if top_p < 1.0:
        values, where = torch.unique(x[keep], return_inverse=True)
        mass = torch.zeros_like(values).index_add_(0, where, torch.exp(x[keep]))
        above = mass.flip(0).cumsum(0).flip(0) - mass            # of the larger values
        keep &= x >= values[above <= top_p * mass.sum()].min()
    weights = torch.where(keep, torch.exp(x), torch.zeros_like(x))
    running, target = torch.cumsum(weights, 0), u * float(weights.sum())
    index = int(torch.searchsorted(running, torch.tensor(target, dtype=torch.float64), right=True))
    return min(index, int(torch.nonzero(weights > 0)[-1])), running, target


def test_blocks_of_a_row_run_at_once(native):
    """A block has an SM to itself and clusters fit only whole: the rows of a call are cut so that they take no more rounds
    than they have to."""
    parts = native.lib().fe_sample_parts
    assert [parts(n, 151936) for n in (1, 8, 24, 28, 64, 128)] == [8, 8, 4, 4, 4, 1]
    assert [parts(n, 32000) for n in (1, 16, 28, 40, 70, 128, 256)] == [4, 4, 4, 2, 2, 1, 1]
    assert [parts(n, 300000) for n in (12, 28, 64, 128)] == [8, 8, 2, 2] and parts(1, 8191) == 1 and parts(1, 8192) == 2


@pytest.mark.parametrize("rows, vocab", ((1, 4096), (3, 16385), (40, 32768), (64, 151936), (5, 300000), (25, 300000), (2, 700001)))
@pytest.mark.parametrize("top_k, top_p", ((0, 1.0), (37, 1.0), (0, 0.8), (50, 0.9)))
def test_sampling_of_long_rows(native, rows, vocab, top_k, top_p):
    """Slices that are kept in shared memory and slices that are not, rows in one block and in several; ties
    at the k-th value.  A draw may differ only where its target lies within rounding of a boundary."""
    gen = torch.Generator().manual_seed(rows + vocab)
    base = torch.randn(vocab, generator=gen) * 2.0
    base[torch.randint(0, vocab, (60,), generator=gen)] = 9.0
    seeds = torch.arange(rows, dtype=torch.int64) * 31 + 3
    out, status = torch.empty(rows, dtype=torch.int32, device=DEV), status_word()
    dev = lambda value, dtype: torch.full((rows,), value, dtype=dtype, device=DEV)  # noqa: E731
    native.sample(base[None].repeat(rows, 1).to(DEV), out, status, temperature=dev(0.8, torch.float32), top_k=dev(top_k, torch.int32),
                  top_p=dev(top_p, torch.float32), min_p=dev(0.0, torch.float32), seeds=seeds.to(DEV),
                  counters=torch.zeros(rows, dtype=torch.int64, device=DEV))
    assert int(status.item()) == 0
    for r in range(min(rows, 4)):
        want, running, target = drawn(base, 0.8, top_k, top_p, twin_uniform(int(seeds[r]), 0))
        if int(out[r]) != want:
            assert float((running - target).abs().min()) < 1e-5 * float(running[-1]), (r, int(out[r]), want)


# -- attention over cached latents -------------------------------------------------------------------
@pytest.mark.parametrize("window, sink", ((None, False), (200, True), (40, False)))
@pytest.mark.parametrize("heads, dim, rot, vdim, rank", ((3, 64, 32, 64, 64), (2, 96, 32, 128, 48), (4, 16, 16, 32, 32)))
def test_expanded_latent_attention(native, monkeypatch, window, sink, heads, dim, rot, vdim, rank):
    """Portions of 129 tokens and more beside shorter ones, keys and values expanded, against the absorbed form
    of the same layer and against 64 bits."""
    import dataclasses

    from forge_engine_b200.config.registry import read_model_config
    from forge_engine_b200.engine import ModelRunner, StepEntry
    from forge_engine_b200.engine.batch import build_batch
    from forge_engine_b200.parts import latent_attention as part

    width, q_rank = 128, 64
    raw = {"architecture": "Zofadra", "vocab": 32, "width": width, "norm": {"eps": 1e-5}, "layers": [{"type": "latent_attention", "mixer": {
        "heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": q_rank, "kv_rank": rank,
        "rot": {"base": 1e4, "dims": rot}, "scale": (dim + rot) ** -0.5}}]}
    arch, _, spec = read_model_config(raw)
    layer = spec.layers[0]
    spec = dataclasses.replace(spec, layers=(dataclasses.replace(layer, mixer=dataclasses.replace(layer.mixer, window=window, sink=sink)),))
    gen = torch.Generator().manual_seed(heads + dim)
    weights = {name: ((1 + 0.1 * torch.randn(info.shape, generator=gen)) if "norm" in name else
                      torch.randn(info.shape, generator=gen) * (info.shape[-1] ** -0.5 if len(info.shape) > 1 else 1.0)).bfloat16().to(DEV)
               for name, info in arch.expected_tensors(spec).items()}
    counts, starts = [130, 5, 257, 1, 400], [0, 60, 37, 9, 250]
    x = torch.randn((sum(counts), width), generator=gen).bfloat16().to(DEV)
    before = torch.randn((max(starts), rank + rot), generator=gen).bfloat16().to(DEV)
    results = {}
    for name, step in (("expanded", 512), ("absorbed", 1 << 30)):
        monkeypatch.setattr(part, "EXPAND_STEP", step)
        monkeypatch.setattr(part, "EXPAND_BESIDE", 0.0)
        runner = ModelRunner.from_tensors(spec, dict(weights), dtype="bfloat16", device=DEV, page_size=16, num_pages=128, max_requests=6,
                                          architecture=arch)
        cache = runner.cache
        for i, start in enumerate(starts):
            runner.begin(i)
            if start:
                cache.reserve(i, start)
                cache.advance(i, start)
                pages = cache.request(i).tables[0].pages
                for p in range(start):
                    if pages[p // 16] >= 0:
                        cache.kv_of_run(0)[0][pages[p // 16], 0, p % 16] = before[p]
        entries = [StepEntry(i, [0] * c) for i, c in enumerate(counts)]
        for i, (start, count) in enumerate(zip(starts, counts)):
            cache.reserve(i, start + count)
        batch = build_batch(entries, cache, DEV)
        results[name] = runner.model.blocks[0].mixer.attend(x, batch, cache.view(0)).clone()
        assert batch.plans[runner.model.blocks[0].mixer.plan_key][1] == (tuple(zip(starts, counts)) if name == "expanded" else None)
        runner.check_status()
    w = {k.split(".mix.")[-1]: v.double().cpu() for k, v in weights.items()}
    rms = lambda t, g: t * torch.rsqrt((t * t).mean(-1, keepdim=True) + 1e-5) * g  # noqa: E731

    def turned(t, positions):
        angle = positions.double()[:, None] * 1e4 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / rot)
        cos, sin = torch.cos(angle), torch.sin(angle)
        if t.dim() == 3:
            cos, sin = cos[:, None], sin[:, None]
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack((a * cos - b * sin, b * cos + a * sin), dim=-1).flatten(-2)

    at = 0
    for start, count in zip(starts, counts):
        h = x[at : at + count].double().cpu()
        positions = torch.arange(start, start + count)
        q = (rms(h @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(count, heads, dim + rot)
        q = torch.cat((q[..., :dim], turned(q[..., dim:], positions)), dim=-1)
        both = h @ w["dkv"].T
        own = torch.cat((rms(both[:, :rank], w["dkv.norm"]), turned(both[:, rank:], positions)), dim=-1)
        latents = torch.cat((before[:start].double().cpu(), own))
        keys = torch.cat(((latents[:, :rank] @ w["uk"].T).view(-1, heads, dim), latents[:, None, rank:].expand(-1, heads, -1)), dim=-1)
        values = (latents[:, :rank] @ w["uv"].T).view(-1, heads, vdim)
        scores = torch.einsum("thd,shd->hts", q, keys) * (dim + rot) ** -0.5
        distance = positions[:, None] - torch.arange(start + count)[None, :]
        hidden = (distance < 0) | ((distance >= window) if window else torch.zeros_like(distance, dtype=torch.bool))
        e = torch.exp(scores.masked_fill(hidden, float("-inf")))
        total = e.sum(-1, keepdim=True) + (torch.exp(w["sink"])[:, None, None] if sink else 0.0)
        want = torch.einsum("hts,shd->thd", e / total, values).reshape(count, -1)
        for name, got in results.items():
            off = float((got[at : at + count].double().cpu() - want).norm() / want.norm())
            assert off < 1e-2, (name, start, count, off)
        at += count


# -- deep 32-bit products on the tensor cores --------------------------------------------------------
@pytest.mark.parametrize("o, k", ((1, 256), (127, 260), (129, 320), (300, 1028), (4224, 448), (2500, 3072)))
def test_deep_product_of_any_number_of_rows(native, o, k):
    """Row counts at the edges of the four tiles, depths with and without a rest of a stretch of 64 and with fewer stretches
    than parts: a row's bits do not depend on the others (nor on how k is cut over blocks, which changes with them).  Bound: a
    stretch's sum is off by its 24 additions in the tensor core (2^-23 of the sum of magnitudes each), the sums outside by
    2^-24 each; along a random result far less, and less than one chain of multiply-adds (2.9e-7 at 256)."""
    gen = torch.Generator().manual_seed(o + k)
    w, rows = (torch.randn(shape, generator=gen).to(DEV) for shape in ((o, k), (300, k)))
    bias = torch.randn(o, generator=gen).to(DEV)
    want = rows.double() @ w.double().t()
    bound = (rows.double().abs() @ w.double().abs().t()) * (24 * 2.0**-23 + (k // 64 + 10) * 2.0**-24) + 2.0**-22 * bias.double().abs()
    whole = torch.empty((300, o), device=DEV)
    native.gemm_simt(rows, w, whole)
    assert float((whole.double() - want).norm() / want.norm()) < 2.5e-7
    for n in (1, 16, 17, 32, 33, 64, 65, 128, 129):
        got = torch.empty((n, o), device=DEV)
        native.gemm_simt(rows[:n].contiguous(), w, got)
        assert torch.equal(got, whole[:n]), n
        added = torch.ones((n, o), device=DEV)
        native.gemm_simt(rows[:n].contiguous(), w, added, bias, accumulate=True)
        assert bool(((added.double() - 1.0 - bias.double() - want[:n]).abs() <= bound[:n] + 2.0**-22).all()), n


def test_deep_batched_product_with_strided_rows(native):
    gen = torch.Generator().manual_seed(3)
    batch, o, k = 3, 140, 272
    w = torch.randn((batch, o, k), generator=gen).to(DEV)
    for n in (1, 20, 150):
        x = torch.randn((n, batch, k + 8), generator=gen).to(DEV)[:, :, :k]
        out = torch.full((n, batch, o + 3), 7.0, device=DEV)
        native.gemm_simt_batched(x, w, out[:, :, :o])
        want = torch.einsum("nbk,bok->nbo", x.double(), w.double())
        assert float((out[:, :, :o].double() - want).norm() / want.norm()) < 2.5e-7
        assert float((out[:, :, o:] - 7.0).abs().max()) == 0.0


@pytest.mark.parametrize("n", (3, 40, 200))
def test_deep_product_of_values_that_are_not_finite(native, n):
    """Infinities, NaN and numbers that round to infinity in 16 bits give what one chain of multiply-adds gives, and
    reach no other row or column."""
    gen = torch.Generator().manual_seed(n)
    k, o = 512, 150
    x, w = torch.randn((n, k), generator=gen), torch.randn((o, k), generator=gen)
    clean = torch.empty((n, o), device=DEV)
    native.gemm_simt(x.to(DEV), w.to(DEV), clean)
    x[0, 5], x[1, 9], x[2, 1], w[7, 3], w[9, 2] = float("inf"), float("nan"), 3.4e38, float("-inf"), -3.4e38
    got = torch.empty((n, o), device=DEV)
    native.gemm_simt(x.to(DEV), w.to(DEV), got)
    want = x.double() @ w.double().t()                       # 64 bits hold what overflows 32
    got, clean = got.cpu(), clean.cpu()
    keep = [c for c in range(o) if c not in (7, 9)]
    assert torch.equal(got[3:, keep], clean[3:, keep])
    assert bool(got[1].isnan().all()) and bool((got[0, keep] == want[0, keep]).all())
    big = want[2, keep].abs() > 3.5e38
    assert bool(torch.isinf(got[2, keep][big]).all()) and bool((got[3:, 7] == want[3:, 7]).all())
    sound = want[2, keep].abs() < 3.3e38
    assert float((got[2, keep][sound].double() / want[2, keep][sound] - 1).abs().max()) < 1e-5


@pytest.mark.parametrize("n, tiles, k, cuts", ((128, 15, 1024, 8), (128, 16, 1024, 4), (64, 16, 3072, 4), (32, 33, 512, 4), (32, 34, 512, 1), (4, 16, 1024, 8)))
def test_products_are_cut_into_clusters_that_run_at_once(native, n, tiles, k, cuts):
    """15 clusters of eight blocks and 33 of four fit the chip where a block has an SM; the bits of any cut are the same."""
    assert native.lib().fe_gemm_split_cuts(n, tiles * 128, k, 1) == cuts
    gen = torch.Generator().manual_seed(n + k)
    x, w = torch.randn((n, k), generator=gen).to(DEV), torch.randn((tiles * 128, k), generator=gen).to(DEV)
    got, alone = torch.empty((n, tiles * 128), device=DEV), torch.empty((n, 128), device=DEV)
    native.gemm_simt(x, w, got)
    native.gemm_simt(x, w[-128:].contiguous(), alone)
    assert torch.equal(got[:, -128:], alone)


@pytest.mark.parametrize("n, o, k", ((3, 40100, 256), (20, 20100, 320), (50, 20100, 260), (300, 4210, 448)))
def test_values_that_are_not_finite_in_tiles_of_one_block(native, n, o, k):
    """The same in each tile size where one block takes all of k and writes its outputs itself: single lanes take the chain
    between two accesses of the whole warp to tensor memory, and lanes past the last column leave early."""
    assert native.lib().fe_gemm_split_cuts(n, o, k, 1) == 1
    gen = torch.Generator().manual_seed(n + o)
    x, w = torch.randn((n, k), generator=gen).to(DEV), torch.randn((o, k), generator=gen).to(DEV)
    clean = torch.empty((n, o), device=DEV)
    native.gemm_simt(x, w, clean)
    rows, columns = {0: float("inf"), n // 2: float("nan"), n - 1: float("-inf")}, {1: float("inf"), 70: float("nan"), o - 2: float("-inf")}
    for row, value in rows.items():
        x[row, (7 * row) % k] = value
    for column, value in columns.items():
        w[column, (5 * column + 1) % k] = value
    got = torch.full((n, o), 7.0, device=DEV)
    native.gemm_simt(x, w, got)
    want = x.double() @ w.double().t()
    keep = torch.ones((n, o), dtype=torch.bool, device=DEV)
    keep[list(rows)] = False
    keep[:, list(columns)] = False
    assert torch.equal(got[keep], clean[keep])
    assert torch.equal(got[~keep].isnan(), want[~keep].isnan())
    infinite = ~keep & want.isinf()
    assert bool(infinite.any()) and torch.equal(got[infinite].double(), want[infinite])


@pytest.mark.parametrize("n, o, k", ((4, 32100, 256), (16, 300, 1028), (40, 700, 512), (200, 300, 448), (300, 4224, 256)))
def test_products_without_a_finite_sum_are_chains(native, n, o, k):
    """NaN in every row, NaN in every column, and an infinity in every row: every output is taken again, as the chain of
    multiply-adds that kernels without tensor cores take (the same rows off 16 bytes go there), bit for bit."""
    gen = torch.Generator().manual_seed(n + k)
    x, w = torch.randn((n, k), generator=gen).to(DEV), torch.randn((o, k), generator=gen).to(DEV)
    for loud in ("rows", "columns", "infinite"):
        a, b = x.clone(), w.clone()
        if loud == "rows":
            a[:, 3] = float("nan")
        elif loud == "columns":
            b[:, k - 2] = float("nan")
        else:
            a[:, 9], b[:, 9] = float("inf"), b[:, 9].abs() + 0.1
            a[0, 9] = float("-inf")
        got, chain = torch.empty((n, o), device=DEV), torch.empty((n, o), device=DEV)
        native.gemm_simt(a, b, got)
        off = torch.empty(n * k + 1, device=DEV)[1:].view(n, k).copy_(a)           # rows that start off 16 bytes
        assert off.data_ptr() % 16 != 0
        native.gemm_simt(off, b, chain)
        assert torch.equal(got.nan_to_num(nan=7.0), chain.nan_to_num(nan=7.0)), loud
        assert not bool(got.isfinite().any())


@pytest.mark.parametrize("n, o, k", ((4, 2048, 1024), (40, 3000, 512), (300, 4224, 1024)))
def test_operands_that_the_kernel_before_writes(native, n, o, k):
    """Both operands are products of the kernels right before, which let the next one start early: the same bits as with the
    device idle in between.  New operands in every turn, so that whoever reads too soon finds those of the turn before."""
    gen = torch.Generator(device=DEV).manual_seed(n)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV)  # noqa: E731
    x, w, got, want = torch.empty((n, k), device=DEV), torch.empty((o, k), device=DEV), torch.empty((n, o), device=DEV), torch.empty((n, o), device=DEV)

    def chain(left, right, mix, out, pause):
        torch.cuda.synchronize()
        for a, b in ((left, x), (right, w)):
            native.gemm_simt(a, mix, b)
            pause()
        native.gemm_simt(x, w, out)
        torch.cuda.synchronize()

    for _ in range(6):
        left, right, mix = rand(n, 256), rand(o, 256), rand(k, 256) / 16
        chain(left, right, mix, got, lambda: None)
        chain(rand(n, 256), rand(o, 256), mix, want, torch.cuda.synchronize)
        chain(left, right, mix, want, torch.cuda.synchronize)
        assert torch.equal(got, want)


@pytest.mark.parametrize("exponent", (-100, -111, -118, -126, -130))
@pytest.mark.parametrize("n, o, k", ((3, 300, 1024), (40, 150, 256), (300, 4224, 448)))
def test_deep_product_of_small_numbers(native, n, o, k, exponent):
    """Rows of either operand whose numbers lie where bfloat16 ends (2^-133): no further from 64 bits than a chain of
    multiply-adds may be, (k + 1) 2^-24 of the sum of magnitudes and half a step of 2^-149 an addition.  Zeros stay zeros,
    and the other rows and columns keep their bits."""
    gen = torch.Generator().manual_seed(n - exponent)
    x, w = torch.randn((n, k), generator=gen).to(DEV), torch.randn((o, k), generator=gen).to(DEV)
    clean, got = torch.empty((n, o), device=DEV), torch.empty((n, o), device=DEV)
    native.gemm_simt(x, w, clean)
    rows, columns = [0, n // 2], [5, o - 1]
    x[rows], w[columns] = (x[rows].double() * 2.0**exponent).float(), (w[columns].double() * 2.0**exponent).float()
    x[n - 1], w[o // 2] = 0.0, 0.0
    native.gemm_simt(x, w, got)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert bool(((got.double() - want).abs() <= size * (k + 1) * 2.0**-24 + k * 2.0**-149).all())
    off = (got.double() - want)[rows][:, 6 : o // 2].norm() / want[rows][:, 6 : o // 2].norm()
    assert float(off) < (2e-6 if exponent > -120 else 1e-5)
    assert float(got[n - 1].abs().max()) == float(got[:, o // 2].abs().max()) == 0.0
    keep = torch.ones((n, o), dtype=torch.bool, device=DEV)
    keep[rows + [n - 1]], keep[:, columns + [o // 2]] = False, False
    assert torch.equal(got[keep], clean[keep])


# -- the largest logits alone ------------------------------------------------------------------------
def drawn_among(row, temperature, top_k, top_p, min_p, u):
    """(index, distance of the target from the nearest boundary of the running sum, over the sum) in 64 bits: of equal
    logits the first ones are kept by top-k and all of them by top-p."""
    x = ((row - row.max()) * (1.0 / torch.tensor(temperature))).double()
    order = torch.argsort(-x, stable=True)
    keep = torch.zeros(len(x), dtype=torch.bool)
    keep[order[:top_k]] = True
    weights = torch.where(keep, torch.exp(x), 0.0)
    if top_p < 1.0:
        values, inverse = torch.unique(x, return_inverse=True)
        mass = torch.zeros(len(values), dtype=torch.float64).index_add_(0, inverse, weights)
        above = mass.flip(0).cumsum(0).flip(0) - mass
        weights = torch.where(above[inverse] <= top_p * weights.sum(), weights, 0.0)
    weights = torch.where(torch.exp(x) < min_p, 0.0, weights)
    running = weights.cumsum(0)
    target = u * running[-1]
    index = min(int(torch.searchsorted(running, target, right=True)), int(weights.nonzero()[-1]))
    return index, float((running - target).abs().min() / running[-1])


@pytest.mark.parametrize("vocab", (300, 4097, 70001))
@pytest.mark.parametrize("shape", ("normal", "ties", "sorted", "masked"))
def test_sampling_among_the_largest(native, vocab, shape):
    """Top-k at the ends of what is decided among the collected elements (512) and past it, with more elements above the
    bound than there is room for (equal logits) and the largest all in one block's slice: the draw of 64-bit arithmetic.
    Only a target within rounding (1e-5 of the sum) of a boundary of the running sum may differ."""
    gen = torch.Generator().manual_seed(vocab)
    logits = torch.randn((12, vocab), generator=gen) * 2.0
    if shape == "ties":
        logits = logits.round()
    if shape == "sorted":
        logits = logits.sort(dim=1, descending=True).values.contiguous()
    if shape == "masked":
        logits[torch.rand(logits.shape, generator=gen) < 0.99] = float("-inf")
        logits[:, 0] = 1.0
    top_k = [1, 2, 50, 200, 511, 512, 513, 20, 20, 50, 50, 1024]
    top_p = [1.0, 1.0, 0.95, 0.9, 1.0, 0.99, 0.9, 1.0, 0.5, 1e-6, 1.0, 0.9]
    min_p = [0.0] * 7 + [0.05, 0.0, 0.0, 0.3, 0.0]
    asked = [(0.8, min(k, vocab), p, m) for k, p, m in zip(top_k, top_p, min_p)]
    wishes = b"".join(struct.pack("=3fi2Q", t, p, m, k, 11 + r, 2**40 + r) for r, (t, k, p, m) in enumerate(asked))
    out, status = torch.empty(12, dtype=torch.int32, device=DEV), status_word()
    native.sample_rows(logits.to(DEV), out, status, wishes)
    assert int(status.item()) == 0
    for r, got in enumerate(out.tolist()):
        want, gap = drawn_among(logits[r], *asked[r], twin_uniform(11 + r, 2**40 + r))
        assert got == want or gap < 1e-5, (r, got, want, gap)


@pytest.mark.parametrize("temperature", (1e39, 3.4e38, 1e-50))
def test_temperatures_past_32_bits(native, temperature):
    """Finite temperatures that 32 bits hold as infinity or zero draw the same by the rows of a launch (up to 64) and by
    arrays."""
    from forge_engine_b200.sampling.params import SamplingParams
    from forge_engine_b200.sampling.sampler import Sampler

    logits = torch.randn((65, 5000), generator=torch.Generator().manual_seed(4)).to(DEV)
    params = [SamplingParams(temperature=temperature, top_k=50.0 if r % 2 else None, top_p=0.9) for r in range(65)]
    status = status_word()
    sampler = Sampler(DEV, status)
    seeds, counters = list(range(65)), [3] * 65
    by_arrays = sampler.sample(logits, params, seeds, counters)
    by_rows = [sampler.sample(logits[a:b].contiguous(), params[a:b], seeds[a:b], counters[a:b]) for a, b in ((0, 1), (1, 65))]
    assert int(status.item()) == 0 and torch.equal(torch.cat(by_rows), by_arrays)
