"""Causal attention over one cached latent per token.

Queries pass through a normalised latent of their own: c_q = rmsnorm(W_dq x), q = W_uq c_q,
every head [head_dim elements that are not rotated | rot_dim that are].  Keys and values are
expanded from a second latent: W_dkv x gives kv_rank + rot_dim numbers; the first kv_rank,
RMS-normalised, are the latent c, the last rot_dim, rotated, are a key part that all heads
share.  Head h's key is [W_uk,h c | shared part], its value W_uv,h c.  Only c and the shared
part are kept in the cache: one vector of kv_rank + rot_dim per token for all heads.

In decoding and short portions the expansion is never carried out.  Since q_h . (W_uk,h c) =
(W_uk,h^T q_h) . c, the step's queries are taken through W_uk,h^T once (kv_rank numbers per
head), attention then runs with one shared "kv head" whose key is the cached vector itself
and whose value is its first kv_rank elements, and the weighted sum of latents is expanded by
W_uv,h afterwards.  A step's cost does not depend on how many heads read the cache.

For a long prompt portion that is the dearer way: a query against a key then takes 2 kv_rank + rot_dim
multiply-adds per head instead of head_dim + rot_dim + v_head_dim.  There the portion's context is taken
out of its pages, expanded for all heads by one product (the shared part rides along through an identity
block) and read by the tcgen05 prefill kernel, keys and values padded to 128.

A layer with ``kv_from`` has no W_dkv and reads the cache of the layer named there.

``window``: a query sees its own and the window - 1 tokens before it, and the pages the window
has passed go back to the pool.  ``sink``: a learned number per head whose exponential joins
the softmax's denominator once, as a weight on no key and no value.
"""

from __future__ import annotations

import os

import torch

from ..cache.manager import CacheNeeds, PagedKVSpec
from ..config.specs import local_name
from ..ops import native
from .base import BuildContext, CacheView, Mixer, WeightInfo, build_part, register_part
from .linear import Linear, fused_rows


# Portions of more than EXPAND_FROM tokens (EXPAND_FROM_CHEAP where rank and rotated part are small) are expanded, in steps of more than EXPAND_STEP tokens.  Which
# rows of a step's expansion belong to whom depends on every entry's length, so such a step could not be
# replayed for another one: the line is the most tokens a replayed step has (engine/graphs.py).  1,500
# tokens after 500 (32 heads, 64 + 32 / 64, rank 256): the mixer takes 575 us in the absorbed
# form (464 of them attention), 196 to 204 expanded; 128 tokens are where a head's 128-row tile is full.
# Kernels of the mixer, absorbed / expanded, us, 129 tokens after 0, 2,000, 16,000 and 60,000 cached ones (32 heads,
# width 2,560): rank 512 (+ 64) 66 / 43, 338 / 103, 2227 / 512, 8177 / 1774; rank 256 (+ 32) 55 / 41, 195 / 93, 1163 / 470,
# 4214 / 1623; rank 64 41 / 39, 103 / 86, 527 / 447, 1863 / 1542; rank 32 39 / 37, 88 / 85, 426 / 434, 1488 / 1499; rank 16
# 39 / 39, 82 / 86, 388 / 438, 1348 / 1510.  The expansion's multiply-adds run several times as fast as those of the
# absorbed attention, so the context hardly moves the line; the rank does where a query against a key is cheap:
# up to 64 multiply-adds a head the line lies at 384 tokens (rank 16: 256 tokens after 4,000 131 / 144, 400 after
# 8,000 288 / 261).
EXPAND_FROM, EXPAND_FROM_CHEAP, EXPAND_CHEAP = 128, 384, 64
EXPAND_STEP = max(512, int(os.environ.get("FORGE_ENGINE_GRAPH_TOKENS", "512")))
# A step that holds other entries too runs both forms, each on the rows of its own entries, and the host launches
# a layer's mixer almost twice (about 100 us more): there the portions are expanded only where the absorbed
# attention over them takes longer than that.  Its operations, two per multiply-add, at about 1.4e14 a second.
# Steps of 6 layers of width 2,560, 32 heads, us a layer, absorbed / both: rank 256, 8 decoding and 510 tokens
# (4.5e9) 433 / 468, 8 and 700 (8.5e9) 486 / 501, 48 and 1,000 (1.7e10) 675 / 598, 100 and 500 after 2,000 (3.9e10)
# 927 / 726; rank 512, 100 and 430 (6.4e9) 767 / 794, 16 and twice 257 (2.2e10) 566 / 496; width 1,024, 16
# heads, 8 and 700 (4.3e9) 364 / 453, 100 and 500 after 2,000 (2.0e10) 654 / 682.
EXPAND_BESIDE = 2e10
# Keys and values of all heads take 512 bytes a head and token of context, up to this many at a time: heads beyond
# go through the same buffer after them (one head at least, which is about what the cached latents take).
EXPAND_BYTES = 1 << 30


class _Rows:
    """Entries of a step that take the same form, as a batch of their own: which rows of the step are theirs (None:
    all, a slice, or an index), and the integers of that batch."""

    def __init__(self, batch) -> None:
        """All entries of the step."""
        self.tokens = self.of_table = None
        self.n_tokens, self.n_entries, self.max_new = batch.n_tokens, batch.n_entries, batch.max_new
        self.cu_tokens, self.starts, self.positions, self.token_entry = batch.cu_tokens, batch.starts, batch.positions, batch.token_entry

    def pick(self, batch, spans: tuple, chosen: list, flat: list) -> list:
        """Keep the entries ``chosen`` (in order) of the step's ``spans`` ((cached, new) each).  What the device has
        to be sent is appended to ``flat``; answers where it lies there, for ``sent``."""
        first, cu, ends = [], [0], 0
        for _, count in spans:
            first.append(ends)
            ends += count
        for e in chosen:
            cu.append(cu[-1] + spans[e][1])
        self.n_tokens, self.n_entries, self.max_new = cu[-1], len(chosen), max(spans[e][1] for e in chosen)
        lists = [cu]
        if chosen[-1] - chosen[0] + 1 == len(chosen):             # neighbours: their rows are a range
            self.tokens, self.of_table = slice(first[chosen[0]], first[chosen[0]] + cu[-1]), slice(chosen[0], chosen[-1] + 1)
        else:
            lists += [[t for e in chosen for t in range(first[e], first[e] + spans[e][1])], chosen,
                      [i for i, e in enumerate(chosen) for _ in range(spans[e][1])]]
        return [_place(flat, values) for values in lists]

    def sent(self, batch, flat: torch.Tensor, places: list) -> None:
        lists = [flat[a:b] for a, b in places]
        self.cu_tokens = lists[0]
        if len(lists) > 1:
            self.tokens, self.of_table, self.token_entry = lists[1].long(), lists[2], lists[3]
        else:
            self.token_entry = batch.token_entry[self.tokens] - self.of_table.start
        self.starts, self.positions = self._take(batch.starts, self.of_table), self._take(batch.positions, self.tokens)

    @staticmethod
    def _take(x: torch.Tensor, which) -> torch.Tensor:
        return x if which is None else x[which] if isinstance(which, slice) else x.index_select(0, which)

    def of(self, x: torch.Tensor) -> torch.Tensor:
        """Their rows of ``x`` [tokens, ...]."""
        return self._take(x, self.tokens)

    def table(self, table: torch.Tensor) -> torch.Tensor:
        """Their rows of a block table [entries, pages]."""
        return self._take(table, self.of_table)

    def room(self, x: torch.Tensor) -> torch.Tensor:
        """Where their rows of ``x`` are worked out; ``put`` then stores them."""
        return x.new_empty((self.n_tokens, *x.shape[1:])) if isinstance(self.tokens, torch.Tensor) else self.of(x)

    def put(self, x: torch.Tensor, room: torch.Tensor) -> None:
        if isinstance(self.tokens, torch.Tensor):
            x.index_copy_(0, self.tokens, room)


def _place(flat: list, values: list) -> tuple:
    """Append ``values`` to ``flat``, where the next ones begin on a 16-byte boundary again; where they lie."""
    begin = len(flat)
    flat += values
    flat += [0] * (-len(flat) % 4)
    return begin, begin + len(values)


class LatentAttention(Mixer):
    graph_safe = True

    def __init__(self, spec, weights: dict, ctx: BuildContext) -> None:
        self.spec, self.ctx = spec, ctx
        self.h, self.d, self.r, self.dv = spec.num_heads, spec.head_dim, spec.rot_dim, spec.v_head_dim
        self.q_rank, self.kv_rank = spec.q_rank, spec.kv_rank
        self.own = spec.kv_from is None
        name = lambda canonical: local_name(spec, canonical)  # noqa: E731
        # one projection for both latents of a layer that has both
        if self.own:
            down = fused_rows(weights, [name("dq"), name("dkv")], [self.q_rank, self.kv_rank + self.r])
        else:
            down = weights[name("dq")]
        self.down = Linear(down, status=ctx.status)
        self.q_norm = weights[name("dq.norm")].float().contiguous()
        self.kv_norm = weights[name("dkv.norm")].float().contiguous() if self.own else None
        self.up_q = Linear(weights[name("uq")], status=ctx.status)
        uk = weights[name("uk")]
        # [head, kv_rank, head_dim]: the transpose of every head's key expansion
        self.uk_t = uk.view(self.h, self.d, self.kv_rank).transpose(1, 2).contiguous()
        del uk
        self.uv = weights[name("uv")].contiguous().view(self.h, self.dv, self.kv_rank)
        self.o_proj = Linear(weights[name("o")], status=ctx.status)
        self.position = build_part(spec.position, {}, ctx)
        self.rot_dims = self.position.rotary()[1]
        self.window = getattr(spec, "window", None) or None
        self.sinks = None
        if getattr(spec, "sink", False):
            self.sinks = weights[name("sink")].to(device=ctx.device, dtype=torch.float32).contiguous()
        self.expanded = None
        wide = native.EXPANDED_DIM
        # the expanded form: both sizes fit the kernel's head, outputs are stored 32 at a time
        if (self.d + self.r <= wide and self.dv <= wide and self.dv % 32 == 0 and spec.scale > 0 and (self.kv_rank + self.r) % 8 == 0
                and native.general_mma_takes(ctx.dtype, self.kv_rank + self.r, self.kv_rank)
                and all(t.dtype == torch.bfloat16 for t in (self.up_q.weight, self.uk_t, self.uv))):
            # [heads x 2 x 128, kv_rank + rot_dim]: a head's key rows (expansion, then the identity on the
            # shared part), then its value rows; rows of zeros pad both to 128
            both = torch.zeros((self.h, 2, wide, self.kv_rank + self.r), dtype=torch.bfloat16, device=self.uv.device)
            both[:, 0, : self.d, : self.kv_rank] = self.uk_t.transpose(1, 2)
            both[:, 0, self.d : self.d + self.r, self.kv_rank :] = torch.eye(self.r, dtype=torch.bfloat16, device=self.uv.device)
            both[:, 1, : self.dv, : self.kv_rank] = self.uv
            queries = torch.zeros((self.h, wide, self.q_rank), dtype=torch.bfloat16, device=self.uv.device)
            queries[:, : self.d + self.r] = self.up_q.weight.view(self.h, self.d + self.r, self.q_rank)
            self.expanded = (both.view(2 * self.h * wide, -1).t(), Linear(queries.view(self.h * wide, -1), status=ctx.status))
        self.expand_from = EXPAND_FROM_CHEAP if 2 * self.kv_rank + self.r <= EXPAND_CHEAP else EXPAND_FROM
        # layers share a step's plan only where all of them can carry it out
        self.plan_key = ("latent_attention", self.h, self.kv_rank, self.r, self.window, self.expanded is not None)

    def plan_step(self, entries: list, page_size: int, plans: dict) -> None:
        """The host's decision for a step of ``entries`` ((slot, cached, new) each; layers of one
        geometry share it): how many blocks share the keys of one tile of query rows (None: no entry
        takes the absorbed form), and (cached, new) of the entries if some are expanded."""
        if self.plan_key not in plans:
            short, expanded = list(entries), None
            if self.expanded is not None and sum(count for _, _, count in entries) > EXPAND_STEP:
                long = [e for e in entries if e[2] > self.expand_from]
                if long and (len(long) == len(entries) or 2 * self.h * (2 * self.kv_rank + self.r) * self._pairs(long) > EXPAND_BESIDE):
                    short = [e for e in entries if e[2] <= self.expand_from]
                    expanded = tuple((start, count) for _, start, count in entries)
            splits = 1 if short else None
            if short and native.general_mma_takes(self.ctx.dtype, self.kv_rank + self.r, self.kv_rank):
                splits = native.general_splits(short, self.h, 1, self.window)
            plans[self.plan_key] = (splits, expanded)

    def _heads_at_once(self, rows: int) -> int:
        """Heads whose keys and values of ``rows`` tokens are held at a time, in stretches that are about equal."""
        most = max(1, EXPAND_BYTES // (rows * 2 * native.EXPANDED_DIM * 2))
        return -(-self.h // -(-self.h // most))

    def _pairs(self, entries: list) -> int:
        """How many (query, key) pairs a head works on for the new tokens of ``entries``."""
        total = 0
        for _, start, count in entries:
            whole = max(0, min(count, (self.window or start + count) - start))      # queries that see every earlier token
            total += whole * start + whole * (whole + 1) // 2 + (count - whole) * (self.window or 0)
        return total

    def _forms(self, spans: tuple, batch) -> tuple:
        """The step's rows by the form they take, worked out once a step: (those that take the absorbed one or
        None, those that are expanded, where the latter's contexts lie in the expansion).  That is, int32 on the
        device, (entry, first position, first position needed) per stretch of 128 rows, and [expanded entries, L]
        the stretch of positions 128 j .. (-1: none)."""
        key = (self.plan_key, "forms")
        if key in batch.shared:
            return batch.shared[key]
        size = native.PREFILL_TC5_KEYS
        short, long, where, tables = [], [], [], []
        for entry, (start, count) in enumerate(spans):
            if count <= self.expand_from:
                short.append(entry)
                continue
            long.append(entry)
            needed = max(0, start - self.window + 1) if self.window else 0
            first, last = needed // size, -(-(start + count) // size)
            stretch = len(where) // 3
            tables.append([-1] * first + list(range(stretch, stretch + last - first)))
            for j in range(first, last):
                where += (entry, size * j, needed)
        width = max(map(len, tables))
        flat: list = []
        at = _place(flat, where)
        of_entry = _place(flat, [v for row in tables for v in row + [-1] * (width - len(row))])
        parts = [(None, None), (_Rows(batch), None)]
        if short:
            parts = [(rows, rows.pick(batch, spans, chosen, flat)) for rows, chosen in ((_Rows(batch), short), (_Rows(batch), long))]
        device = torch.tensor(flat, dtype=torch.int32).pin_memory().to(self.ctx.device, non_blocking=True)
        for rows, places in parts:
            if places is not None:
                rows.sent(batch, device, places)
        batch.shared[key] = parts[0][0], parts[1][0], (device[at[0] : at[1]].view(-1, 3), device[of_entry[0] : of_entry[1]].view(len(long), width))
        return batch.shared[key]

    def _attend_expanded(self, c_q, rows: _Rows, stretches: tuple, batch, latent_cache, table, angles, heads) -> None:
        """The rows ``rows`` of ``heads`` [N, heads, v_head_dim]."""
        h, d, r, dv, wide = self.h, self.d, self.r, self.dv, native.EXPANDED_DIM
        expand, up_q = self.expanded
        with self.ctx.section("mixer.qkv_rope_cache"):
            q = up_q(rows.of(c_q))
            native.qkv_prepare(
                q=q[:, d:], q_heads=h, q_dim=r, q_head_stride=wide, q_rot_off=0,
                q_out=q, q_out_strides=(h * wide, wide), q_out_offset=d,
                table=rows.of(angles), rot_dims=self.rot_dims, interleaved=self.position.interleaved,
                positions=rows.positions, token_entry=rows.token_entry, status=self.ctx.status,
            )
            where, of_entry = stretches
            latents = torch.empty((where.shape[0] * native.PREFILL_TC5_KEYS, self.kv_rank + r), dtype=torch.bfloat16, device=c_q.device)
            native.latent_rows(latent_cache, table, where, batch.ctx_lens, latents, self.ctx.status)
        room = rows.room(heads)
        out, most = room.view(rows.n_tokens, h * dv), self._heads_at_once(latents.shape[0])
        if most == h:
            turns = [(h, expand, q, out, self.sinks)]
        else:
            turns = [(min(h, a + most) - a, expand[:, 2 * wide * a : 2 * wide * (a + most)], q[:, wide * a : wide * (a + most)],
                      out[:, dv * a : dv * (a + most)], None if self.sinks is None else self.sinks[a : a + most]) for a in range(0, h, most)]
        for n_heads, weight, queries, into, sinks in turns:
            with self.ctx.section("mixer.qkv_rope_cache"):
                kv = torch.mm(latents, weight)
            with self.ctx.section("mixer.attention"):
                native.attention_prefill_expanded(queries, kv, into, of_entry, rows.cu_tokens, rows.starts, rows.n_entries, rows.max_new,
                                                  n_heads, dv, self.window, self.spec.scale, sinks, self.ctx.status)
            del kv
        rows.put(heads, room)

    @classmethod
    def weight_shapes(cls, spec) -> dict:
        name = lambda canonical: local_name(spec, canonical)  # noqa: E731
        h, w = spec.num_heads, spec.hidden_size
        shapes = {
            name("dq"): WeightInfo((spec.q_rank, w)),
            name("dq.norm"): WeightInfo((spec.q_rank,), "norm"),
            name("uq"): WeightInfo((h * (spec.head_dim + spec.rot_dim), spec.q_rank)),
        }
        if spec.kv_from is None:
            shapes[name("dkv")] = WeightInfo((spec.kv_rank + spec.rot_dim, w))
            shapes[name("dkv.norm")] = WeightInfo((spec.kv_rank,), "norm")
        shapes[name("uk")] = WeightInfo((h * spec.head_dim, spec.kv_rank))
        shapes[name("uv")] = WeightInfo((h * spec.v_head_dim, spec.kv_rank))
        shapes[name("o")] = WeightInfo((w, h * spec.v_head_dim))
        if getattr(spec, "sink", False):
            shapes[name("sink")] = WeightInfo((h,), "bias")
        return shapes

    def cache_needs(self) -> CacheNeeds:
        return CacheNeeds(kv=PagedKVSpec(1, self.kv_rank + self.r, self.window, 0))

    def forward(self, x, batch, cache: CacheView):
        out = self.attend(x, batch, cache)
        with self.ctx.section("mixer.o_proj"):
            return self.o_proj(out)

    def _per_head(self, x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> None:
        """out[n, h] = x[n, h] @ w[h].T for x [N, heads, k], w [heads, o, k], out [N, heads, o]
        (x and out may be strided).  The 32-bit engine uses the 32-bit kernels; bfloat16
        the library's batched product, as the large projections do."""
        if x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[0] > native.TC5_MAX_ROWS:
            out.copy_(torch.bmm(x.transpose(0, 1), w.transpose(1, 2)).transpose(0, 1))
        else:
            native.gemm_simt_batched(x, w, out, status=self.ctx.status)

    def attend(self, x, batch, cache: CacheView):
        n, h, d, r, dv, rank = x.shape[0], self.h, self.d, self.r, self.dv, self.kv_rank
        latent_cache = cache.kv[0]
        table = batch.group_tables[cache.group]
        dtype = latent_cache.dtype
        with self.ctx.section("mixer.qkv_rope_cache"):
            down = self.down(x, out_dtype=torch.float32)
            angles = self.position.table(batch)
            c_q = torch.empty((n, self.q_rank), dtype=dtype, device=x.device)
            writes = self.own and cache.owns
            # the query latent is normalised; the key/value latent is normalised, its last
            # rot_dim elements are rotated instead, and the vector goes to its page
            native.qkv_prepare(
                q=down[:, : self.q_rank], q_heads=1, q_dim=self.q_rank,
                q_norm=(native.PREP_NORM_HEAD, self.q_rank, self.q_norm), q_rot_off=-1,
                q_out=c_q, q_out_strides=(self.q_rank, self.q_rank),
                k=down[:, self.q_rank:] if writes else None, k_heads=1, k_dim=rank + r,
                k_norm=(native.PREP_NORM_HEAD if writes else native.PREP_NORM_NONE, rank, self.kv_norm), k_rot_off=rank,
                eps=self.spec.norm_eps, table=angles, rot_dims=self.rot_dims, interleaved=self.position.interleaved,
                k_cache=latent_cache, block_table=table, positions=batch.positions, token_entry=batch.token_entry,
                status=self.ctx.status,
            )
        heads = torch.empty((n, h, dv), dtype=dtype, device=x.device)
        if self.plan_key not in batch.plans:
            self.plan_step(batch.entries, latent_cache.shape[2], batch.plans)
        splits, spans = batch.plans[self.plan_key]
        if spans is None:
            self._attend_absorbed(c_q, splits, _Rows(batch), latent_cache, table, angles, heads)
        else:
            short, long, stretches = self._forms(spans, batch)
            if short is not None:
                self._attend_absorbed(c_q, splits, short, latent_cache, table, angles, heads)
            self._attend_expanded(c_q, long, stretches, batch, latent_cache, table, angles, heads)
        return heads.view(n, h * dv)

    def _attend_absorbed(self, c_q, splits: int, rows: _Rows, latent_cache, table, angles, heads) -> None:
        """The rows ``rows`` of ``heads`` [N, heads, v_head_dim]."""
        n, h, d, r, rank = rows.n_tokens, self.h, self.d, self.r, self.kv_rank
        with self.ctx.section("mixer.qkv_rope_cache"):
            q = self.up_q(rows.of(c_q))                            # [n, heads * (d + r)]
            q_eff = torch.empty((n, h, rank + r), dtype=c_q.dtype, device=c_q.device)
            # rotated parts of the queries straight to where attention reads them
            native.qkv_prepare(
                q=q[:, d:], q_heads=h, q_dim=r, q_head_stride=d + r, q_rot_off=0,
                q_out=q_eff, q_out_strides=(h * (rank + r), rank + r), q_out_offset=rank,
                table=rows.of(angles), rot_dims=self.rot_dims, interleaved=self.position.interleaved,
                positions=rows.positions, token_entry=rows.token_entry, status=self.ctx.status,
            )
            # the other parts through the transposed key expansion
            self._per_head(q.view(n, h, d + r)[:, :, :d], self.uk_t, q_eff[:, :, :rank])
        mixed = torch.empty((n, h, rank), dtype=c_q.dtype, device=c_q.device)
        with self.ctx.section("mixer.attention"):
            native.attention_general(q_eff, (h * (rank + r), rank + r), latent_cache, rank + r, latent_cache, rank,
                                     mixed, (h * rank, rank), rows.table(table), rows.positions, rows.token_entry, h, None, self.window,
                                     self.spec.scale, self.ctx.status,
                                     entries=(rows.cu_tokens, rows.starts, rows.n_entries, rows.max_new),
                                     splits=splits, sinks=self.sinks)
        with self.ctx.section("mixer.expand"):
            out = rows.room(heads)
            self._per_head(mixed, self.uv, out)
            rows.put(heads, out)


register_part("latent_attention", LatentAttention, replace=True)
