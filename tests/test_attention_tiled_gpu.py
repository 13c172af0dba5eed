"""The general attention kernel's tiles: runs of tokens of one request, single tokens between them, the edges of tiles and of
splits, every option, and rows that must not see what their neighbours see."""
import pytest
import torch

import fake_ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _batch(seed, lens, starts, G, hd, ps, dtype, pad=0):
    """Portions ``lens`` after ``starts`` tokens each, then ``pad`` padding rows; pages in a shuffled order."""
    g = torch.Generator().manual_seed(seed)
    total = [n + s for n, s in zip(lens, starts)]
    blocks = [-(-n // ps) for n in total] + [1] * pad
    perm = torch.randperm(sum(blocks), generator=g).tolist()
    table = torch.zeros(len(blocks), max(blocks), dtype=torch.int32)
    at = 0
    for s, b in enumerate(blocks):
        table[s, :b] = torch.tensor(perm[at:at + b], dtype=torch.int32)
        at += b
    pos = torch.cat([torch.arange(s, s + n) for n, s in zip(lens, starts)] + [torch.tensor([-1])] * pad).to(torch.int32)
    seg = torch.repeat_interleave(torch.arange(len(blocks)), torch.tensor(lens + [1] * pad)).to(torch.int32)
    k, v = (torch.randn(sum(blocks), G, ps, hd, generator=g).to(dtype) for _ in range(2))
    return g, k, v, seg, pos, table


def _check(dtype, H, G, hd, ps, lens, starts, splits=1, pad=0, window=None, seed=0, part_keys=0, off=0, **extra):
    from pico_vllm_b200 import ops
    g, k, v, seg, pos, table = _batch(seed, lens, starts, G, hd, ps, dtype, pad)
    T = seg.shape[0]
    q = torch.randn(T, H * hd + 32, generator=g).to(dtype)[:, :H * hd]
    for name in ("slopes", "sinks", "rates"):
        if extra.get(name):
            extra[name] = torch.rand(H, generator=g) * (2.0 if name == "sinks" else 0.2)
    want = torch.zeros(T, H * hd)
    scale = hd ** -0.5
    fake_ops.paged_attention(q.float(), k.float(), v.float(), want, seg, pos, table, H, G, hd, ps, window, scale, **extra)
    d = lambda t: t.to(DEV) if torch.is_tensor(t) else t
    out = torch.full((T, H * hd), float("nan"), dtype=dtype, device=DEV)
    scratch = torch.full((max(1, ops.attention_scratch_floats(T, H, hd, splits)) + off,), float("nan"), device=DEV)[off:]
    ops.paged_attention(d(q), d(k), d(v), out, d(seg), d(pos), d(table), H, G, hd, ps, window, scale, splits, scratch, part_keys=part_keys,
                        **{n: d(t) for n, t in extra.items()})
    # float32: sums of up to some hundreds of terms of order 1; bfloat16: the result's own rounding, 2^-9, of values up to 4
    tol = dict(atol=2e-5, rtol=2e-5) if dtype == torch.float32 else dict(atol=1e-2, rtol=1e-2)
    assert torch.allclose(out.float().cpu(), want, **tol), float((out.float().cpu() - want).abs().max())


OPTIONS = [dict(), dict(window=37), dict(chunk=24), dict(softcap=5.0), dict(slopes=True), dict(slopes=True, rates=True),
           dict(sinks=True), dict(window=9, slopes=True, sinks=True)]


@pytest.mark.parametrize("i", range(len(OPTIONS)))
@pytest.mark.parametrize("splits", [1, 3])
def test_options_over_portions_and_single_tokens(i, splits):
    # portions that start and end inside tiles of keys and groups of tokens, singles between them, a padding row
    _check(torch.float32, 12, 2, 48, 4, [1, 33, 1, 1, 2, 17], [70, 0, 0, 129, 31, 8], splits, pad=1, seed=i, **OPTIONS[i])


@pytest.mark.parametrize("i", [0, 1, 6])
@pytest.mark.parametrize("splits,part_keys", [(4, 16), (4, 40), (3, 1), (2, 1000), (8, 17)])
def test_runs_in_as_many_parts_as_they_have_keys_for(splits, part_keys, i):
    # whole runs beside runs in parts; parts that the tiles of keys leave without any; a padding row
    _check(torch.float32, 12, 2, 48, 4, [1, 33, 1, 1, 2, 17], [70, 0, 0, 129, 31, 8], splits, pad=1, seed=i, part_keys=part_keys, **OPTIONS[i])


@pytest.mark.parametrize("splits,part_keys", [(3, 0), (4, 40)])
@pytest.mark.parametrize("lens,starts", [([1, 1], [70, 129]), ([1, 33, 2], [70, 0, 31])])
def test_scratch_may_begin_at_any_float(lens, starts, splits, part_keys):
    _check(torch.float32, 12, 2, 48, 4, lens, starts, splits, part_keys=part_keys, off=1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd", [(1, 1, 16), (8, 8, 128), (9, 3, 144), (40, 1, 256), (2, 1, 272), (12, 1, 640)])
def test_head_sizes_and_groups(dtype, H, G, hd):
    _check(dtype, H, G, hd, 16, [1, 19, 1, 9], [40, 0, 16, 3])


@pytest.mark.parametrize("hd,H,G", [(32, 32, 8), (160, 32, 8), (320, 10, 10)])
def test_many_rows_share_their_keys(hd, H, G):
    # enough full tiles for the form with 32 rows a block; runs of 1, of a whole group and one more
    _check(torch.float32, H, G, hd, 8, [1, 290, 8, 9, 15, 1], [3, 0, 5, 64, 1, 77], window=None if hd == 32 else 50)
    if H == G:
        _check(torch.float32, H, G, hd, 8, [970], [0], window=33)


@pytest.mark.parametrize("T", [40, 320])
def test_a_value_that_is_no_number_stays_with_the_rows_that_see_it(T):
    from pico_vllm_b200 import ops
    H, G, hd, ps = 32, 8, 32, 8
    g, k, v, seg, pos, table = _batch(5, [T], [0], G, hd, ps, torch.float32)
    bad = T - 3
    v[table[0, bad // ps], :, bad % ps] = float("inf")
    q = torch.randn(T, H * hd, generator=g)
    out = torch.zeros(T, H * hd, device=DEV)
    ops.paged_attention(q.to(DEV), k.to(DEV), v.to(DEV), out, seg.to(DEV), pos.to(DEV), table.to(DEV), H, G, hd, ps, None, 0.2)
    finite = torch.isfinite(out).all(1).cpu()
    assert finite[:bad].all() and not finite[bad:].any()


def test_as_many_key_heads_as_a_grid_has_rows():
    """33,000 key heads of 33 query heads each: two tiles of rows a token, more blocks than a grid has in its second dimension."""
    from pico_vllm_b200 import ops
    G, n, hd = 33000, 33, 16
    g = torch.Generator(device=DEV).manual_seed(1)
    q, k, v = (torch.randn(*s, generator=g, device=DEV) for s in ((1, G * n * hd), (1, G, 4, hd), (1, G, 4, hd)))
    at = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out = torch.zeros_like(q)
    ops.paged_attention(q, k, v, out, at([0]), at([2]), at([[0]]), G * n, G, hd, 4, None, 0.25)
    p = torch.softmax(torch.einsum("gnd,gkd->gnk", q.view(G, n, hd).double(), k[0, :, :3].double()) * 0.25, -1)
    want = torch.einsum("gnk,gkd->gnd", p, v[0, :, :3].double())
    assert float((out.view(G, n, hd) - want).abs().max()) <= 2e-5        # float32 sums of 16 products and of three values


@pytest.mark.parametrize("what", ["query", "key"])
@pytest.mark.parametrize("T,start,splits", [(1, 48, 1), (1, 48, 2), (1, 200, 1), (40, 0, 1), (40, 0, 3), (320, 0, 1)])
def test_a_score_that_is_no_number_makes_its_row_none(what, T, start, splits):
    """A query that is no number (none of its row's scores is one), or a key (one score of each row that sees it is none; with 49
    keys it is the only one a warp, or the second part, has): those rows of the output are no numbers, all others are."""
    from pico_vllm_b200 import ops
    H, G, hd, ps = 32, 8, 32, 8
    g, k, v, seg, pos, table = _batch(6, [T], [start], G, hd, ps, torch.float32)
    q = torch.randn(T, H * hd, generator=g)
    row = max(0, T - 3)
    if what == "query":
        q[row] = float("nan")
    else:
        k[table[0, (start + row) // ps], :, (start + row) % ps] = float("nan")
    out = torch.zeros(T, H * hd, device=DEV)
    scratch = torch.zeros(max(1, ops.attention_scratch_floats(T, H, hd, splits)), device=DEV)
    ops.paged_attention(q.to(DEV), k.to(DEV), v.to(DEV), out, seg.to(DEV), pos.to(DEV), table.to(DEV), H, G, hd, ps, None, 0.2, splits, scratch)
    want = torch.arange(T) == row if what == "query" else torch.arange(T) >= row
    assert torch.equal(out.isnan().all(1).cpu(), want) and torch.equal(out.isnan().any(1).cpu(), want)
