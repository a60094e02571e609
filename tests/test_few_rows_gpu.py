"""Kernels whose time at a few rows is a chain of loads: the weights they ask for ahead, what lies beyond those, rows one by one and many."""

from __future__ import annotations

import pytest
import torch

from tests.test_kernels_gpu import PagedCase

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from research_2_b200.kernels import ops as o

    return o


# widths inside and beyond the 1,024 numbers kept in registers, and one that is no multiple of four; outputs around a CTA's eight
@pytest.mark.parametrize("width,n_out", [(768, 24), (1024, 7), (1600, 9), (770, 8), (36, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_small_linear_rows_do_not_depend_on_their_number(width, n_out, dtype):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(width)
    h = torch.randn(300, width, generator=gen, device=DEV).to(dtype)
    w, b = torch.randn(n_out, width, generator=gen, device=DEV), torch.randn(n_out, generator=gen, device=DEV)
    many = o.small_linear(h, w, b)
    for n in (1, 5, 256):
        assert torch.equal(o.small_linear(h[:n], w, b), many[:n])
    want = h.double() @ w.double().T + b.double()
    # a lane adds width / 128 terms to each of four sums, the warp's 32 meet in five steps: far fewer roundings than terms
    bound = (width / 128 + 16) * 2.0 ** -24 * (h.double().abs() @ w.double().abs().T + b.double().abs())
    assert ((many.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("rows,n_out", [(1, 8 * 65535 + 9), (8 * 65535 + 9, 1)])   # eight outputs or eight rows to a CTA: beyond a grid's second extent
def test_small_linear_of_any_number_of_rows_and_outputs(rows, n_out):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(rows)
    h, w = torch.randn(rows, 4, generator=gen, device=DEV), torch.randn(n_out, 4, generator=gen, device=DEV)
    got = o.small_linear(h, w)
    # four products and their sum: 2^-22 of the terms' sizes
    assert ((got.double() - h.double() @ w.double().T).abs() <= 2.0 ** -22 * (h.abs().double() @ w.abs().double().T)).all()



@pytest.mark.parametrize("width", [768, 1600, 770])
def test_router_logits_beyond_what_is_asked_for_ahead(width):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(width)
    h = torch.randn(9, width, generator=gen, device=DEV).bfloat16()
    w, b = torch.randn(20, width, generator=gen, device=DEV), torch.randn(20, generator=gen, device=DEV)
    dense, chosen, weight = o.route_top_k(h, w, b, 3)
    z = h.double() @ w.double().T + b.double()
    best = z.topk(3, dim=1)
    assert torch.equal(chosen.long(), best.indices)
    torch.testing.assert_close(weight.double(), torch.softmax(best.values, dim=1), atol=1e-4, rtol=1e-4)
    assert torch.equal(dense.gather(1, chosen.long()), weight)


# one, two and three pieces of K; rows around a warp's 16 and the tile's 64; gates read in pairs or one by one
@pytest.mark.parametrize("rows,k,n,offset", [(1, 64, 64, 0), (12, 128, 64, 0), (65, 136, 72, 0), (17, 128, 70, 1)])
@pytest.mark.parametrize("w_is_nk", [False, True])
def test_gated_products_per_head(rows, k, n, offset, w_is_nk):
    o, heads = ops(), 3
    gen = torch.Generator(device=DEV).manual_seed(rows + k)
    a = torch.randn(rows, heads * k, generator=gen, device=DEV).bfloat16()
    w = (torch.randn(heads * (n if w_is_nk else k), k if w_is_nk else n, generator=gen, device=DEV) * k ** -0.5).bfloat16()
    gate = torch.randn(rows, heads * n + offset, generator=gen, device=DEV).bfloat16()[:, offset:]
    out = torch.empty(rows, heads * n, dtype=torch.bfloat16, device=DEV)
    o.head_linear(a, k, w, w_is_nk, out, n, heads, k, n, gate=gate)
    wide = w.double().view(heads, -1, w.shape[1])
    want = torch.einsum("thk,hkn->thn", a.double().view(rows, heads, k), wide.transpose(1, 2) if w_is_nk else wide).reshape(rows, -1)
    want = want * torch.sigmoid(gate.double())
    torch.testing.assert_close(out.double(), want, atol=2.0 ** -8, rtol=2.0 ** -8)


# slices that are a cluster (up to eight) and more of them than that; contexts from one key to several tiles a warp
@pytest.mark.parametrize("max_context", [129, 260, 1024, 1030, 4096])
@pytest.mark.parametrize("window", [0, 40])
def test_slices_of_decode_attention_meet_in_their_cluster(max_context, window):
    case = PagedCase([(c, 1) for c in (0, 31, 128, 500, 1000)], 4, 2, 64, 16, torch.bfloat16, seed=max_context)
    got = case.run_fused(0.125, window, max_context).float().cpu()
    torch.testing.assert_close(got, case.plain(0.125, window), atol=2e-2, rtol=2e-2)
    one = PagedCase([(c, 1) for c in (0, 31, 128, 500, 1000)], 4, 2, 64, 16, torch.bfloat16, seed=max_context).run_fused(0.125, window, 100).float().cpu()
    # the same rounding of every weight to bfloat16 against another maximum, and the output's own: two roundings of 2^-9
    torch.testing.assert_close(got, one, atol=2.0 ** -7, rtol=2.0 ** -7)


# groups inside and beyond the columns that a thread keeps: four of a warp's 32 lanes, four of a CTA's 256 threads
@pytest.mark.parametrize("rows,groups,size", [(1, 3, 1), (5, 2, 64), (4, 3, 128), (3, 2, 130), (2, 1, 1024), (2, 2, 1030)])
@pytest.mark.parametrize("order", [True, False, "silu_after"])
def test_gated_norms_inside_and_beyond_what_is_kept(rows, groups, size, order):
    o, eps = ops(), 1e-5
    gen = torch.Generator(device=DEV).manual_seed(size)
    y = torch.randn(rows, groups * size, generator=gen, device=DEV)
    gate, w = torch.randn(rows, groups * size, generator=gen, device=DEV).bfloat16(), torch.randn(groups * size, generator=gen, device=DEV)
    got = o.group_norm_gated(y, gate, w, groups, eps, order, torch.bfloat16)
    z, v = gate.double(), y.double()
    if order is True:
        v = v * torch.nn.functional.silu(z)
    v = v.view(rows, groups, size)
    v = (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps)).view(rows, -1) * w.double()
    if order is not True:
        v = v * (torch.nn.functional.silu(z) if order == "silu_after" else torch.sigmoid(z))
    torch.testing.assert_close(got.double(), v, rtol=2.0 ** -8, atol=1e-6)   # one rounding to bfloat16, 2^-9, and float sums before it


def made_just_before(rows, cols, consumer, dtype=torch.float32, size=1.0):
    """consumer(w) right behind the launch that writes w [rows, cols] (a long one), and again once w has settled: the same bits."""
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(rows + cols)
    a, b = (torch.randn(*s, generator=gen, device=DEV) for s in ((rows, 4096), (cols, 4096)))
    for turn in range(10):
        w = torch.full((rows, cols), float(turn), dtype=dtype, device=DEV)
        if dtype == torch.bfloat16:
            o.linear((a * (size / 64)).bfloat16(), b.bfloat16(), None, w_is_nk=True, out=w)
        else:
            o.linear(a * (size / 64), b, None, w_is_nk=True, out=w)
        soon = consumer(w)
        torch.cuda.synchronize()
        late = consumer(w)
        for x, y in zip(soon if isinstance(soon, tuple) else (soon,), late if isinstance(late, tuple) else (late,)):
            assert torch.equal(x, y)


def test_operands_that_the_launch_just_before_writes():
    """Without the word that its weights are fixed, a kernel reads them only after the launch before it."""
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(3)
    h = torch.randn(4, 768, generator=gen, device=DEV)
    made_just_before(768, 640, lambda w: o.linear(h, w))
    made_just_before(640, 768, lambda w: o.linear(h, w, w_is_nk=True))
    made_just_before(24, 768, lambda w: o.small_linear(h, w))
    made_just_before(16, 768, lambda w: o.route_top_k(h, w, None, 2))
    q, gate = torch.randn(4, 12 * 64, generator=gen, device=DEV).bfloat16(), torch.randn(4, 12 * 128, generator=gen, device=DEV).bfloat16()
    made_just_before(12 * 64, 128, lambda w: o.head_linear(q, 64, w, False, torch.empty_like(gate), 128, 12, 64, 128, gate=gate), torch.bfloat16)
    made_just_before(1, 768, lambda w: o.group_norm_gated(h, h, w[0], 12, 1e-5, True, torch.float32))
    made_just_before(1, 768, lambda w: o.group_norm_gated(h, h, w[0], 1, 1e-5, False, torch.float32))
    one = torch.arange(5, dtype=torch.int32, device=DEV)
    old, new = torch.zeros_like(one), torch.ones_like(one)
    state = torch.randn(4, 12 * 64 * 64, generator=gen, device=DEV)
    made_just_before(768, 4, lambda w: o.causal_conv(h, w, None, state, 0, one[:4], one, one[:4], old))
    # retention's decays: a decode step, and chunks of a prompt (fresh entries: the slots' contents are not read)
    for n in (4, 100):
        x = torch.randn(n, 12 * 64, generator=gen, device=DEV).bfloat16()
        start = one if n == 4 else torch.tensor([0, n], dtype=torch.int32, device=DEV)
        freq, positions = torch.rand(16, generator=gen, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
        made_just_before(1, 12, lambda w: o.retention_scan(x, x, x, w[0], 0.125, freq, 32, positions, state, start, one, new, 12, 64, 64, n_tiles=2), size=0.2)


def test_fixed_operands_change_no_bit():
    """With that word weights and the batch's arrays are asked for ahead of the wait, in instances of their own."""
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(4)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    one = torch.arange(9, dtype=torch.int32, device=DEV)
    fresh = (one % 2).int()
    for n in (3, 80):
        h, start = rand(n, 768), one[: n + 1] if n == 3 else torch.tensor([0, n], dtype=torch.int32, device=DEV)
        entry = one[:n] if n == 3 else torch.zeros(n, dtype=torch.int32, device=DEV)
        w, taps, gain, state = rand(24, 768), rand(768, 4), rand(768), rand(8, 12 * 64 * 64)
        q, gate, heads = rand(n, 768).bfloat16(), rand(n, 1536).bfloat16(), rand(768, 128).bfloat16()
        freq, positions, decay = torch.rand(16, generator=gen, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV), torch.full((12,), 0.9, device=DEV)

        def retention(fixed, silu):
            mine = state.clone()
            out = o.retention_scan(q, q, q, decay, 0.125, None if silu else freq, 0 if silu else 32, positions, mine, start, one, fresh, 12, 64, 64, silu, 2, fixed=fixed)
            return torch.cat([out.reshape(-1), mine.reshape(-1)])

        calls = [lambda f: o.small_linear(h, w, None, fixed=f), lambda f: o.small_linear(h[:, :766], w[:, :766].contiguous(), None, fixed=f),
                 lambda f: o.route_top_k(h, w, None, 2, fixed=f)[0], lambda f: o.causal_conv(h, taps, gain, state, 0, entry, start, one, fresh, fixed=f),
                 lambda f: o.head_linear(q, 64, heads, False, torch.empty_like(gate), 128, 12, 64, 128, fixed=f),
                 lambda f: o.head_linear(q, 64, heads, False, torch.empty_like(gate), 128, 12, 64, 128, gate=gate, fixed=f),
                 lambda f: retention(f, False), lambda f: retention(f, True)]
        calls += [lambda f, g=g: o.group_norm_gated(h, h, gain, g, 1e-5, True, torch.float32, fixed=f) for g in (24, 12, 6, 1)]
        for i, call in enumerate(calls):
            assert torch.equal(call(True), call(False)), (n, i)


def few_rows_case(m, n, k, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed + m + 7 * n + 31 * k)
    a = torch.randn(m, k + 8, generator=gen, device=DEV).bfloat16()[:, :k]          # rows with a stride of their own
    w = (torch.randn(n, k + 16, generator=gen, device=DEV) * k ** -0.5).bfloat16()[:, 8: k + 8]
    return gen, a, w


def sums_bound(a, w, k):
    """float32 sums of k exact products: under two roundings a term and some that join the shares, each 2^-23 of the terms' sizes."""
    return (k + 32) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)


# rows around the tiles of 8, 16 and 32; features and K around the rules that pick a split, no multiples of a tile, K beside blocks of 32
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n,k", [(1, 8), (24, 40), (768, 768), (1184, 1000), (1185, 96), (2369, 256), (4737, 64), (2376, 1032), (8192, 32), (72, 2048), (65, 5128), (768, 3072)])
def test_products_of_few_rows(m, n, k):
    o = ops()
    gen, a, w = few_rows_case(m, n, k)
    bias, residual = torch.randn(n, generator=gen, device=DEV), torch.randn(m, n, generator=gen, device=DEV)
    want = a.double() @ w.double().T
    bound = sums_bound(a, w, k)
    got = o.linear(a, w, bias, w_is_nk=True, residual=residual)
    assert ((got.double() - (want + bias.double() + residual.double())).abs() <= bound + 2.0 ** -22 * (bias.abs() + residual.abs() + want.abs())).all()
    out = torch.full((m, n + 3), 7.0, dtype=torch.bfloat16, device=DEV)
    o.linear(a, w, None, w_is_nk=True, out=out[:, 1: n + 1])
    assert ((out[:, 1: n + 1].double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()
    assert (out[:, 0] == 7.0).all() and (out[:, n + 1:] == 7.0).all()


@pytest.mark.parametrize("act", ["gelu_new", "gelu"])
def test_products_of_few_rows_with_an_activation(act):
    o = ops()
    gen, a, w = few_rows_case(5, 200, 768)
    bias = torch.randn(200, generator=gen, device=DEV)
    z = a.double() @ w.double().T + bias.double()
    want = torch.nn.functional.gelu(z, approximate="tanh" if act == "gelu_new" else "none")
    exact = o.linear(a, w, bias, w_is_nk=True, act=act, out_dtype=torch.float32)
    torch.testing.assert_close(exact.double(), want, atol=2e-5, rtol=2e-5)
    rounded = o.linear(a, w, bias, w_is_nk=True, act=act)
    # the hardware's tanh is within 2^-11 of the value and the result is rounded to 2^-9
    torch.testing.assert_close(rounded.double(), want, atol=2.0 ** -10, rtol=2.0 ** -8)


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("k", [64, 768, 1000, 1024])
@pytest.mark.parametrize("centred", [True, False])
def test_products_of_few_rows_with_a_norm(m, k, centred):
    """Rows far from zero: the mean is 30 times the spread."""
    o = ops()
    n = 100
    gen, _, w = few_rows_case(m, n, k)
    x = torch.randn(m, k, generator=gen, device=DEV) + (30.0 if centred else 0.0)
    gain, shift = 1.0 + 0.3 * torch.randn(k, generator=gen, device=DEV), torch.randn(k, generator=gen, device=DEV)
    rows = x.double()
    if centred:
        normed = torch.nn.functional.layer_norm(rows, (k,), gain.double(), shift.double(), 1e-5)
    else:
        normed = rows * torch.rsqrt((rows * rows).mean(-1, keepdim=True) + 1e-5) * gain.double()
    got = o.linear(o.NormedRows(x, gain, shift if centred else None, 1e-5, torch.bfloat16), w, None, w_is_nk=True, out_dtype=torch.float32)
    # each normed value is rounded to bfloat16 once (2^-9 of it, independent signs: a root of the squares' sum, six of them)
    bound = 6 * 2.0 ** -9 * ((normed ** 2) @ (w.double() ** 2).T).sqrt()
    assert ((got.double() - normed @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("t,groups,per,k", [(1, 4, 128, 64), (9, 3, 768, 768), (40, 2, 160, 40), (3, 2, 24, 64)])   # (the last: groups that are no multiple of a CTA's features)
def test_products_of_few_rows_side_by_side(t, groups, per, k):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(t)
    a = torch.randn(t, groups, k, generator=gen, device=DEV).bfloat16()
    w = torch.randn(groups * per, k, generator=gen, device=DEV).bfloat16()
    got = o.grouped_linear(a, w).double().view(t, groups, per)
    for s in range(groups):
        want = a[:, s].double() @ w[s * per: (s + 1) * per].double().T
        assert ((got[:, s] - want).abs() <= sums_bound(a[:, s], w[s * per: (s + 1) * per], k) + 2.0 ** -8 * want.abs()).all()


# one warp to eight, rows that end inside a thread's eight values, the widest row in registers and the next one beyond
@pytest.mark.parametrize("width", [4, 36, 256, 260, 768, 1600, 2048, 2052])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gathered", [False, True])
def test_norms_of_rows(width, dtype, gathered, n_rows=37):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(width)
    x = torch.randn(n_rows, width, generator=gen, device=DEV) + 20.0   # (a mean far beyond the spread)
    gain, shift = torch.randn(width, generator=gen, device=DEV), torch.randn(width, generator=gen, device=DEV)
    rows = torch.tensor([36, 0, 5, 5], dtype=torch.int32, device=DEV) if gathered else None
    read = x[rows.long()].double() if gathered else x.double()
    want = torch.nn.functional.layer_norm(read, (width,), gain.double(), shift.double(), 1e-5)
    # the statistics' roundings grow with mean / spread (20): 2^-24 * 20 a value, some tens of them, beside the result's own rounding
    bound = 2.0 ** -16 * (gain.abs().double() + 1.0) * (1.0 + want.abs()) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0)
    assert ((o.layer_norm(x, gain, shift, 1e-5, dtype, rows=rows).double() - want).abs() <= bound).all()
    want = read * torch.rsqrt((read * read).mean(-1, keepdim=True) + 1e-5) * gain.double()
    bound = 2.0 ** -20 * want.abs() + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0)
    assert ((o.rms_norm(x, gain, 1e-5, dtype, rows=rows).double() - want).abs() <= bound).all()


# contexts (before the new token) around a tile, a CTA's tiles (16 and 24 warps' worth at head size 64, 8 and 12 at 128) and clusters' runs
@pytest.mark.parametrize("h,hkv,hd", [(4, 4, 64), (8, 2, 64), (6, 1, 64), (2, 1, 128), (2, 2, 16)])
@pytest.mark.parametrize("window", [0, 260])
def test_decode_attention_of_every_plan(h, hkv, hd, window, monkeypatch):
    o = ops()
    contexts = [0, 1, 31, 32, 255, 256, 383, 511, 512, 513, 767, 768, 1100]
    wide = 16 if hd <= 64 else 8
    for plan in ((1, 4), (6, 4), (1, wide // 2), (1, wide), (2, wide), (3, wide)):
        pc = PagedCase([(c, 1) for c in contexts], h, hkv, hd, 16, torch.bfloat16, seed=hd + window, garbage=1e4)
        monkeypatch.setattr(o, "decode_plan", lambda *a, **k: plan)
        got = o.decode_attention_fused(pc.q_rows, pc.k_new, pc.v_new, pc.slots, pc.k_cache, pc.v_cache, pc.page_stride, pc.page, pc.n_pages,
                                       pc.tables, pc.row_entry, pc.positions, pc.seq_lens, h, hkv, hd, hd ** -0.5, window, 2048, cache_settled=True)
        torch.testing.assert_close(got.float().cpu(), pc.plain(hd ** -0.5, window), atol=3e-2, rtol=3e-2, msg=lambda m: f"plan {plan}: {m}")
        cached = o.paged_attention(pc.q_rows, pc.k_cache, pc.v_cache, pc.page_stride, pc.page, pc.n_pages, pc.tables, pc.row_entry, pc.positions,
                                   pc.seq_lens, h, hkv, hd, hd ** -0.5, window)   # the new rows are in the cache
        torch.testing.assert_close(cached.float(), got.float(), atol=2e-2, rtol=2e-2)


def test_decode_plans():
    o = ops()
    assert o.decode_plan(8, 12, 64, 1024) == (1, 16) and o.decode_plan(1, 12, 64, 4096) == (4, 16) and o.decode_plan(1, 12, 64, 1024) == (1, 16)
    assert o.decode_plan(16, 12, 64, 1024) == (1, 8) and o.decode_plan(64, 12, 64, 1024) == (1, 4)
    assert o.decode_plan(1, 2, 128, 600) == (2, 8) and o.decode_plan(8, 12, 256, 1024) == (6, 4)   # (head sizes beyond 128 have narrow CTAs alone)


@pytest.mark.parametrize("n_rows", [401, 1500, 1501])   # sixteen values a thread; the most rows of a CTA each, and a warp a row beyond
@pytest.mark.parametrize("width", [260, 1028, 2048])
def test_norms_of_many_rows(n_rows, width):
    for dtype in (torch.float32, torch.bfloat16):
        test_norms_of_rows(width, dtype, False, n_rows)


# a CTA a row and group beside four rows a CTA: taps up to four (five take the other kernel), vectors that are no multiples of four or of a warp
@pytest.mark.parametrize("heads,groups,dim,vdim,taps_n,width", [(4, 2, 24, 16, 4, 52), (6, 6, 7, 5, 3, 768), (12, 6, 64, 64, 4, 768), (3, 1, 40, 90, 1, 1028), (2, 2, 8, 8, 5, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_what_the_delta_rule_walks_over_for_few_rows(heads, groups, dim, vdim, taps_n, width, dtype):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(width + dim)
    channels, n = 2 * groups * dim + heads * vdim, 400
    raw, h = torch.randn(n, channels, generator=gen, device=DEV).to(dtype), torch.randn(n, width, generator=gen, device=DEV).to(dtype)
    weights = (torch.randn(channels, taps_n, generator=gen, device=DEV), (0.1 * torch.randn(2 * heads, width, generator=gen, device=DEV)).to(dtype),
               torch.randn(heads, generator=gen, device=DEV), torch.randn(heads, generator=gen, device=DEV))
    state = torch.randn(2, 8 + (taps_n - 1) * channels + 8, generator=gen, device=DEV)

    def prepared(rows, entry_of, starts, fresh):
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
        return o.delta_prepare(raw[:rows], h[:rows], *weights, 0.2, 1e-6, heads, groups, dim, vdim, state, 8, i32(entry_of), i32(starts), i32([1, 0]), i32(fresh))

    for fresh in (0, 1):
        many, few = prepared(n, [0] * n, [0, n, n], [fresh, 0]), prepared(7, [0] * 6 + [-1], [0, 6, 6], [fresh, 0])   # (the last a pad row)
        for a, b in zip(many, few):
            assert torch.equal(a[:6], b[:6])
            assert torch.isfinite(b).all()


@pytest.mark.parametrize("experts,groups,keep,top", [(8, 4, 2, 2), (10, 2, 1, 3), (31, 1, 1, 31), (32, 8, 3, 5), (33, 3, 2, 4), (1, 1, 1, 1)])
@pytest.mark.parametrize("scoring", ["sigmoid", "softmax"])
@pytest.mark.parametrize("rows", [5, 700])
def test_routers_around_a_warp_of_outputs(experts, groups, keep, top, scoring, rows):
    """Scores of a few values only, so that ties are common: the lower index wins, among groups and among experts."""
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(experts)
    h = torch.zeros(rows, 64, device=DEV)
    h[:, :experts] = torch.randint(-2, 3, (rows, experts), generator=gen, device=DEV).float()
    w = torch.eye(64, device=DEV)[:experts].contiguous()
    dense, chosen, weight, _ = o.route_scored(h, w, None, top, groups, keep, scoring=scoring, group_mark="best", normalise=False)
    z = h[:, :experts].double()
    score = torch.sigmoid(z) if scoring == "sigmoid" else torch.softmax(z, dim=1)
    mark = z.view(rows, groups, -1).amax(-1)
    kept = torch.sort(mark, dim=1, descending=True, stable=True).indices[:, :keep]
    allowed = torch.zeros(rows, groups, dtype=torch.bool, device=DEV).scatter_(1, kept, True).repeat_interleave(experts // groups, dim=1)
    want = torch.sort(z.masked_fill(~allowed, -float("inf")), dim=1, descending=True, stable=True).indices[:, :top]
    assert torch.equal(chosen.long(), want)
    torch.testing.assert_close(weight.double(), score.gather(1, want), atol=1e-6, rtol=1e-6)
    assert torch.equal(dense.gather(1, want), weight) and torch.equal((dense != 0).sum(1), torch.full((rows,), top, device=DEV))
    # rows that are not numbers: indices stay inside
    h[0], h[1, :1], h[2] = float("nan"), float("nan"), float("inf")
    _, chosen, _, _ = o.route_scored(h, w, None, top, groups, keep, scoring=scoring, group_mark="two_best")
    assert int(chosen.min()) >= 0 and int(chosen.max()) < experts


# widths around every number of chunks that a warp may have; the last number of rows of a CTA each, and beyond
@pytest.mark.parametrize("width", [4, 128, 132, 256, 260, 512, 768, 772, 1024, 1028, 1600, 2048])
@pytest.mark.parametrize("gathered", [False, True])
def test_float32_norms_have_the_same_bits_beside_any_number_of_rows(width, gathered):
    o = ops()
    gen = torch.Generator(device=DEV).manual_seed(width)
    x = torch.randn(2100, width, generator=gen, device=DEV) + 3.0
    gain, shift = torch.randn(width, generator=gen, device=DEV), torch.randn(width, generator=gen, device=DEV)
    order = torch.randperm(2100, generator=gen, device=DEV).to(torch.int32) if gathered else torch.arange(2100, dtype=torch.int32, device=DEV)
    read = x if gathered else x[order.long()]
    whole = [o.layer_norm(x, gain, shift, 1e-5, torch.float32, rows=order), o.rms_norm(x, gain, 1e-5, torch.float32, rows=order)]
    for n in (1, 2, 150, 151, 401, 1500, 1501, 1776, 1777, 2099):
        rows = order[:n] if gathered else None
        few = read if gathered else read[:n]
        assert torch.equal(o.layer_norm(few, gain, shift, 1e-5, torch.float32, rows=rows), whole[0][:n]), n
        assert torch.equal(o.rms_norm(few, gain, 1e-5, torch.float32, rows=rows), whole[1][:n]), n
