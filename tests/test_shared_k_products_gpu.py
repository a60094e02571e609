"""Products of many rows: tiles of 64 to 192 columns, and few tiles whose K the CTAs of a cluster share (they finish the tile's columns
between them)."""

from __future__ import annotations

import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from research_2_b200.kernels import ops as o

    return o


def plan_of(m, n, k, nk):
    out = [C.c_int(0) for _ in range(3)]
    ops()._lib("gemm_tc").r2_gemm_tc_plan(m, n, k, int(nk), *[C.byref(x) for x in out])
    return out[0].value, out[1].value


# K shares of unequal length, a K tail, rows and features that end inside a tile, one k-block
SHAPES = [(512, 1024, 1024), (512, 4096, 1024), (576, 6000, 1024), (65, 3080, 136), (130, 4096, 2048), (512, 6392, 1600), (200, 2048, 520), (1024, 1600, 3200), (700, 2040, 4608),
          (2048, 64, 200)]


def shapes_by_plan(w_is_nk):
    """A ragged shape for every (tile width, shares of K) that the plan gives anywhere on a grid of sizes, whatever its constants are."""
    found = {}
    for m in (65, 130, 200, 333, 576, 700, 1000, 2040):
        for k in (200, 1032, 2040, 4096, 6392):
            for n in (136, 520, 1032, 2056, 3208, 4616):
                found.setdefault(plan_of(m, n, k, w_is_nk), (m, k, n))
    return found


@pytest.mark.parametrize("w_is_nk", [False, True])
def test_every_form_that_the_plan_knows(w_is_nk):
    found = shapes_by_plan(w_is_nk)
    assert {bn for bn, _ in found} >= {64, 128, 192} and {bn for bn, shares in found if shares > 1} >= {64, 128}, found
    for shape in found.values():
        check(shape, w_is_nk)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("w_is_nk", [False, True])
def test_tiles_and_shares_of_k(shape, w_is_nk):
    check(shape, w_is_nk)


def check(shape, w_is_nk):
    o = ops()
    m, k, n = shape
    gen = torch.Generator(device=DEV).manual_seed(m + k + n)
    a = torch.randn(m, k, generator=gen, device=DEV).bfloat16()
    w = (torch.randn((n, k) if w_is_nk else (k, n), generator=gen, device=DEV) * k ** -0.5).bfloat16()
    bias, res = torch.randn(n, generator=gen, device=DEV), torch.randn(m, n, generator=gen, device=DEV)

    def run():
        return (o.linear(a, w, None, w_is_nk=w_is_nk, out_dtype=torch.float32), o.linear(a, w, bias, w_is_nk=w_is_nk, residual=res),
                o.linear(a, w, bias, w_is_nk=w_is_nk, act="gelu_new"), o.linear(a, w, bias, w_is_nk=w_is_nk, act="gelu"))

    shared, again = run(), run()
    before = o.use_pair_gemm(False)
    try:
        assert plan_of(m, n, k, w_is_nk)[1] == 1
        whole = run()
    finally:
        o.use_pair_gemm(before)
    assert o.device_errors() == 0
    assert all(torch.equal(x, y) for x, y in zip(shared, again)), "the order of the sums is fixed"
    exact = a.double() @ (w.double().T if w_is_nk else w.double())
    scale = a.double().abs() @ (w.double().abs().T if w_is_nk else w.double().abs())
    # products of bfloat16 are exact in float32; K additions in any order err by at most K 2^-24 of the terms' sizes (and those of the
    # bias and the residual by theirs); errors of a sum grow with its square root in practice, which 1/8 of the bound still holds
    bound = k * 2.0 ** -24 * scale / 8 + 2.0 ** -22
    assert ((shared[0].double() - exact).abs() <= bound).all() and ((whole[0].double() - exact).abs() <= bound).all()
    wanted = exact + bias.double() + res.double()
    assert ((shared[1].double() - wanted).abs() <= bound + 2.0 ** -23 * (wanted.abs() + 8)).all()
    for x, act in ((shared[2], "tanh"), (shared[3], "none")):
        want = F.gelu(exact + bias.double(), approximate=act)
        # a rounding to bfloat16 (2^-9 of the value); the fast tanh errs by 2^-11 of |x|
        assert ((x.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -10 * (exact + bias.double()).abs() + 2.0 ** -12).all()


def test_keys_and_values_of_shared_products_go_to_the_cache():
    o = ops()
    m, heads, kv_heads, hd, page, k_in = 200, 6, 3, 64, 16, 4096
    qw, kvw = heads * hd, kv_heads * hd
    gen = torch.Generator(device=DEV).manual_seed(5)
    a = torch.randn(m, k_in, generator=gen, device=DEV).bfloat16()
    w = (torch.randn(k_in, qw + 2 * kvw, generator=gen, device=DEV) * k_in ** -0.5).bfloat16()
    assert plan_of(m, qw + 2 * kvw, k_in, False)[1] > 1
    n_pages = -(-m // page) + 3
    stride = 2 * kv_heads * page * hd
    slots = (torch.randperm((n_pages - 1) * page)[:m] + page).to(torch.int32).to(DEV)
    pool_a = torch.full((n_pages, stride), 7.0).bfloat16().to(DEV)
    pool_b = pool_a.clone()
    whole = o.linear(a, w)
    o.kv_write(whole[:, qw: qw + kvw], whole[:, qw + kvw:], pool_a.view(-1), pool_a.view(-1)[kv_heads * page * hd:], slots, kv_heads, hd, page, stride, n_pages)
    got, written = o.linear(a, w, None, kv=o.kv_scatter(slots, pool_b.view(-1), pool_b.view(-1)[kv_heads * page * hd:], stride, page, n_pages, qw, kvw, hd))
    assert written and o.device_errors() == 0
    assert torch.equal(got[:, :qw], whole[:, :qw]) and torch.equal(pool_a, pool_b)
