"""The float32 path's product and attention at the sizes where their plans change: a row's bits must not depend on which of the
product's kernels took it, and errors stay inside the bound of a sum of slices."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from research_2_b200.kernels import ops as o

    return o


# K around the slices' length (16 a slice up to 512, then 32, ...) and past what the few-row kernel stages; N around its 32 columns
# and the tiles' 32 and 64; an unaligned N and K take the loads one by one
@pytest.mark.parametrize("k,n", [(1, 5), (15, 32), (16, 33), (512, 64), (513, 31), (768, 2304), (3072, 768), (4100, 40), (8200, 36), (96, 9600), (770, 100)])
@pytest.mark.parametrize("w_is_nk", [False, True])
def test_rows_of_a_product_are_the_same_bits_in_every_kernel(k, n, w_is_nk):
    gen = torch.Generator(device=DEV).manual_seed(k * 7 + n)
    a = torch.randn(700, k, generator=gen, device=DEV)
    w = torch.randn((n, k) if w_is_nk else (k, n), generator=gen, device=DEV)
    bias, res = torch.randn(n, generator=gen, device=DEV), torch.randn(700, n, generator=gen, device=DEV)
    wide = w.double().T if w_is_nk else w.double()
    whole = ops().linear(a, w, bias, w_is_nk=w_is_nk, residual=res)
    # a slice of L terms and at most 32 slices: |error| <= (L + 32 + 3) 2^-24 sum |a w| (+ the two additions' roundings in it)
    length = 16 * -(-k // 512)
    scale = a.double().abs() @ wide.abs() + bias.double().abs() + res.double().abs()
    assert ((whole.double() - (a.double() @ wide + bias.double() + res.double())).abs() <= (length + 35) * 2.0 ** -24 * scale).all()
    for m in (1, 2, 4, 5, 8, 16, 17, 64, 130, 333):
        part = ops().linear(a[:m], w, bias, w_is_nk=w_is_nk, residual=res[:m])
        assert torch.equal(part, whole[:m]), m
    shifted = torch.empty(33, k + 1, device=DEV)[:, 1:].copy_(a[:33])   # rows that start off a 16-byte boundary
    assert torch.equal(ops().linear(shifted, w, bias, w_is_nk=w_is_nk, residual=res[:33]), whole[:33])


# head sizes that are and are not whole 16-byte pieces; contexts around a tile of 32 keys and the eight warps' 256
@pytest.mark.parametrize("head_dim,page", [(64, 16), (30, 12), (128, 32), (200, 8), (264, 16)])
@pytest.mark.parametrize("window", [0, 40])
def test_attention_rows_do_not_depend_on_the_batch(head_dim, page, window):
    o, heads, kv_heads = ops(), 4, 2
    lens = [1, 31, 32, 33, 255, 257, 300]
    tables, at = [], 1
    width = max(-(-n // page) for n in lens)
    for n in lens:
        own = list(range(at, at + -(-n // page)))
        at += len(own)
        tables.append(own + [0] * (width - len(own)))
    gen = torch.Generator(device=DEV).manual_seed(head_dim + window)
    k = torch.randn(at, kv_heads, page, head_dim, generator=gen, device=DEV)
    v = torch.randn(at, kv_heads, page, head_dim, generator=gen, device=DEV)
    pool = torch.stack([k, v], dim=1).contiguous()   # [page][K | V]
    rows = [(e, p) for e, n in enumerate(lens) for p in range(n)]
    q = torch.randn(len(rows), heads * head_dim, generator=gen, device=DEV)

    def run(sel):
        entries = torch.tensor([rows[i][0] for i in sel], dtype=torch.int32, device=DEV)
        positions = torch.tensor([rows[i][1] for i in sel], dtype=torch.int32, device=DEV)
        out = torch.full((len(sel), heads * head_dim), 7.0, device=DEV)
        lib = o._lib("attention_simt")
        import ctypes as C
        tab = torch.tensor(tables, dtype=torch.int32, device=DEV)
        seq = torch.tensor(lens, dtype=torch.int32, device=DEV)
        qs = q[sel].contiguous()
        half = kv_heads * page * head_dim
        status = lib.r2_attention_simt(
            C.c_void_p(qs.data_ptr()), heads * head_dim, C.c_void_p(out.data_ptr()), heads * head_dim, C.c_void_p(pool.data_ptr()),
            C.c_void_p(pool.data_ptr() + 4 * half), C.c_longlong(2 * half), page, C.c_void_p(tab.data_ptr()), width,
            C.c_void_p(entries.data_ptr()), C.c_void_p(positions.data_ptr()), C.c_void_p(seq.data_ptr()), len(sel), heads, kv_heads, head_dim,
            head_dim, C.c_float(head_dim ** -0.5), window, 0, 0, None, 0, at, 0, C.c_float(0.0), None, None, 0, 0, 0, None, 0, C.c_float(1.0),
            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert status == 0
        torch.cuda.synchronize()
        return out

    whole = run(list(range(len(rows))))
    for sel in ([0], [5, 40, 900 % len(rows)], list(range(len(rows) - 9, len(rows)))):
        assert torch.equal(run(sel), whole[sel])
    keys = [torch.cat([k[p] for p in t if p], dim=1) for t in tables]       # [kv_heads][positions][head_dim]
    values = [torch.cat([v[p] for p in t if p], dim=1) for t in tables]
    worst = 0.0
    for i, (e, p) in enumerate(rows):
        lo = max(0, p - window + 1) if window else 0
        kk = keys[e][:, lo: p + 1].double().repeat_interleave(heads // kv_heads, dim=0)
        vv = values[e][:, lo: p + 1].double().repeat_interleave(heads // kv_heads, dim=0)
        s = (kk @ q[i].double().view(heads, head_dim, 1))[..., 0] * head_dim ** -0.5
        want = (torch.softmax(s, dim=-1)[:, None] @ vv)[:, 0].reshape(-1)
        worst = max(worst, float((whole[i].double() - want).abs().max()))
    # scores up to about 5 carry a relative error of some head_dim / 4 roundings, which is the weights' too; outputs are of size one
    assert worst < 5 * (head_dim / 4 + 40) * 2.0 ** -24 * 4


# a bias by distance that forbids all but the nearest keys: whole tiles of 32 keys score -inf, the first ones of most warps among them
@pytest.mark.parametrize("near", [1, 20, 70])
@pytest.mark.parametrize("with_sinks", [False, True])
@pytest.mark.parametrize("dtype,decoded", [(torch.float32, False), (torch.bfloat16, False), (torch.float32, True), (torch.bfloat16, True)])
def test_tiles_of_forbidden_keys_weigh_nothing(near, with_sinks, dtype, decoded):
    from tests.test_kernels_gpu import PagedCase

    heads, dim, scale = 4, 64, 0.125
    entries = [(n - 1, 1) for n in (1, 33, 300, 700)] if decoded else [(0, 300), (250, 90), (0, 1)]
    case = PagedCase(entries, heads, 2, dim, 16, dtype, seed=near)
    gen = torch.Generator().manual_seed(near)
    bias = torch.full((heads, near + 1), float("-inf"))
    bias[:, :near] = torch.randn(heads, near, generator=gen)
    sinks = torch.randn(heads, generator=gen) if with_sinks else None
    want = []
    for e, (start, rows) in enumerate(entries):
        k, v = (x[e].double().repeat_interleave(2, dim=1) for x in (case.k_dense, case.v_dense))
        back = torch.arange(start, start + rows)[:, None] - torch.arange(start + rows)[None]
        s = torch.einsum("thd,jhd->htj", case.q[e].double(), k) * scale + bias.double()[:, back.clamp(0, near)]
        s = s.masked_fill(back < 0, float("-inf"))
        if with_sinks:
            s = torch.cat([s, sinks.double()[:, None, None].expand(heads, rows, 1)], dim=2)
        want.append(torch.einsum("htj,jhd->thd", torch.softmax(s, dim=2)[..., : start + rows], v).reshape(rows, -1))
    want = torch.cat(want)
    extras = dict(dist_bias=bias.to(DEV), sinks=None if sinks is None else sinks.to(DEV))
    # float32: scores of size one over 64 numbers, a dozen roundings each; bfloat16: the output's rounding and the weights' (2^-9 each)
    close = dict(atol=2e-5, rtol=2e-5) if dtype == torch.float32 else dict(atol=1.2e-2, rtol=1.2e-2)
    o = ops()
    old = o.use_fast_attention(False)   # the general kernel
    try:
        torch.testing.assert_close(case.run(scale, **extras).double().cpu(), want, **close)
    finally:
        o.use_fast_attention(old)
    if dtype == torch.bfloat16:
        torch.testing.assert_close(case.run(scale, q_start=case.q_start, n_tiles=case.n_tiles, **extras).double().cpu(), want, **close)
    if dtype == torch.bfloat16 and decoded:
        got = o.decode_attention_fused(case.q_rows, case.k_new, case.v_new, case.slots, case.k_cache, case.v_cache, case.page_stride, case.page, case.n_pages,
                                       case.tables, case.row_entry, case.positions, case.seq_lens, heads, 2, dim, scale, 0, 700, **extras)
        torch.testing.assert_close(got.double().cpu(), want, **close)


def test_threads_with_products_of_different_sizes():
    """Two host threads on streams of their own take turns on one kernel instance with different needs of shared memory: no launch is refused."""
    import threading

    o, failed = ops(), []
    gen = torch.Generator(device=DEV).manual_seed(9)
    sizes = [(8, 4096, 2600), (8, 1600, 2600)]   # (rows, K, N): eight rows of K floats are staged
    operands = [(torch.randn(m, k, generator=gen, device=DEV), torch.randn(k, n, generator=gen, device=DEV)) for m, k, n in sizes]
    want = [o.linear(a, w) for a, w in operands]
    torch.cuda.synchronize()

    def work(i):
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                a, w = operands[i]
                out = torch.empty_like(want[i])
                for _ in range(1500):
                    o.linear(a, w, out=out)
            stream.synchronize()
            assert torch.equal(out, want[i])
        except Exception as ex:  # noqa: BLE001
            failed.append(ex)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
