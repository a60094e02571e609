"""Products of few rows run on the kernel that the rule names, and the tcgen05 kernel still does what it did for matrices stored [out, in]."""

from __future__ import annotations

import pytest
import torch

from tests import test_kernels_gpu as general

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from research_2_b200.kernels import ops as o

    return o


def uses():
    return ops().kernel_uses().get("few_rows", 0)


# sizes of tests/test_few_rows_gpu.py and sizes beyond the rule; K that is no multiple of eight
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("n,k", [(1, 8), (24, 40), (768, 768), (1184, 1000), (1185, 96), (2369, 256), (4737, 64), (8192, 32), (72, 2048), (65, 5128), (768, 3072), (2560, 2560), (64, 100)])
def test_the_rule_names_the_kernel(m, n, k):
    o = ops()
    a, w = torch.zeros(m, k, dtype=torch.bfloat16, device=DEV), torch.zeros(n, k, dtype=torch.bfloat16, device=DEV)
    takes = k % 8 == 0 and bool(o._lib("few_rows").r2_few_rows_takes(m, n, k, 0))
    before = uses()
    o.linear(a, w, None, w_is_nk=True)
    assert uses() - before == int(takes)
    o.linear(a, w.t().contiguous(), None)   # (stored [in, out])
    assert uses() - before == int(takes)
    if m <= 16 and k <= 1024 and k % 8 == 0:
        x, gain = torch.zeros(m, k, device=DEV), torch.ones(k, device=DEV)
        for shift, norm in ((gain, 2), (None, 1)):
            before = uses()
            o.linear(o.NormedRows(x, gain, shift, 1e-5, torch.bfloat16), w, None, w_is_nk=True)
            assert uses() - before == int(bool(o._lib("few_rows").r2_few_rows_takes(m, n, k, norm)))


@pytest.mark.parametrize("per,takes", [(128, 1), (24, 4)])   # groups of no multiple of 32 features run one by one
def test_products_side_by_side_run_on_it(per, takes):
    o = ops()
    before = uses()
    o.grouped_linear(torch.zeros(3, 4, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(4 * per, 64, dtype=torch.bfloat16, device=DEV))
    assert uses() - before == takes


@pytest.mark.parametrize("m,k,n", [(1, 96, 288), (7, 104, 1031), (16, 768, 3072), (64, 768, 2304), (8, 768, 12800)])
def test_matrices_stored_by_feature_on_the_tcgen05_kernel(m, k, n):
    o = ops()
    before, on = uses(), o.use_few_rows(False)
    try:
        general.test_linear(m, k, n, torch.bfloat16, True)
        if m <= 16:
            general.test_linear_with_the_norm_inside(m, k, n, True)
    finally:
        o.use_few_rows(on)
    assert uses() == before


def plain_rows(case, scale, window, keep_first, chunk, softcap, bias, sink_logit, gate, head_gate, factor):
    """Every row's attention in 64 bits; sink_logit [heads] or None."""
    outs = []
    for e, (start, _) in enumerate(case.entries):
        rep = case.n_heads // case.n_kv
        k, v = (x[e].double().repeat_interleave(rep, 1) for x in (case.k_dense, case.v_dense))
        at = torch.arange(start + 1)
        seen = at >= 0
        if window:
            seen = (at > start - window) | (at < keep_first)
        elif chunk:
            seen = at >= start // chunk * chunk
        s = torch.einsum("hd,khd->hk", case.q[e][0].double(), k) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if bias is not None:
            s = s + bias.double()[:, (start - at).clamp(max=bias.shape[1] - 1)]
        s = s.masked_fill(~seen, -float("inf"))
        if sink_logit is not None:
            s = torch.cat([s, sink_logit.double()[:, None]], 1)
        p = torch.softmax(s, 1)[:, : start + 1]
        o = torch.einsum("hk,khd->hd", p, v) * factor
        if gate is not None:
            o = o * torch.sigmoid(gate[e].double().view(o.shape))
        if head_gate is not None:
            o = o * torch.sigmoid(head_gate[e].double())[:, None]
        outs.append(o.reshape(-1))
    return torch.stack(outs).float()


# narrow CTAs alone and in clusters, wide ones with two pairs, one, and in clusters; every extra of the kernel's two richer forms
@pytest.mark.parametrize("h,hkv,hd", [(4, 4, 64), (8, 2, 64), (6, 2, 80), (8, 1, 128), (2, 2, 16)])
@pytest.mark.parametrize("kind", ["kept", "capped", "chunk", "bias"])
def test_decode_attention_of_every_plan_with_its_extras(h, hkv, hd, kind, monkeypatch):
    o = ops()
    contexts = [0, 1, 31, 32, 255, 256, 511, 513, 767, 1100]
    wide = 16 if hd <= 64 else 8
    gen = torch.Generator().manual_seed(h + hd)
    t, scale = len(contexts), hd ** -0.5
    gate, head_gate = torch.randn(t, h * hd, generator=gen).bfloat16(), torch.randn(t, h, generator=gen)
    sinks, bias = torch.randn(h, generator=gen) * 2, torch.randn(h, 300, generator=gen)
    how = {"kept": dict(window=260, keep_first=5, gate=gate), "capped": dict(softcap=3.0, sinks=sinks, head_gate=head_gate),
           "chunk": dict(chunk=400, sinks=sinks, out_scale=0.7), "bias": dict(dist_bias=bias, sinks=sinks, out_scale=1.5)}[kind]
    call = {k: v.to(DEV) if isinstance(v, torch.Tensor) else v for k, v in how.items() if k != "window"}
    if kind == "kept":
        call["sink"] = True
    for plan in ((1, 4), (2, 4), (1, wide // 2), (1, wide), (2, wide), (3, wide)):
        pc = general.PagedCase([(c, 1) for c in contexts], h, hkv, hd, 16, torch.bfloat16, seed=hd, garbage=1e4)
        monkeypatch.setattr(o, "decode_plan", lambda *a, **k: plan)
        got = o.decode_attention_fused(pc.q_rows, pc.k_new, pc.v_new, pc.slots, pc.k_cache, pc.v_cache, pc.page_stride, pc.page, pc.n_pages, pc.tables, pc.row_entry,
                                       pc.positions, pc.seq_lens, h, hkv, hd, scale, how.get("window", 0), 2048, exact_weights=True, cache_settled=True, **call)
        want = plain_rows(pc, scale, how.get("window", 0), how.get("keep_first", 0), how.get("chunk", 0), how.get("softcap", 0.0), how.get("dist_bias"),
                          torch.zeros(h) if kind == "kept" else how.get("sinks"), how.get("gate"), how.get("head_gate"), how.get("out_scale", 1.0))
        # weights carry 16 bits; the result is rounded to bfloat16 (2^-9 of it), and scores have float32's and the fast exponential's errors
        torch.testing.assert_close(got.float().cpu(), want, atol=2.0 ** -10, rtol=2.0 ** -8, msg=lambda m: f"plan {plan}: {m}")
