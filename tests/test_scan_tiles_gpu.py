"""The recurrences that walk row by row, at the edges of their tiles of rows and slices of columns: outputs and final states against a
walk in 64 bits, the same bits whether rows can be copied in 16-byte pieces or not, the same bits of the last entry in one step and in
three, and which prompts are copied ahead."""

from __future__ import annotations

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROWS = [15, 16, 0, 33, 1, 64, 3, 97]   # of the entries: around tiles of 16 and 32 rows and groups of four


def ops():
    from research_2_b200.kernels import ops as o

    return o


def entries(rows):
    start = torch.tensor([0] + rows).cumsum(0).int()
    gen = torch.Generator().manual_seed(len(rows))
    return start.to(DEV), torch.randperm(len(rows), generator=gen).int().to(DEV), torch.tensor([i % 2 for i in range(len(rows))]).int().to(DEV)


def shifted(t, by):
    """The same numbers as columns of a wider tensor, `by` columns in (one: no row starts on a 16-byte boundary)."""
    wide = torch.zeros(t.shape[0], t.shape[1] + 8, dtype=t.dtype, device=t.device)
    wide[:, by: by + t.shape[1]] = t
    return wide[:, by: by + t.shape[1]]


def walk64(kind, rows, start, slot, fresh, state, heads, dim, vdim, data):
    """-> (outputs, states by slot: [slots, heads, dim, vdim], or for the memory the tuple that `memory_parts` gives)."""
    out = torch.zeros(sum(rows), heads * vdim, dtype=torch.float64)
    after = [x.clone() for x in state] if kind == "memory" else state.clone()
    for e, n in enumerate(rows):
        if kind == "memory":
            s, z, m = (torch.zeros_like(x[0]) if fresh[e] else x[slot[e]].clone() for x in state)
        else:
            s = torch.zeros_like(state[0]) if fresh[e] else state[slot[e]].clone()
        for t in range(int(start[e]), int(start[e]) + n):
            if kind == "delta":
                q, k, v, num = (data[x][t] for x in ("q", "k", "v", "num"))
                s = s * num[:, 0, None, None]
                u = num[:, 1, None] * (v - torch.einsum("hij,hi->hj", s, k))
                o = torch.einsum("hij,hi->hj", s, q) + num[:, 2, None] * u
                s = s + k[:, :, None] * u[:, None, :]
            elif kind == "mix":
                kv = data["k"][t][:, :, None] * data["v"][t][:, None, :]
                o = torch.einsum("hij,hi->hj", s + data["bonus"][:, :, None] * kv, data["r"][t])
                s = data["w"][t][:, :, None] * s + kv
            elif kind == "memory":
                gates = 15.0 * torch.tanh(data["gates"][t] / 15.0)
                log_in, log_keep = gates[:heads], torch.nn.functional.logsigmoid(gates[heads:])
                top = torch.maximum(log_keep + m, log_in)
                keep, take, m = torch.exp(log_keep + m - top), torch.exp(log_in - top), top
                k, q = data["k"][t], data["q"][t] * dim ** -0.5
                s = keep[:, None, None] * s + take[:, None, None] * k[:, :, None] * data["v"][t][:, None, :]
                z = keep[:, None] * z + take[:, None] * k
                o = torch.einsum("hij,hi->hj", s, q) / (torch.maximum((z * q).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
            else:
                step = torch.nn.functional.softplus(data["steps"][t] + data["bias"])
                s = torch.exp(-torch.exp(data["rate"]) * step)[:, None, None] * s + step[:, None, None] * data["b"][t][None, :, None] * data["x"][t][:, None, :]
                o = torch.einsum("hij,i->hj", s, data["c"][t]) + data["skip"][:, None] * data["x"][t]
            out[t] = o.reshape(-1)
        if n == 0:
            continue
        if kind == "memory":
            for x, y in zip(after, (s, z, m)):
                x[slot[e]] = y
        else:
            after[slot[e]] = s
    return out, after


def unpacked(state, heads, dim, vdim):
    """Slots of [dim / 4][vdim][4] a head as [slots, heads, dim, vdim]."""
    return state.double().cpu().view(-1, heads, -(-dim // 4), vdim, 4).transpose(3, 4).reshape(state.shape[0], heads, -1, vdim)[:, :, :dim]


def memory_parts(state, heads, dim, vdim):
    """A matrix memory's slots: matrices, normalisers and maxima (of the copies that a slice of the columns each has, the first)."""
    per = state.double().cpu().view(state.shape[0], heads, -1)
    return [per[:, :, : dim * vdim].reshape(-1, heads, dim, vdim), per[:, :, dim * vdim: dim * vdim + dim], per[:, :, dim * vdim + dim]]


def scan_plan(dim, vdim, n, heads, dtype, aligned=True):
    out = [C.c_int(0) for _ in range(3)]
    ops()._lib("recurrent").r2_scan_plan(dim, vdim, n, heads, ops().dtype_code(dtype), int(aligned), *[C.byref(x) for x in out])
    return out[0].value, out[1].value, bool(out[2].value)


# heads of whole and of odd pieces, one to sixteen lanes a column, 32 rows of a column a thread, slices of one and of many columns
@pytest.mark.parametrize("heads,dim,vdim", [(3, 64, 64), (2, 32, 40), (2, 20, 36), (3, 4, 8), (2, 8, 10), (1, 200, 24), (2, 128, 64), (1, 96, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_walks_at_the_edges_of_their_tiles(heads, dim, vdim, dtype):
    o, total = ops(), sum(ROWS)
    gen = torch.Generator().manual_seed(dim)
    rand = lambda *s: torch.randn(*s, generator=gen)
    start, slot, fresh = entries(ROWS)
    # (float32 sums of at most `dim` terms behind a decaying state: well below 1e-4 of values around one; the random walks here reach some ten)
    close = lambda got, want: torch.testing.assert_close(got.double().cpu(), want, rtol=1e-4, atol=1e-4 * max(1.0, float(want.abs().max())))
    cpu = (start.cpu(), slot.cpu(), fresh.cpu())

    def compare(kind, run, per_row, state, states_of, data, vd):
        """run(rows' operands, state, start, slot, fresh) for the whole batch, aligned and not, and for its last entry in three steps.
        Which operands can be unaligned is `run`'s."""
        both = []
        for by in (0, 1):
            mine = state.clone().to(DEV)
            both.append((run([t.to(DEV) for t in per_row], by, mine, start, slot, fresh), mine))
        assert torch.equal(both[0][0], both[1][0]) and torch.equal(both[0][1], both[1][1])
        want, after = walk64(kind, ROWS, *cpu, states_of(state), heads, dim, vd, data)
        close(both[0][0], want)
        got_after = states_of(both[0][1])
        for x, y in zip(got_after, after) if kind == "memory" else [(got_after, after)]:
            close(x, y)
        last = len(ROWS) - 1
        row0, n, mine = int(start[last]), ROWS[last], state.clone().to(DEV)
        for begin, end in ((0, 1), (1, 40), (40, n)):
            part = [t.to(DEV)[row0 + begin: row0 + end].contiguous() for t in per_row]
            got = run(part, 0, mine, torch.tensor([0, end - begin], dtype=torch.int32, device=DEV), slot[last:].contiguous(),
                      torch.tensor([int(fresh[last]) if begin == 0 else 0], dtype=torch.int32, device=DEV))
            assert torch.equal(got, both[0][0][row0 + begin: row0 + end])
        assert torch.equal(mine[slot[last]], both[0][1][slot[last]])

    # the delta rule, over prepared rows (contiguous by its contract: unaligned values are a tensor that starts one number late)
    d4 = -(-dim // 4) * 4
    qk = torch.zeros(total, heads, 2, d4)
    qk[..., :dim] = torch.nn.functional.normalize(rand(total, heads, 2, dim), dim=-1)
    num = torch.zeros(total, heads, 4)
    num[..., 0], num[..., 1], num[..., 2] = 0.8 + 0.2 * torch.rand(total, heads, generator=gen), torch.rand(total, heads, generator=gen), (qk[:, :, 0] * qk[:, :, 1]).sum(-1)
    v, packed = rand(total, heads * vdim), rand(len(ROWS), heads * o.scan_state_floats(dim, vdim))
    packed.view(-1, heads, d4 // 4, vdim, 4)[:, :, -1, :, 4 - (d4 - dim):] = 0.0   # (the rows that round a head up: nobody's)

    def late(t):
        wide = torch.empty(t.numel() + 1, device=DEV)[1:].view(t.shape)
        wide.copy_(t)
        return wide

    compare("delta", lambda t, by, s, *b: o.delta_scan(t[0], late(t[1]) if by else t[1], t[2], dim, s, *b), (qk, v, num), packed,
            lambda s: unpacked(s, heads, dim, vdim),
            {"q": qk[:, :, 0, :dim].double(), "k": qk[:, :, 1, :dim].double(), "v": v.double().view(total, heads, vdim), "num": num.double()}, vdim)

    # time mixing
    r, k, x = (rand(total, heads * dim).to(dtype) for _ in range(3))
    w, bonus, packed = 0.5 + 0.5 * torch.rand(total, heads * dim, generator=gen), rand(heads * dim), rand(len(ROWS), heads * o.scan_state_floats(dim, dim))
    packed.view(-1, heads, d4 // 4, dim, 4)[:, :, -1, :, 4 - (d4 - dim):] = 0.0
    view = lambda t: t.double().view(total, heads, dim)
    compare("mix", lambda t, by, s, *b: o.time_mix_scan(*(shifted(x, by) for x in t), bonus.to(DEV), s, *b, heads, dim), (r, k, x, w), packed,
            lambda s: unpacked(s, heads, dim, dim),
            {"r": view(r), "k": view(k), "v": view(x), "w": view(w), "bonus": bonus.double().view(heads, dim)}, dim)

    # the state-space recurrence, whose slot is [heads][dim][vdim]
    x, b, c = rand(total, heads * vdim).to(dtype), rand(total, dim).to(dtype), rand(total, dim).to(dtype)
    steps, bias, rate, skip, state = rand(total, heads), rand(heads), rand(heads), rand(heads), rand(len(ROWS), heads * dim * vdim)
    compare("ssd", lambda t, by, s, *e: o.ssd_scan(*(shifted(x, by) for x in t[:3]), t[3], bias.to(DEV), rate.to(DEV), skip.to(DEV), s, *e, heads, 1, dim, vdim),
            (x, b, c, steps), state, lambda s: s.double().cpu().view(-1, heads, dim, vdim),
            {"x": x.double().view(total, heads, vdim), "b": b.double(), "c": c.double(), "steps": steps.double(), "bias": bias.double(), "rate": rate.double(), "skip": skip.double()}, vdim)

    # the matrix memory (its slots hold a copy of normaliser and maximum for every slice of the columns: the same ones)
    q, k, x, gates = rand(total, heads * dim).to(dtype), rand(total, heads * dim).to(dtype), rand(total, heads * vdim).to(dtype), rand(total, 2 * heads)
    memory = rand(len(ROWS), heads, o.mlstm_state_floats(dim, vdim)).abs()
    copies = memory[:, :, dim * vdim:].view(len(ROWS), heads, -1, dim + 1)
    copies[:] = copies[:, :, :1].clone()
    compare("memory", lambda t, by, s, *b: o.mlstm_scan(*(shifted(x, by) for x in t[:3]), t[3], 15.0, dim ** -0.5, s, *b, heads, dim, vdim), (q, k, x, gates),
            memory.view(len(ROWS), -1), lambda s: memory_parts(s, heads, dim, vdim), {"q": view(q), "k": view(k), "v": x.double().view(total, heads, vdim), "gates": gates.double()}, vdim)
    assert o.device_errors() == 0


@pytest.mark.parametrize("dim,vdim,dtype,copied", [(64, 64, torch.bfloat16, True), (32, 64, torch.float32, True), (96, 40, torch.bfloat16, True), (128, 64, torch.bfloat16, True),
                                                   (64, 64, torch.float32, True), (200, 64, torch.bfloat16, True), (128, 64, torch.float32, True),
                                                   (20, 36, torch.bfloat16, False), (22, 64, torch.float32, False)])
def test_only_walks_whose_tiles_are_copied_ahead_are_cut_into_narrow_slices(dim, vdim, dtype, copied):
    """A slice stages a row's two vectors again: without the copies ahead 64 threads a CTA are slower than 256."""
    threads, splits, ahead = scan_plan(dim, vdim, 16, 12, dtype)
    assert ahead == copied
    if copied:
        assert threads <= 64 or splits == 8
    lanes = 1   # of a column
    while lanes * min(32, max(4, 1 << (-(-dim // 4) - 1).bit_length())) < dim:
        lanes *= 2
    for t, s, a in [(threads, splits, ahead)] * (not copied) + [scan_plan(dim, vdim, 16, 12, dtype, aligned=False)]:
        assert not a and (s == 1 or -(-vdim // (s // 2)) * lanes > 256), (t, s)   # half as many slices would not fit a CTA
