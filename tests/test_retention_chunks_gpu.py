"""Retention over prompts in chunks of 64 rows and in decode steps, at the chunks' edges: against 64 bits, and no further from them than
the walk row by row."""

from __future__ import annotations

import pytest
import torch

from tests.plain import zudalorn_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from research_2_b200.kernels import ops as o

    return o


# heads, dim, vdim, rotated dimensions: whole 16-byte pieces, odd sizes that take the loads one by one, several slices of the columns
@pytest.mark.parametrize("heads,dim,vdim,rot_dims", [(3, 32, 64, 32), (2, 24, 40, 8), (2, 20, 36, 20), (1, 64, 130, 48), (2, 128, 64, 64)])
def test_rotated_retention_in_chunks(heads, dim, vdim, rot_dims):
    o = ops()
    gen = torch.Generator().manual_seed(dim + vdim)
    rows = [64, 1, 63, 200, 65, 0, 1, 128]           # entries: whole and partial chunks, single decoded rows, none
    starts = [0, 700, 5, 0, 33, 0, 0, 64]            # the positions they start at (0: from a state of zeros)
    total = sum(rows)
    proj = torch.randn(total, heads * (2 * dim + vdim) + 8, generator=gen).bfloat16()
    decay = torch.tensor([1.0 - 2.0 ** (-3.0 - 2 * h) for h in range(heads)], dtype=torch.float64)
    freqs = [10000.0 ** (-2.0 * i / rot_dims) for i in range(rot_dims // 2)]
    first_state = torch.randn(len(rows), heads, dim, vdim, generator=gen)
    q_start = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int32)
    positions = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, rows)]).int()
    slots = torch.tensor([3, 0, 7, 1, 2, 6, 5, 4], dtype=torch.int32)
    fresh = torch.tensor([int(s == 0) for s in starts], dtype=torch.int32)
    dev = proj.to(DEV)
    a, b = heads * dim, 2 * heads * dim
    state0 = torch.zeros(len(rows), heads * dim * vdim)
    state0[slots.long()] = first_state.reshape(len(rows), -1)

    def run(n_tiles):
        state = state0.to(DEV).clone()
        out = o.retention_scan(dev[:, :a], dev[:, a:b], dev[:, b: b + heads * vdim], decay.float().to(DEV), dim ** -0.5,
                               torch.tensor(freqs).float().to(DEV), rot_dims, positions.to(DEV), state, q_start.to(DEV), slots.to(DEV), fresh.to(DEV),
                               heads, dim, vdim, n_tiles=n_tiles)
        return out.double().cpu(), state.double().cpu()

    def walk64(turn, k_scale):
        exact = torch.zeros(total, heads * vdim, dtype=torch.float64)
        exact_state = state0.double().clone()
        cells = decay.float().double()
        for e, n in enumerate(rows):
            if n == 0:
                continue
            at = slice(int(q_start[e]), int(q_start[e]) + n)
            q = turn(proj[at, :a].double().view(n, heads, dim), positions[at])
            k = turn(proj[at, a:b].double().view(n, heads, dim), positions[at]) * k_scale
            v = proj[at, b: b + heads * vdim].double().view(n, heads, vdim)
            s = torch.zeros(heads, dim, vdim, dtype=torch.float64) if starts[e] == 0 else first_state[e].double()
            for t in range(n):
                s = cells[:, None, None] * s + k[t][:, :, None] * v[t][:, None, :]
                exact[int(q_start[e]) + t] = torch.einsum("hdv,hd->hv", s, q[t]).reshape(-1)
            exact_state[slots[e]] = s.reshape(-1)
        return exact, exact_state

    def turn_by_float_angles(x, pos):
        angle = (pos.float()[:, None] * torch.tensor(freqs).float()[None]).double()
        cos, sin, half = angle.cos()[:, None], angle.sin()[:, None], rot_dims // 2
        u, w = x[..., :half], x[..., half: rot_dims]
        return torch.cat([u * cos - w * sin, w * cos + u * sin, x[..., rot_dims:]], dim=-1)

    before = dict(o._uses)
    walked = run(0)
    assert o._uses.get("decay_chunks", 0) == before.get("decay_chunks", 0)
    chunks = run(sum(-(-n // 64) for n in rows) + 3)
    assert o._uses["decay_chunks"] == before.get("decay_chunks", 0) + 1
    for x, y, want in zip(walked, chunks, walk64(lambda x, pos: plain.rotate(x, pos.tolist(), freqs, "half"), dim ** -0.5)):
        off, off_chunks = (x - want).norm() / want.norm(), (y - want).norm() / want.norm()
        # angles of positions up to 700 in float32 err by 700 2^-24 = 4e-5 in both; the sums' own errors lie below that
        assert off_chunks <= 1.25 * off + 2e-7 and off_chunks < 5e-5, (float(off), float(off_chunks))
    # with the angles and the scale that the kernels are given, which both forms share: the sums' own errors. Three terms, large products' sums of
    # 16 added by rounding additions and powers of 48 bits leave less of them than a float chain a row (measured 0.3 to 0.8 of it)
    for x, y, want in zip(walked, chunks, walk64(turn_by_float_angles, float(torch.tensor(dim ** -0.5, dtype=torch.float32)))):
        off, off_chunks = (x - want).norm() / want.norm(), (y - want).norm() / want.norm()
        assert off_chunks <= off, (float(off), float(off_chunks))
    idle = [int(s) for s, n in zip(slots, rows) if n == 0]
    assert torch.equal(chunks[1][idle], state0.double()[idle])


@pytest.mark.parametrize("dim,vdim,rot_dims", [(32, 64, 32), (20, 36, 8), (64, 128, 64)])
def test_rotated_retention_in_a_decode_step(dim, vdim, rot_dims):
    o, heads, n = ops(), 3, 5
    gen = torch.Generator().manual_seed(dim)
    q, k, v = (torch.randn(n, heads * w, generator=gen).bfloat16() for w in (dim, dim, vdim))
    decay = torch.tensor([0.5, 0.9, 0.999])
    freqs = [100.0 ** (-2.0 * i / rot_dims) for i in range(rot_dims // 2)]
    state = torch.randn(n, heads, dim, vdim, generator=gen)
    positions = torch.tensor([0, 3, 900, 17, 64], dtype=torch.int32)
    fresh = (positions == 0).int()
    dev = state.reshape(n, -1).to(DEV).contiguous()
    got = o.retention_scan(q.to(DEV), k.to(DEV), v.to(DEV), decay.to(DEV), dim ** -0.5, torch.tensor(freqs).to(DEV), rot_dims, positions.to(DEV), dev,
                           torch.arange(n + 1, dtype=torch.int32).to(DEV), torch.arange(n, dtype=torch.int32).to(DEV), fresh.to(DEV), heads, dim, vdim)
    qq = plain.rotate(q.double().view(n, heads, dim), positions.tolist(), freqs, "half")
    kk = plain.rotate(k.double().view(n, heads, dim), positions.tolist(), freqs, "half") * dim ** -0.5
    s = state.double() * (1 - fresh.double())[:, None, None, None]
    s = decay.double()[None, :, None, None] * s + kk[..., None] * v.double().view(n, heads, 1, vdim)
    want = torch.einsum("nhdv,nhd->nhv", s, qq).reshape(n, -1)
    # an angle of 900 in float32 is off by up to 900 2^-24 = 5e-5 of a turn's radius
    torch.testing.assert_close(got.double().cpu(), want, atol=2e-4 * dim ** 0.5, rtol=1e-4)
    torch.testing.assert_close(dev.double().cpu(), s.reshape(n, -1), atol=2e-4, rtol=1e-4)
