"""The delta rule chunk by chunk against the walk token by token and against float64, at the edges of chunks (32 tokens), of the
columns of a block (16) and of the key sizes, for requests of different lengths in one step; strong and weak decays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, G, dk, dv, rate", [(4, 2, 128, 128, -2.0), (3, 1, 64, 20, -4.0), (2, 2, 4, 16, 0.0), (6, 3, 100, 36, 2.5), (2, 1, 256, 12, -3.0)])
def test_chunks_against_the_walk(H, G, dk, dv, rate):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H * dk + dv)
    lens = [100, 1, 32, 33, 64, 7]
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    u, p = rnd(T, 2 * G * dk + H * dv), rnd(T, 2 * H + 3)
    A_log, dt_bias, state = rnd(H) * 0.5 + rate, rnd(H) * 0.5, rnd(R + 1, H, dv, dk) * 0.3
    starts, slots = [sum(lens[:i]) for i in range(R + 1)], [3, 0, 5, 1, 6, 2]
    assert ops.gated_delta_chunks(max(lens), G, H, dk, dv) and not ops.gated_delta_chunks(16, G, H, dk, dv) and not ops.gated_delta_chunks(100, G, H, dk + 1, dv)
    run = lambda st, **kw: ops.gated_delta(u.clone(), p, 1, H + 2, A_log, dt_bias, st, i32(starts), i32(slots), R, H, G, dk, dv, **kw)
    s_walk, s_chunk = state.clone(), state.clone()
    o_walk, o_chunk = run(s_walk), run(s_chunk, prepare=True, chunked=True)
    # float64, token by token
    d = lambda x: x.double()
    o, s = torch.zeros(T, H, dv, dtype=torch.float64, device="cuda"), d(state)
    q, k, v = d(u[:, :G * dk]).view(T, G, dk), d(u[:, G * dk:2 * G * dk]).view(T, G, dk), d(u[:, 2 * G * dk:]).view(T, H, dv)
    unit = lambda z: (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    q, k = unit(q) * dk ** -0.5, unit(k)
    beta, decay = torch.sigmoid(d(p[:, 1:1 + H])), torch.exp(-torch.exp(d(A_log)) * torch.nn.functional.softplus(d(p[:, H + 2:2 * H + 2]) + d(dt_bias)))
    for r, n in enumerate(lens):
        S = s[slots[r]]
        for t in range(starts[r], starts[r] + n):
            S = decay[t][:, None, None] * S
            S = S + (beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t])))[:, :, None] * k[t][:, None]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t])
        s[slots[r]] = S
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    for got, walk, want in ((o_chunk.view_as(o), o_walk.view_as(o), o), (s_chunk, s_walk, s)):
        # both sum the same FP32 products, in another order; a chunk's are shorter sums.  1e-6: eight roundings of the result
        assert far(got, want) <= max(1.2 * far(walk, want), 1e-6), (far(got, want), far(walk, want))
    assert torch.equal(s_chunk[4], state[4])                   # a slot of no request of this step


@pytest.mark.parametrize("lens", [[1, 100, 64, 65, 1, 7, 130], [65], [64, 1, 66], [1] * 30 + [97]])
def test_short_portions_beside_long_ones_are_walked(lens):
    """Said that there are short portions, a step walks them as a step of their own would, bit for bit; the long ones go chunk by chunk."""
    from quench6k_b200 import ops
    H, G, dk, dv = 4, 2, 64, 36
    g = torch.Generator().manual_seed(len(lens))
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    u, p = rnd(T, 2 * G * dk + H * dv), rnd(T, 2 * H)
    A_log, dt_bias, state = rnd(H) * 0.5 - 2.0, rnd(H) * 0.5, rnd(R, H, dv, dk) * 0.3
    A_log[0] = 6.0                                                       # decays whose logarithms are below -200
    starts = [sum(lens[:i]) for i in range(R + 1)]

    def run(rows, q_start, slots, **kw):
        s = state.clone()
        o = ops.gated_delta(u[rows].clone(), p[rows].contiguous(), 0, H, A_log, dt_bias, s, i32(q_start), i32(slots), len(slots), H, G, dk, dv, prepare=True, **kw)
        return o, s

    mixed, s_mixed = run(slice(0, T), starts, list(range(R)), chunked=True, shortest=min(lens))
    chunked, s_chunked = run(slice(0, T), starts, list(range(R)), chunked=True)
    for r, n in enumerate(lens):
        rows = slice(starts[r], starts[r + 1])
        o, s = run(rows, [0, n], [r]) if n <= ops.CHUNKS_BEYOND else (chunked[rows], s_chunked)
        assert torch.equal(mixed[rows], o) and torch.equal(s_mixed[r], s[r]), (r, n)


def test_more_scratch_than_the_limit_is_walked(monkeypatch):
    """A step whose chunks' matrices would pass the limit goes token by token: decays, not their logarithms, and the walk's bits."""
    from quench6k_b200 import ops
    H, G, dk, dv, T = 2, 1, 32, 16, 100
    g = torch.Generator().manual_seed(1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    u, p, A_log, dt_bias, state = rnd(T, 2 * G * dk + H * dv), rnd(T, 2 * H), rnd(H), rnd(H), rnd(1, H, dv, dk)

    def run(**kw):
        s = state.clone()
        return ops.gated_delta(u.clone(), p, 0, H, A_log, dt_bias, s, i32([0, T]), i32([0]), 1, H, G, dk, dv, prepare=True, **kw), s

    walk, chunks = run(), run(chunked=True)
    assert not torch.equal(walk[0], chunks[0])
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_FLOATS", 1000)
    assert all(torch.equal(a, b) for a, b in zip(run(chunked=True), walk))
