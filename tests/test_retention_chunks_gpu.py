"""Retention chunk by chunk against the walk token by token and against float64, at the edges of chunks (64 tokens), of the columns
of a block (128) and of the key sizes, for requests of different lengths in one step; strong and weak decays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, dk, dv", [(4, 128, 128), (3, 64, 20), (2, 4, 16), (3, 100, 36), (2, 256, 132)])
def test_chunks_against_the_walk(H, dk, dv):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H * dk + dv)
    lens = [200, 1, 64, 65, 128, 7]
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    p = rnd(T, 2 * H * dk + 2 * H * dv + 4)
    decay = torch.tensor([0.5, 0.97, 0.999, 0.0][:H]).cuda()
    state = rnd(R + 1, H, dk, dv) * 0.3
    starts, slots = [sum(lens[:i]) for i in range(R + 1)], [3, 0, 5, 1, 6, 2]
    q_col, k_col, v_col = 4, 4 + H * dk, 4 + 2 * H * dk
    run = lambda st, **kw: ops.retention(p, q_col, k_col, v_col, decay, st, i32(starts), i32(slots), R, H, dk, dv, **kw)
    s_walk, s_chunk = state.clone(), state.clone()
    o_walk = run(s_walk)
    before = ops.launch_count
    o_chunk = run(s_chunk, longest=max(lens))
    assert ops.launch_count - before == 3, "the chunked kernels did not run"
    d = lambda x: x.double()
    o, s = torch.zeros(T, H, dv, dtype=torch.float64, device="cuda"), d(state)
    q, k, v = (d(p[:, c:c + H * w]).view(T, H, w) for c, w in ((q_col, dk), (k_col, dk), (v_col, dv)))
    for r, n in enumerate(lens):
        S = s[slots[r]]
        for t in range(starts[r], starts[r] + n):
            S = d(decay)[:, None, None] * S + k[t][:, :, None] * v[t][:, None]
            o[t] = torch.einsum("hkv,hk->hv", S, q[t])
        s[slots[r]] = S
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    for got, walk, want in ((o_chunk.view_as(o), o_walk.view_as(o), o), (s_chunk, s_walk, s)):
        # both sum the same FP32 products, in another order; a chunk's are shorter sums.  1e-6: eight roundings of the result
        assert far(got, want) <= max(1.2 * far(walk, want), 1e-6), (far(got, want), far(walk, want))
    assert torch.equal(s_chunk[4], state[4])                   # a slot of no request of this step


@pytest.mark.parametrize("lens", [[1, 100, 64, 65, 1, 7, 130], [64, 1, 66], [1] * 30 + [97]])
def test_short_portions_beside_long_ones_are_walked(lens):
    """Said that there are short portions, a step walks them as a step of their own would, bit for bit; the long ones go chunk by chunk."""
    from quench6k_b200 import ops
    H, dk, dv = 3, 64, 36
    g = torch.Generator().manual_seed(len(lens))
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    p, state = torch.randn(T, 2 * H * dk + H * dv, generator=g).cuda(), torch.randn(R, H, dk, dv, generator=g).cuda()
    decay = torch.tensor([0.5, 0.97, 0.0]).cuda()
    starts = [sum(lens[:i]) for i in range(R + 1)]

    def run(rows, q_start, slots, **kw):
        s = state.clone()
        return ops.retention(p[rows].contiguous(), 0, H * dk, 2 * H * dk, decay, s, i32(q_start), i32(slots), len(slots), H, dk, dv, **kw), s

    before = ops.launch_count
    mixed, s_mixed = run(slice(0, T), starts, list(range(R)), longest=max(lens), shortest=min(lens))
    assert ops.launch_count - before == 4                        # three kernels over chunks, one walk
    chunked, s_chunked = run(slice(0, T), starts, list(range(R)), longest=max(lens))
    for r, n in enumerate(lens):
        rows = slice(starts[r], starts[r + 1])
        o, s = run(rows, [0, n], [r]) if n <= ops.CHUNKS_BEYOND else (chunked[rows], s_chunked)
        assert torch.equal(mixed[rows], o) and torch.equal(s_mixed[r], s[r]), (r, n)


def test_more_scratch_than_the_limit_is_walked(monkeypatch):
    """A step whose chunks' states would pass the limit goes token by token, with the walk's bits."""
    from quench6k_b200 import ops
    H, dk, dv, T = 2, 32, 16, 200
    g = torch.Generator().manual_seed(1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    p, state, decay = torch.randn(T, 2 * H * dk + H * dv, generator=g).cuda(), torch.randn(1, H, dk, dv, generator=g).cuda(), torch.tensor([0.5, 0.97]).cuda()

    def run(**kw):
        s = state.clone()
        return ops.retention(p, 0, H * dk, 2 * H * dk, decay, s, i32([0, T]), i32([0]), 1, H, dk, dv, **kw), s

    walk, chunks = run(), run(longest=T)
    assert not torch.equal(walk[0], chunks[0])
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_FLOATS", 1000)
    assert all(torch.equal(a, b) for a, b in zip(run(longest=T), walk))
