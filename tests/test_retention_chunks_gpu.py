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
