"""Retention's chunks of 128 tokens on the tensor cores, against float64 and the walk: portions at the edges of a chunk, key sizes from 68 to 128, values
beyond one block of 128 columns, more (head, chunk)s than SMs; a value that is infinite reaches no earlier token."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, H, dk, dv):
    g = torch.Generator().manual_seed(H * dk + dv + sum(lens))
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    p = torch.randn(T, 2 * H * dk + H * dv, generator=g).cuda()
    decay = torch.tensor(([0.97, 0.999, 0.5, 1.0, 0.0] * 4)[:H]).cuda()
    state = (torch.randn(R, H, dk, dv, generator=g) * 0.3).cuda()
    starts = [sum(lens[:i]) for i in range(R + 1)]
    from quench6k_b200 import ops

    def run(**kw):
        s = state.clone()
        return ops.retention(p, 0, H * dk, 2 * H * dk, decay, s, i32(starts), i32(list(range(R))), R, H, dk, dv, **kw), s
    return p, decay, state, starts, run


@pytest.mark.parametrize("lens, H, dk, dv", [([127, 128, 129], 2, 128, 128), ([256, 255, 65], 3, 68, 4), ([300], 5, 124, 200), ([1200, 700], 16, 100, 132)])
def test_against_float64(lens, H, dk, dv):
    from quench6k_b200 import ops
    p, decay, state, starts, run = _case(lens, H, dk, dv)
    o_walk, s_walk = run()
    o_chunk, s_chunk = run(longest=max(lens))
    q, k, v = (p[:, c:c + H * w].double().view(-1, H, w) for c, w in ((0, dk), (H * dk, dk), (2 * H * dk, dv)))
    o, s = torch.zeros(len(p), H, dv, dtype=torch.float64, device="cuda"), state.double()
    for r, n in enumerate(lens):
        for t in range(starts[r], starts[r] + n):
            s[r] = decay.double()[:, None, None] * s[r] + k[t][:, :, None] * v[t][:, None]
            o[t] = torch.einsum("hkv,hk->hv", s[r], q[t])
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    for got, walk, want in ((o_chunk.view_as(o), o_walk.view_as(o), o), (s_chunk, s_walk, s)):
        assert far(got, want) <= max(1.2 * far(walk, want), 2.4e-7), (far(got, want), far(walk, want))        # 2.4e-7: two roundings of FP32's last place
    assert ops.tc_status() == 0


def test_an_infinite_value_reaches_no_earlier_token():
    H, dk, dv, lens = 3, 128, 128, [300, 130]
    p, decay, state, starts, run = _case(lens, H, dk, dv)
    clean, _ = run(longest=max(lens))
    p[200, 2 * H * dk + 5] = float("inf")
    p[210, H * dk + 7] = float("nan")
    got, s = run(longest=max(lens))
    walk, s_walk = run()
    assert torch.allclose(got[:200], clean[:200], rtol=1e-5, atol=1e-4) and torch.isfinite(got[:200]).all()
    assert torch.equal(torch.isfinite(got), torch.isfinite(walk)) and torch.equal(torch.isfinite(s), torch.isfinite(s_walk))
    assert torch.equal(got[300:], clean[300:])


def test_results_that_are_not_finite_do_not_hold_a_step_up():
    """A key that is not a number makes a head's results of every later token so: they are summed again, those of other heads and requests keep their bits, and
    the step takes a few times its time (single results one by one took 480 times)."""
    H, dk, dv, lens = 8, 128, 128, [700, 600]
    p, decay, state, starts, run = _case(lens, H, dk, dv)
    decay.fill_(0.99)
    clean, s_clean = run(longest=max(lens))

    def took():
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = 1e9
        for _ in range(3):
            a.record()
            run(longest=max(lens))
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    at_first = took()
    p[200, H * dk + dk + 7] = float("nan")                              # head 1 of the first request
    p[300, 2 * H * dk + 2 * dv + 9] = float("inf")                      # one value column of head 2
    got, s = run(longest=max(lens))
    walk, s_walk = run()
    assert torch.equal(torch.isfinite(got), torch.isfinite(walk)) and torch.equal(torch.isfinite(s), torch.isfinite(s_walk))
    same, heads = torch.isfinite(got), [0] + list(range(3, H))
    assert not same.all() and torch.allclose(got[same], clean[same], rtol=1e-5, atol=1e-4) and torch.equal(s[torch.isfinite(s)], s_clean[torch.isfinite(s)])
    assert torch.equal(got[700:], clean[700:]) and torch.equal(got.view(-1, H, dv)[:, heads], clean.view(-1, H, dv)[:, heads])
    assert took() <= 30 * at_first
