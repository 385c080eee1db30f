"""The selective scan with a lane per state, in one pass, against float64 and against the walk of eight states a lane (which a step of
fewer than eight tokens per request keeps), at the edges of its tiles (64 tokens, walked 16 at a time, and 16 channels) and for state sizes below 16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C, N, taps, dtype, lens", [(40, 16, 4, torch.bfloat16, [33, 1, 32, 97]), (19, 9, 2, torch.float32, [64, 31, 2]),
                                                     (1600, 16, 4, torch.bfloat16, [129]), (16, 12, 1, torch.float32, [16, 48]), (24, 16, 4, torch.bfloat16, [63, 65]),
                                                     (40, 11, 3, torch.float32, [65, 15, 17, 63])])
def test_lanes_against_float64(C, N, taps, dtype, lens):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(C + N)
    T, R = sum(lens), len(lens)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts, slots = [sum(lens[:i]) for i in range(R + 1)], list(range(R, 0, -1))
    u, dt_raw, dt_b, proj = rnd(T, C).to(dtype), rnd(T, C) * 0.5 - 2, rnd(C) * 0.5, rnd(T, 2 * N + 5)
    A, D, xz = -torch.exp(rnd(C, N)), rnd(C), rnd(T, 2 * C)
    state, tail = rnd(R + 1, C, N), rnd(R + 1, taps - 1, C)
    assert ops.library().q6k_selective_scan_lanes_taken(T, R, C, N, 1) == 1 and ops.library().q6k_selective_scan_lanes_taken(1, 1, C, N, 1) == 0
    s1, t1 = state.clone(), tail.clone()
    got = ops.selective_scan(u, dt_raw, dt_b, proj, 5, 5 + N, A, D, xz, C, s1, t1, i32(starts), i32(slots), R)
    s2, t2, walked = state.clone(), tail.clone(), []
    for r, n in enumerate(lens):
        for t in range(starts[r], starts[r] + n):
            walked.append(ops.selective_scan(u[t:t + 1], dt_raw[t:t + 1], dt_b, proj[t:t + 1], 5, 5 + N, A, D, xz[t:t + 1], C, s2, t2, i32([0, 1]), i32([slots[r]]), 1))
    walked = torch.cat(walked)
    d = lambda x: x.double()
    dt = torch.nn.functional.softplus(d(dt_raw) + d(dt_b))
    want, S = torch.zeros(T, C, dtype=torch.float64, device="cuda"), d(state)
    for r, n in enumerate(lens):
        for t in range(starts[r], starts[r] + n):
            S[slots[r]] = torch.exp(dt[t][:, None] * d(A)) * S[slots[r]] + (dt[t] * d(u[t]))[:, None] * d(proj[t, 5:5 + N])
            want[t] = (S[slots[r]] @ d(proj[t, 5 + N:5 + 2 * N]) + d(D) * d(u[t])) * torch.nn.functional.silu(d(xz[t, C:]))
    far = lambda x, y: float((d(x) - y).norm() / y.norm())
    # the same products in the same order over time; a token's 16 are added in another order
    assert far(s1, S) <= 1.01 * far(s2, S) + 1e-8 and torch.equal(t1, t2)
    assert far(got, want) <= 1.05 * far(walked, want) + 1e-7


@pytest.mark.parametrize("C, lens, lanes", [(1600, [65, 1100, 63], True), (256, [65, 1100, 63], False)])
def test_either_side_of_the_line_between_one_pass_and_segments(C, lens, lanes):
    """Portions of several segments in one pass (enough chains) and in segments, against float64."""
    from quench6k_b200 import ops
    N, taps = 16, 4
    g = torch.Generator().manual_seed(C)
    T, R = sum(lens), len(lens)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts = [sum(lens[:i]) for i in range(R + 1)]
    u, dt_raw, dt_b, proj = rnd(T, C), rnd(T, C) * 0.5 - 2, rnd(C) * 0.5, rnd(T, 2 * N)
    A, D, xz, state, tail = -torch.exp(rnd(C, N)), rnd(C), rnd(T, 2 * C), rnd(R, C, N), rnd(R, taps - 1, C)
    segments = ops.selective_scan_segments(lens, u.device)
    assert bool(ops.library().q6k_selective_scan_lanes_taken(T, R, C, N, segments[0])) == lanes
    s, before = state.clone(), ops.launch_count
    got = ops.selective_scan(u, dt_raw, dt_b, proj, 0, N, A, D, xz, C, s, tail, i32(starts), i32(list(range(R))), R, segments=segments, longest=max(lens))
    assert ops.launch_count - before == (1 if lanes else 3)
    d = lambda x: x.double()
    dt = torch.nn.functional.softplus(d(dt_raw) + d(dt_b))
    want, S = torch.zeros(T, C, dtype=torch.float64, device="cuda"), d(state)
    for r, n in enumerate(lens):
        for t in range(starts[r], starts[r] + n):
            S[r] = torch.exp(dt[t][:, None] * d(A)) * S[r] + (dt[t] * d(u[t]))[:, None] * d(proj[t, :N])
            want[t] = (S[r] @ d(proj[t, N:]) + d(D) * d(u[t])) * torch.nn.functional.silu(d(xz[t, C:]))
    far = lambda x, y: float((d(x) - y).norm() / y.norm())
    assert far(s, S) < 1e-6 and far(got, want) < 1e-6          # FP32 sums (6e-8 a rounding), a decayed state: about 16 roundings that matter


def test_which_walk_short_portions_take():
    """Up to 64 tokens: a lane per state where the longest portion outlasts the rounds of its blocks."""
    from quench6k_b200 import ops
    taken = ops.library().q6k_selective_scan_lanes_taken
    assert taken(64, 1, 4096, 16, 1) and taken(64, 2, 4096, 16, 1) and taken(2048, 32, 4096, 16, 1)
    assert not taken(256, 32, 4096, 16, 1) and not taken(32, 32, 4096, 16, 1) and not taken(64, 1, 1 << 20, 16, 1 << 30)
    assert not taken(1 << 12, 1, (1 << 20) + 16, 16, 1)        # more blocks of channels than a grid has rows


@pytest.mark.parametrize("C, N, dtype, lens", [(17, 9, torch.bfloat16, [32, 31, 33, 1, 96]), (16, 15, torch.float32, [64, 95, 97]), (33, 16, torch.float32, [30, 47, 48, 49])])
def test_lanes_of_two_states_at_extremes(C, N, dtype, lens):
    """Tiles of 32 tokens and odd state counts, with steps so short and so long that decays lie on both sides of their series' end, and gates out to
    where the sigmoid is 0 or 1 (infinity included): the states are those of the walk of single tokens bit for bit, the results up to the order in which
    16 products are added."""
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(C * N)
    T, R, taps = sum(lens), len(lens), 4
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts = [sum(lens[:i]) for i in range(R + 1)]
    u, dt_raw, dt_b, proj = rnd(T, C).to(dtype), rnd(T, C) * 8, rnd(C) * 0.5, rnd(T, 2 * N)
    A, D, xz, state, tail = -torch.exp(rnd(C, N)), rnd(C), rnd(T, 2 * C) * 30, rnd(R, C, N), rnd(R, taps - 1, C)
    xz[::7, C] = float("inf")
    xz[1::7, C] = -1e30
    assert ops.library().q6k_selective_scan_lanes_taken(T, R, C, N, 1) == 1
    s1, t1, s2, t2, walked = state.clone(), tail.clone(), state.clone(), tail.clone(), []
    got = ops.selective_scan(u, dt_raw, dt_b, proj, 0, N, A, D, xz, C, s1, t1, i32(starts), i32(list(range(R))), R)
    for r, n in enumerate(lens):
        for t in range(starts[r], starts[r] + n):
            walked.append(ops.selective_scan(u[t:t + 1], dt_raw[t:t + 1], dt_b, proj[t:t + 1], 0, N, A, D, xz[t:t + 1], C, s2, t2, i32([0, 1]), i32([r]), 1))
    walked = torch.cat(walked)
    finite = torch.isfinite(walked)
    assert torch.equal(finite, torch.isfinite(got)) and torch.equal(walked[~finite], got[~finite]) and torch.equal(t1, t2)
    assert torch.equal(s1, s2)
    # 16 FP32 products and a skip in another order (some 20 roundings of 6e-8 of the largest), times the gate; bfloat16: a neighbouring value
    scale = float(walked[finite].abs().max())
    torch.testing.assert_close(got[finite], walked[finite], rtol=2 ** -7 if dtype == torch.bfloat16 else 2e-6, atol=2e-6 * scale)


@pytest.mark.parametrize("lens", [[1500] + [1] * 8, [1] * 8 + [1500]])
def test_a_portion_beside_requests_of_a_token_takes_its_own_time(lens):
    """The portion's blocks of channels start together, on SMs of their own: 74 us where the portion alone takes 71 (151 with the requests' blocks in turn)."""
    from quench6k_b200 import ops
    C, N = 1536, 16
    g = torch.Generator().manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")

    def took(lens):
        T, R = sum(lens), len(lens)
        u, dt_raw, dt_b, proj = rnd(T, C).bfloat16(), rnd(T, C), rnd(C), rnd(T, 2 * N)
        A, D, xz, state, tail = -torch.exp(rnd(C, N)), rnd(C), rnd(T, 2 * C), rnd(R, C, N), rnd(R, 3, C)
        starts, slots, segments = i32([sum(lens[:i]) for i in range(R + 1)]), i32(list(range(R))), ops.selective_scan_segments(lens, u.device)
        best = 1e9
        for _ in range(4):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(8):
                ops.selective_scan(u, dt_raw, dt_b, proj, 0, N, A, D, xz, C, state, tail, starts, slots, R, segments=segments, longest=max(lens))
            end.record()
            end.synchronize()
            best = min(best, begin.elapsed_time(end) / 8)
        return best

    assert took(lens) <= 1.5 * took([1500])
