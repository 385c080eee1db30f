"""Short convolutions of prompt portions, four channels and eight tokens a thread, against the kernels of decode steps (a request at a
time and token by token), which make the same sums: portions that start and end anywhere in a group of eight tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps, C, dtype", [(4, 516, torch.bfloat16), (3, 8, torch.float32), (2, 1028, torch.float32), (4, 514, torch.float32), (1, 64, torch.float32)])
def test_the_same_bits_as_token_by_token(taps, C, dtype):
    _check(taps, C, dtype, [19, 1, 8, 2, 30])


# steps large enough (750,000 values) for the kernel of four channels a thread
@pytest.mark.parametrize("taps, C, dtype", [(4, 4100, torch.bfloat16), (3, 4096, torch.float32), (2, 5000, torch.float32), (1, 4096, torch.float32)])
def test_the_same_bits_in_large_steps(taps, C, dtype):
    _check(taps, C, dtype, [19, 1, 8, 2, 170])


def _check(taps, C, dtype, lens):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(taps * C)
    T, R = sum(lens), len(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts, slots = [sum(lens[:i]) for i in range(R + 1)], [4, 0, 2, 1, 3]
    req = [r for r, n in enumerate(lens) for _ in range(n)]
    x, w, bias, tail = (torch.randn(*s, generator=g).cuda() for s in ((T, C), (C, taps), (C,), (R, taps - 1, C)))
    args = (i32(req), i32(starts), i32(slots))
    silu = ops.conv_silu(x, C, w, bias, tail, *args, dtype)
    t_all, t_one = tail.clone(), tail.clone()
    short = ops.short_conv(x, C, w, bias, t_all, *args, R, act="silu")
    for r, n in enumerate(lens):
        at, hist = starts[r], tail[slots[r]].clone()
        for t in range(at, at + n):                        # one token of one request: the other kernels
            one = (i32([0]), i32([0, 1]), i32([0]))
            assert torch.equal(ops.conv_silu(x[t:t + 1], C, w, bias, hist[None].contiguous(), *one, dtype)[0], silu[t])
            hist = torch.cat([hist, x[t:t + 1]])[1:]
        for t in range(at, at + n):
            got = ops.short_conv(x[t:t + 1], C, w, bias, t_one, i32([0]), i32([0, 1]), i32([slots[r]]), 1, act="silu")
            assert torch.equal(got[0], short[t])
    assert torch.equal(t_all, t_one)
