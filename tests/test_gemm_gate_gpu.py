"""The gate of a gated product (silu(v) * up, rounded to bfloat16) in every form of the tensor-core kernels, out to values where the sigmoid is 0
or 1 and the sum overflows, against float64; and long prompts' rows against the same rows a few at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# rows: tiles of 16, 32, 64 and 128 tokens, CTA pairs (tiles of 192 and 256) with a last tile that ends inside 16, 32 and 48 rows
@pytest.mark.parametrize("M,N", [(9, 136), (32, 200), (61, 4104), (300, 1000), (527, 4872), (1041, 2312), (800, 9480)])
def test_gate_against_float64(M, N):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(M)
    top = 10 ** (torch.rand(M, generator=g) * 6 - 3) * torch.where(torch.rand(M, generator=g) < 0.5, -1.0, 1.0)      # 1e-3 .. 1e3 either side
    top[:6] = torch.tensor([80.0, -80.0, 88.5, -88.5, 0.0, 3e38])
    first = top.to(torch.bfloat16)
    second = (top - first.float()).to(torch.bfloat16)
    second[5] = first[5]                                              # 3e38 twice: infinity
    a = torch.zeros(M, 8, dtype=torch.bfloat16)
    a[:, 0], a[:, 1], a[:, 2] = first, second, 1.0
    scale = 2.0 ** torch.randint(-3, 3, (N,), generator=g)
    scale[1::3] *= -1
    w, w2 = torch.zeros(N, 8, dtype=torch.bfloat16), torch.zeros(N, 8, dtype=torch.bfloat16)
    w[:, 0] = w[:, 1] = scale.to(torch.bfloat16)
    w2[:, 2] = torch.randn(N, generator=g).to(torch.bfloat16)
    v = ((first.double() + second.double())[:, None] * scale).float().cuda()     # exact: two bfloat16 parts, a power of two; beyond FP32's range infinity
    got = ops.gemm_tc(a.cuda(), w.cuda(), w2=w2.cuda())
    want = v.double() * torch.sigmoid(v.double()) * w2[:, 2].cuda().double()
    finite = torch.isfinite(v) & (want.abs() < 3e38)
    # half of bfloat16's last place (of 8 bits), and some four roundings of 6e-8 before it; below e^-70 nothing is asked but nearness to zero
    assert bool(((got.double() - want).abs()[finite] <= want.abs()[finite] * (2.0 ** -8 + 2.0 ** -20) + 1e-28).all())
    infinite = torch.isinf(v)
    division = (v / (1.0 + torch.exp(-v)))[infinite]                  # at infinity: what the division gives
    assert torch.equal(torch.isnan(got[infinite]), torch.isnan(division)) and bool(torch.isinf(got[v == float("inf")]).all())
    assert ops.tc_status() == 0


@pytest.mark.parametrize("M,N,K,act", [(512, 4864, 264, None), (1037, 2304, 64, "gelu_tanh"), (2051, 1160, 136, None)])
def test_pairs_as_rows_a_few_at_a_time(M, N, K, act):
    """CTA pairs and one CTA a tile add the same products in the same order: the same bits."""
    from quench6k_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    a, w, w2 = r(M, K), r(N, K), r(N, K)
    got = ops.gemm_tc(a, w, w2=w2, act=act)
    few = torch.cat([ops.gemm_tc(a[i:i + 256], w, w2=w2, act=act) for i in range(0, M, 256)])
    assert torch.equal(got, few) and ops.tc_status() == 0


@pytest.mark.parametrize("M", [48, 304, 1040])                        # tiles of 64 and of 128 tokens, CTA pairs
def test_a_gate_does_not_depend_on_the_rows_beside_it(M):
    """A dense sweep of gates, from subnormal numbers to beyond where e^-v overflows: the bits of the division, alone or with a neighbour (of the 16
    rows that a thread gates together) that is large."""
    from quench6k_b200 import ops
    N = 264
    g = torch.Generator().manual_seed(M)
    e = torch.rand(M, N, generator=g)
    v = torch.where(e < 0.3, 10 ** (torch.rand(M, N, generator=g) * 42 - 41), torch.rand(M, N, generator=g) * 100)
    v = torch.where(torch.rand(M, N, generator=g) < 0.5, -v, v)
    v[3, :5] = torch.tensor([-87.0, -87.4, -88.7, -88.73, 1e38])
    # one product a row and column: a one-hot row of A picks the gate from W, so v (two bfloat16 parts, exact in FP32) comes out as it is
    first = v.to(torch.bfloat16)
    second = (v - first.float()).to(torch.bfloat16)
    K = (2 * M + 7) // 8 * 8
    a = torch.zeros(M, K, dtype=torch.bfloat16)
    a[torch.arange(M), torch.arange(M)] = 1
    a[torch.arange(M), M + torch.arange(M)] = 1
    w, w2 = torch.zeros(N, K, dtype=torch.bfloat16), torch.zeros(N, K, dtype=torch.bfloat16)
    w[:, :M], w[:, M:2 * M] = first.T, second.T
    w2[:, :M] = torch.randn(N, M, generator=g).to(torch.bfloat16)
    a, w, w2 = a.cuda(), w.cuda(), w2.cuda()
    gate, up = ops.gemm_tc(a, w), ops.gemm_tc(a, w2)                   # the products themselves, FP32
    want = (gate / (1.0 + torch.exp(-gate)) * up).to(torch.bfloat16)
    alone = ops.gemm_tc(a, w, w2=w2)
    assert torch.equal(alone.view(torch.int16), want.view(torch.int16))
    w[:, 15:M:16] = torch.tensor([300.0, -300.0, 1e30, -1e30], dtype=torch.bfloat16, device="cuda").repeat(N // 4 + 1)[:N, None]
    beside = ops.gemm_tc(a, w, w2=w2)
    rows = torch.arange(M) % 16 != 15
    assert torch.equal(beside[rows].view(torch.int16), alone[rows].view(torch.int16))
    assert ops.tc_status() == 0


def test_gates_beyond_80_cost_no_divisions():
    """Gates that spread over +-100 (nearly every warp holds one beyond 80) take the time of small ones: 90 and 88 us here, 235 with divisions for those."""
    from quench6k_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    a, w, w2 = r(4096, 2048).bfloat16(), r(4096, 2048) * 2048 ** -0.5, (r(4096, 2048) * 2048 ** -0.5).bfloat16()
    took = {}
    for spread in (1, 45, 1, 45):
        ws = (w * spread).bfloat16()
        ops.gemm_tc(a, ws, w2=w2)
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        for _ in range(3):
            begin.record()
            for _ in range(10):
                ops.gemm_tc(a, ws, w2=w2)
            end.record()
            end.synchronize()
            took[spread] = min(took.get(spread, 1e9), begin.elapsed_time(end))
    assert took[45] <= 1.5 * took[1], took
