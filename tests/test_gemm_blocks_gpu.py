"""How the tcgen05 products' results leave: whole blocks of 16 rows x 32 columns as tensor stores (or additions in L2), what reaches
beyond a tile's rows, or lies off 16 bytes, from registers.  Sizes at the edges of both, results and the columns beside them."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _t(*shape, seed=0, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).to(dtype)


# CTA pairs (512 rows and more, tiles of 192 and of 256 tokens), one CTA with tiles of 128 to 256 tokens, K in slices; N off 32 and off 4
@pytest.mark.parametrize("M,N,K", [(1522, 2048, 256), (512, 4864, 72), (513, 4870, 64), (767, 4867, 64), (1041, 2304, 128), (2048, 2052, 64),
                                   (129, 1000, 64), (160, 36, 64), (255, 33, 200), (300, 4100, 64), (700, 130, 2048), (527, 260, 1024)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_and_columns_at_the_edges(M, N, K, shift):
    from quench6k_b200 import ops
    a, w, w2 = _t(M, K), _t(N, K, seed=1), _t(N, K, seed=2)
    ref = a.double() @ w.double().T
    tol = 1e-5 * math.sqrt(K) * float(ref.abs().max())          # FP32 accumulation of K products of the operands' spread
    base = _t(M * N + 8, seed=3, dtype=torch.float32)                   # the results lie 16 (or 20) bytes behind its start, with 16 (or 12) behind them
    for add in (False, True):
        whole = base.clone()
        out = whole[4 + shift:4 + shift + M * N].view(M, N)
        ops.gemm_tc(a, w, out=out, accumulate=add)
        want = ref + base[4 + shift:4 + shift + M * N].view(M, N).double() if add else ref
        assert float((out.double() - want).abs().max()) <= tol
        assert torch.equal(whole[:4 + shift], base[:4 + shift]) and torch.equal(whole[4 + shift + M * N:], base[4 + shift + M * N:])
    if not shift:
        gate = ops.gemm_tc(a, w, w2=w2)
        want = torch.nn.functional.silu(ref) * (a.double() @ w2.double().T)
        assert float((gate.double() - want).abs().max()) <= 1e-2 * float(want.abs().max())
    assert ops.tc_status() == 0


def test_groups_end_inside_a_block():
    """Rows of one group next to those of another, in tiles of 128 rows that end anywhere: FP32 and bfloat16 results."""
    from quench6k_b200 import ops
    sizes, N, K = [1, 15, 16, 17, 128, 129, 143, 200, 0, 31], 200, 64
    offsets = torch.tensor([sum(sizes[:i]) for i in range(len(sizes) + 1)], dtype=torch.int32, device=DEV)
    rows = sum(sizes)
    a, w, w2 = _t(rows, K), _t(len(sizes), N, K, seed=1), _t(len(sizes), N, K, seed=2)
    tiles = ops.tile_list(offsets, rows, 128)
    group = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), torch.tensor(sizes, device=DEV))
    ref = torch.einsum("rk,rnk->rn", a.double(), w.double()[group])
    up = torch.einsum("rk,rnk->rn", a.double(), w2.double()[group])
    got = ops.gemm_tc(a, w, groups=tiles, bt=128, rows=rows)
    assert float((got.double() - ref).abs().max()) <= 1e-5 * math.sqrt(K) * float(ref.abs().max())
    rounded = ops.gemm_tc(a, w, groups=tiles, bt=128, rows=rows, rounded=True)
    assert torch.equal(rounded, got.to(torch.bfloat16))
    want = torch.nn.functional.silu(ref) * up
    gate = ops.gemm_tc(a, w, w2=w2, groups=tiles, bt=128, rows=rows)
    assert float((gate.double() - want).abs().max()) <= 1e-2 * float(want.abs().max())
    assert ops.tc_status() == 0


@pytest.mark.parametrize("M", [300, 1041])                           # one CTA a tile, CTA pairs; a last block that leaves from registers
def test_additions_of_subnormal_numbers(M):
    """What blocks add in L2 and what a thread adds itself are the same bits, also where an operand or the sum is subnormal (PTX lets the former flush them)."""
    from quench6k_b200 import ops
    N, K, tiny = 2048, 64, 2.0 ** -126                                  # the smallest normal number
    a, w = torch.zeros(M, K, device=DEV, dtype=torch.bfloat16), torch.zeros(N, K, device=DEV, dtype=torch.bfloat16)
    a[:, 0], w[:, 0], w[::2, 0] = 1, tiny, -tiny
    for shift in (0, 1):
        out = torch.zeros(M * N + 8, device=DEV)[4 + shift:4 + shift + M * N].view(M, N)
        out.fill_(1.5 * tiny)                                           # less tiny: subnormal
        out[:, 1::4] = tiny / 16                                        # subnormal before
        want = out.double() + a.double() @ w.double().T
        ops.gemm_tc(a, w, out=out, accumulate=True)
        assert torch.equal(out.double(), want) and float(out.abs().min()) < tiny
    assert ops.tc_status() == 0
