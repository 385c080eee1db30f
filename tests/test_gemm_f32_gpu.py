"""FP32 products from three bfloat16 parts of each operand, at the edges of the tiles (32 and 64 tokens, 128 and 64 weight rows) and of the
chunks of 64 k, against float64; rows of groups; operands that are infinite, not a number or near the ends of the range."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _bound(a, w):
    """The parts left out and the accumulator's truncation, 2^-22 of the sum of the products' sizes; a rounding for each chunk of 64."""
    return (2.0 ** -22 + -(-a.shape[1] // 64) * 2.0 ** -24) * float((a.double().abs() @ w.double().abs().T).max())


@pytest.mark.parametrize("M, N, K", [(31, 127, 64), (32, 128, 63), (33, 129, 65), (63, 64, 128), (64, 65, 129), (65, 63, 1000), (129, 256, 68), (200, 1, 4), (1, 300, 2048)])
def test_against_float64(M, N, K):
    from quench6k_b200 import ops
    a, w, w2 = _t(M, K), _t(N, K, seed=1), _t(N, K, seed=2)
    ref, up = a.double() @ w.double().T, a.double() @ w2.double().T
    got = ops.gemm_simt(a, w)
    assert float((got.double() - ref).abs().max()) <= _bound(a, w)
    assert torch.equal(ops.gemm_simt(a, w, out=got.clone(), accumulate=True), got + got)
    gate = ops.gemm_simt(a, w, w2=w2)
    want = torch.nn.functional.silu(ref) * up
    assert float((gate.double() - want).abs().max()) <= 2e-6 * float(want.abs().max())
    assert ops.tc_status() == 0


def test_rows_of_groups_have_the_bits_of_a_product_of_their_own():
    from quench6k_b200 import ops
    sizes, N, K = [1, 0, 63, 64, 65, 130], 200, 260
    offsets = torch.tensor([sum(sizes[:i]) for i in range(len(sizes) + 1)], dtype=torch.int32, device="cuda")
    rows = sum(sizes)
    a, w = _t(rows + 5, K), _t(len(sizes), N, K, seed=1)
    order = torch.randperm(rows + 5, generator=torch.Generator().manual_seed(3))[:rows].to(torch.int32).cuda()
    got = ops.gemm_simt(a, w, a_rows=order, groups=ops.tile_list(offsets, rows, ops.simt_tile_rows()), rows=rows)
    for g, n in enumerate(sizes):
        if n:
            at = int(offsets[g])
            assert torch.equal(got[at:at + n], ops.gemm_simt(a[order[at:at + n].long()].contiguous(), w[g].contiguous()))


@pytest.mark.parametrize("K", [64, 70, 200])
def test_operands_that_are_not_finite_or_near_the_ends_of_the_range(K):
    from quench6k_b200 import ops
    a, w = _t(70, K), _t(130, K, seed=1)
    inf, nan = float("inf"), float("nan")
    a[3, 5], a[4, 6], a[5, 7], w[9, 8] = inf, -inf, nan, inf
    a[6], w[10] = 0.0, 0.0
    a[6, 0], w[10, 0] = 3.4e38, 0.5                              # beyond bfloat16's largest
    a[7], w[11] = 1e-25, 1e-12
    ref = a.double() @ w.double().T
    got = ops.gemm_simt(a, w)
    want = ref.float()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    fine = torch.isfinite(want)
    assert float(got[6, 10]) == float(want[6, 10])
    size = torch.nan_to_num(a.double()).abs() @ torch.nan_to_num(w.double()).abs().T
    assert bool(((got.double() - ref).abs()[fine] <= (2.0 ** -22 + K * 2.0 ** -24) * size[fine] + 2.0 ** -149).all())
