"""The row kernels that put queries, keys and values in place 16 bytes at a time, against the kernels they stand in for, which run when an
operand does not start on 16 bytes (or a head is not a power of two): all head widths, biases, norms, rotations, slices."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _at(t, aligned):
    """t as rows that start on 16 bytes, or 4 bytes behind that."""
    buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = buf[:-1] if aligned else buf[1:]
    view.copy_(t.reshape(-1))
    return view.view(t.shape)


@pytest.mark.parametrize("Hq, Hkv, hd, vd, Hv, rd, bias, norm, same", [
    (8, 2, 64, 128, 2, 0, True, True, False), (4, 1, 128, 128, None, 64, False, True, False), (8, 8, 16, 32, 4, 16, True, False, False),
    (2, 2, 64, 64, None, 32, False, False, True), (40, 4, 128, 64, 6, 128, True, True, False)])
def test_rows_against_a_warp_per_head(Hq, Hkv, hd, vd, Hv, rd, bias, norm, same):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(Hq * hd + vd)
    T, page, P = 21, 4, 12
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    width = Hq * hd + Hkv * hd + (0 if same else (Hv or Hkv) * vd)
    x, b = rnd(T, width), rnd(width) if bias else None
    qn, kn = (rnd(hd), rnd(hd)) if norm else (None, None)
    rot = (torch.rand(rd // 2, generator=g).cuda(), rd, Hq == 8) if rd else None
    results = []
    for aligned in (True, False):
        k = torch.zeros(Hkv, P, page, hd, dtype=torch.bfloat16, device="cuda")
        v = torch.zeros(Hv or Hkv, P, page, vd, dtype=torch.bfloat16, device="cuda")
        q = ops.qkv_pages(_at(x, aligned), Hq, Hkv, hd, vd, qn, kn, 1e-6, rot, i32(list(range(3, 3 + T))), i32([0] * T), i32([[5, 3, 0, 7, 1, 11]]), page, k, v,
                          torch.bfloat16, v_heads=Hv, bias=b, values_are_keys=same, value_norm=same)
        results.append((q, k, v))
    for one, other in zip(*results):
        # sums of squares in another order: an FP32 rounding, which may move a value over a bfloat16 boundary
        assert torch.allclose(one.float(), other.float(), rtol=2.0 ** -7, atol=1e-6)
        assert (one != other).float().mean() < 0.01


@pytest.mark.parametrize("H, dim, rd, rank, turn, near, write", [(16, 128, 64, 96, 64, False, True), (3, 32, 16, 40, 8, True, True), (5, 4, 4, 8, 0, False, False), (2, 64, 0, 24, 0, False, True)])
def test_latent_rows_against_a_block_per_head(H, dim, rd, rank, turn, near, write):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H * dim + rank)
    T, page, P = 9, 4, 6
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    x = torch.randn(T, H * (dim + rd) + rank + rd, generator=g).cuda()
    w, freq = torch.randn(rank, generator=g).cuda(), torch.rand(max(1, turn // 2), generator=g).cuda()
    results = []
    for aligned in (True, False):
        pages = torch.zeros(1, P, page, rank + rd, dtype=torch.bfloat16, device="cuda")
        qn, qr = ops.latent_prep(_at(x, aligned), H, dim, rd, rank, w, 1e-6, freq if turn else None, turn, i32(list(range(5, 5 + T))), i32([0] * T), i32([[2, 0, 5, 1]]), page,
                                 pages, neighbours=near, write=write)
        results.append((qn, qr, pages))
    for one, other in zip(results[0][:2], results[1][:2]):
        assert torch.equal(one, other)
    assert torch.allclose(results[0][2].float(), results[1][2].float(), rtol=2.0 ** -7, atol=1e-6)        # the latent's squares in another order
    maps = torch.randn(T, H, 2, dim, generator=g).cuda()
    one, other = (ops.map_difference(_at(maps.view(T, -1), a), H, dim, 0.4, 1e-6, 0.6, torch.bfloat16) for a in (True, False))
    assert torch.allclose(one.float(), other.float(), rtol=2.0 ** -7, atol=1e-6)
    src = torch.randn(H * T, dim, generator=g).cuda()
    assert torch.equal(ops.heads_to_rows(_at(src, True), H, torch.bfloat16), ops.heads_to_rows(_at(src, False), H, torch.bfloat16))


@pytest.mark.parametrize("H, dk, rd, scale, dv", [(16, 128, 128, 0.3, 128), (3, 24, 8, 1.0, 20), (40, 64, 32, 0.5, 256), (1, 8, 8, 2.0, 4)])
def test_recurrent_rows_against_four_bytes_at_a_time(H, dk, rd, scale, dv):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H * dk + dv)
    T, width = 7, 4 + 2 * H * dk + H * dv
    p, o, w = (torch.randn(*s, generator=g).cuda() for s in ((T, width), (T, H * dv), (dv,)))
    rot = (torch.rand(rd // 2, generator=g).cuda(), rd, False)
    pos = torch.arange(11, 11 + T, dtype=torch.int32, device="cuda")
    turned = []
    for aligned in (True, False):
        x = _at(p, aligned)
        ops.retention_prep(x, H, dk, 4, 4 + H * dk, rot, scale, pos)
        turned.append(x)
    assert torch.allclose(*turned, rtol=1e-6, atol=1e-6 * float(p.abs().max()))          # the same products; their sums may be contracted otherwise
    for dtype in (torch.bfloat16, torch.float32):
        one, other = (ops.delta_out(_at(o, a), _at(p, a), 4 + 2 * H * dk, _at(w, a), 1e-6, H, dv, dtype) for a in (True, False))
        assert torch.allclose(one.float(), other.float(), rtol=2.0 ** -7 if dtype == torch.bfloat16 else 1e-6, atol=1e-6)       # squares in another order
