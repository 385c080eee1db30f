"""The two kernels that carry the FP32 path's prompts: row tiles of attention against the kernel of decode steps, which sums in the same
order, and the FP32 product at the edges of its tiles, for both widths of its copies."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq, Hkv, hd, window, page, dtype", [
    (8, 2, 128, None, 16, torch.float32), (8, 2, 128, 40, 4, torch.float32), (3, 3, 16, 7, 8, torch.float32), (6, 2, 32, None, 4, torch.float32),
    (40, 1, 48, 33, 16, torch.float32),                  # more heads than a tile has rows
    (5, 1, 256, None, 16, torch.float32), (4, 2, 80, 64, 16, torch.bfloat16)])
def test_row_tiles_give_the_bits_of_the_decode_kernel(Hq, Hkv, hd, window, page, dtype):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(hd + Hq)
    q_lens, starts = [37, 1, 9, 70], [0, 90, 31, 64]
    tables, at = [], 0
    n_pages = sum((s + n + page - 1) // page for s, n in zip(starts, q_lens))
    order = torch.randperm(n_pages, generator=g).tolist()
    for s, n in zip(starts, q_lens):
        k = (s + n + page - 1) // page
        tables.append(order[at:at + k])
        at += k
    ctx = helpers.make_context(q_lens, starts, [tables])
    kp, vp = (torch.randn(Hkv, n_pages, page, hd, generator=g).to(dtype).cuda() for _ in range(2))
    for r, (s, n) in enumerate(zip(starts, q_lens)):       # what no step has written
        if (s + n) % page:
            kp[:, tables[r][-1], (s + n) % page:] = vp[:, tables[r][-1], (s + n) % page:] = float("nan")
    q = torch.randn(ctx.T, Hq, hd, generator=g).to(dtype).cuda()
    sinks = torch.randn(Hq, generator=g).cuda()
    whole = ops.attention_generic(q, kp, vp, ctx.block_tables[0], ctx.req_of_token, ctx.positions, window, sinks)
    zero = torch.zeros(1, dtype=torch.int32, device="cuda")
    for t in range(ctx.T):                                  # a request of one token: the decode kernel
        r = int(ctx.req_of_token[t])
        one = ops.attention_generic(q[t:t + 1], kp, vp, ctx.block_tables[0][r:r + 1].contiguous(), zero, ctx.positions[t:t + 1], window, sinks)
        assert torch.equal(one[0], whole[t]), (t, r)
    assert bool(torch.isfinite(whole).all())


@pytest.mark.parametrize("window", [None, 9])
def test_rows_in_any_order(window):
    """Rows of one request whose positions do not ascend: every row sees its own keys."""
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(3)
    Hq, Hkv, hd, page, T = 4, 2, 32, 4, 50
    k, v = (torch.randn(Hkv, 13, page, hd, generator=g).cuda() for _ in range(2))
    q, table = torch.randn(T, Hq, hd, generator=g).cuda(), torch.randperm(13, generator=g).to(torch.int32).cuda()[None]
    orders = [torch.arange(T).flip(0), torch.randperm(T, generator=g), torch.randint(0, T, (T,), generator=g)]
    if window:                                              # two stretches, and no pages between their windows
        table[0, 3:9] = -1
        orders = [torch.cat([torch.arange(11, -1, -1), torch.arange(49, 43, -1)])]
    for order in orders:
        T = len(order)
        pos, req = order.to(torch.int32).cuda(), torch.zeros(T, dtype=torch.int32, device="cuda")
        whole = ops.attention_generic(q[:T], k, v, table, req, pos, window, None)
        for t in range(T):
            assert torch.equal(ops.attention_generic(q[t:t + 1], k, v, table, req[:1], pos[t:t + 1], window, None)[0], whole[t]), (t, int(pos[t]))


@pytest.mark.parametrize("Hq, Hkv, hd", [(8, 8, 64), (8, 2, 128), (12, 2, 32)])          # tiles of 32, 8 and 5 tokens
def test_decoding_requests_beside_a_portion_do_not_wait_for_one_another(Hq, Hkv, hd):
    """A portion beside 32 requests deep in their contexts takes less than three times what it takes beside one of them: each is
    walked by warps of its own, not one after the other in the block of a row tile (32 times)."""
    from quench6k_b200 import ops
    depth, page, portion, most = 2000, 16, 640, 32
    pages = -(-depth // page)
    k, v = (torch.randn(Hkv, pages * (most + 1), page, hd, device="cuda") for _ in range(2))
    table = torch.arange(pages * (most + 1), dtype=torch.int32, device="cuda").view(most + 1, pages)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")

    def took(n):
        q = torch.randn(portion + n, Hq, hd, device="cuda")
        req, pos = i32([0] * portion + list(range(1, n + 1))), i32(list(range(portion)) + [depth - 1] * n)
        run = lambda: ops.attention_generic(q, k, v, table[:n + 1].contiguous(), req, pos, None, None)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(); run(); b.record(); torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])

    one, many = took(1), took(most)
    assert many < 3 * one, (one, many)


@pytest.mark.parametrize("M, N, K, offset", [(1, 1, 1, 0), (64, 64, 32, 0), (65, 63, 33, 0), (3, 130, 36, 0), (130, 70, 100, 1), (17, 257, 1000, 0), (200, 65, 4, 0)])
def test_fp32_product_at_the_edges_of_its_tiles(M, N, K, offset):
    """offset: the operands start off a 16-byte boundary (copies of 4 bytes)."""
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(M * N + K)
    make = lambda *s: torch.randn(offset + s[0] * s[1], generator=g).cuda()[offset:].view(*s)
    a, w, w2 = make(M, K), make(N, K), make(N, K)
    want = (a.double() @ w.double().T)
    bound = K * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T).max()      # a sum of K products in order, each step rounded
    got = ops.gemm_simt(a, w)
    assert float((got.double() - want).abs().max()) <= bound
    assert torch.equal(ops.gemm_simt(a, w, out=got.clone(), accumulate=True), got + got)
    for r in {0, M // 2, M - 1}:                            # a row's result does not depend on its tile
        assert torch.equal(ops.gemm_simt(a[r:r + 1].clone(), w)[0], got[r])
    up = ops.gemm_simt(a, w2)
    both = ops.gemm_simt(a, w, w2=w2)
    assert torch.allclose(both, torch.nn.functional.silu(got) * up, rtol=1e-6, atol=1e-6 * float((got * up).abs().max()))
