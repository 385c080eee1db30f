"""Attention of decoded tokens side by side with that of a step's prompt portions (the launch before it): the same bits as one after the other,
with inputs written just before and results read just after, for few and for more prompt tiles than SMs."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("q_lens,Hkv,G,ps,window", [([300, 1, 1, 2], 2, 8, 16, None), ([1, 129, 700, 1], 4, 4, 64, None), ([5000, 1, 1], 8, 8, 32, 100),
                                                    ([200, 9, 1], 1, 1, 16, None), ([260, 1], 8, 2, 128, 300)])
def test_side_by_side_as_in_turn(q_lens, Hkv, G, ps, window):
    from quench6k_b200 import ops
    hd, Hq, R = 128, Hkv * G, len(q_lens)
    g = torch.Generator(device=DEV).manual_seed(sum(q_lens))
    starts = [0 if n > 8 else 900 + 333 * i for i, n in enumerate(q_lens)]
    need = [-(-(s + n) // ps) for s, n in zip(starts, q_lens)]
    tables = [list(range(sum(need[:i]), sum(need[:i + 1]))) for i in range(R)]
    bt = torch.tensor([t + [-1] * (max(need) - len(t)) for t in tables], dtype=torch.int32, device=DEV)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    kp, vp, T = r(Hkv, sum(need), ps, hd), r(Hkv, sum(need), ps, hd), sum(q_lens)
    ctx = helpers.make_context(q_lens, starts, [tables])
    tile = ops.attention_tc_tile_tokens(G)
    cut = tile // 2
    count, _, _, most, _ = ctx.short_requests(cut)
    assert count
    rows = ops.attention_mma_tile_rows(hd, G, most)
    long0, longn, _ = ctx.query_tile_pairs(tile, False, more_than=cut)
    tok0, ntok, n_tiles = ctx.query_tiles(rows // G, cut)
    plan = ops.attention_plan(ctx.positions, ctx.req_of_token, tok0, ntok, window, ops.attention_mma_resident_ctas(hd, rows) // Hkv, min_per=2)
    queries, results = [r(T, Hq, hd) for _ in range(4)], {}
    q = torch.empty_like(queries[0])
    for beside in (False, True):
        read = []
        for i in range(24):
            out = torch.full((T, Hq * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
            q.copy_(queries[i % 4])
            ops.attention_tc(q, kp, vp, bt, ctx.req_of_token, ctx.positions, long0, longn, window, None, out=out)
            ops.attention_mma(q, kp, vp, bt, ctx.req_of_token, ctx.positions, tok0, ntok, rows, window, None, out=out, plan=plan, plan_is_old=True, beside_tc=beside)
            read.append(out.clone())
        results[beside] = read
    assert ops.tc_status() == 0 and not any(bool(torch.isnan(x).any()) for x in results[False])
    assert all(torch.equal(x, y) for x, y in zip(results[False], results[True]))


# one and many prompt tiles an SM; the decoding requests' keys in parts (a merge lies between) and whole (nothing does)
@pytest.mark.parametrize("q_lens,Hkv,G,parts", [([300, 1, 1], 2, 8, False), ([5000, 1, 1], 8, 8, False), ([5000, 1, 1], 8, 8, True), ([1, 2100, 1300, 1], 4, 4, False)])
def test_the_next_product_finds_both_results(q_lens, Hkv, G, parts):
    """The product that follows waits for its direct predecessor alone, the decoding requests' attention, and fetches its weights before: it must still find every
    row of the prompt portions, whose attention may end last."""
    from quench6k_b200 import ops
    hd, Hq, R, ps, N = 128, Hkv * G, len(q_lens), 16, 512
    g = torch.Generator(device=DEV).manual_seed(sum(q_lens))
    starts = [0 if n > 8 else 200 + 33 * i for i, n in enumerate(q_lens)]
    need = [-(-(s + n) // ps) for s, n in zip(starts, q_lens)]
    tables = [list(range(sum(need[:i]), sum(need[:i + 1]))) for i in range(R)]
    bt = torch.tensor([t + [-1] * (max(need) - len(t)) for t in tables], dtype=torch.int32, device=DEV)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    kp, vp, T, w = r(Hkv, sum(need), ps, hd), r(Hkv, sum(need), ps, hd), sum(q_lens), r(N, Hq * hd)
    ctx = helpers.make_context(q_lens, starts, [tables])
    tile = ops.attention_tc_tile_tokens(G)
    cut = tile // 2
    rows = ops.attention_mma_tile_rows(hd, G, ctx.short_requests(cut)[3])
    long0, longn, _ = ctx.query_tile_pairs(tile, False, more_than=cut)
    tok0, ntok, n_tiles = ctx.query_tiles(rows // G, cut)
    plan = ops.attention_plan(ctx.positions, ctx.req_of_token, tok0, ntok, None, ops.attention_mma_resident_ctas(hd, rows) // Hkv if parts else n_tiles, min_per=2)
    assert (plan[0].shape[0] > n_tiles) == parts
    q, results = r(T, Hq, hd), {}
    for beside in (False, True):
        read = []
        for i in range(8):
            out = torch.full((T, Hq * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
            ops.attention_tc(q, kp, vp, bt, ctx.req_of_token, ctx.positions, long0, longn, None, None, out=out)
            ops.attention_mma(q, kp, vp, bt, ctx.req_of_token, ctx.positions, tok0, ntok, rows, None, None, out=out, plan=plan, plan_is_old=True, beside_tc=beside)
            read.append(ops.gemm_tc(out, w))
        results[beside] = read
    assert ops.tc_status() == 0 and not any(bool(torch.isnan(x).any()) for x in results[False])
    assert all(torch.equal(x, y) for x, y in zip(results[False], results[True]))
