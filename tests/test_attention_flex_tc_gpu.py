"""The tcgen05 flexible attention kernel against the CUDA-core kernel on the same data: every layout it is given by the latent, the
mixed-heads and the difference attention layers, at the edges of its tiles (64 keys, 128 / G tokens), with one key range and with
several, pages in shuffled order, and what no step has written filled with NaN."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


def _pages(q_lens, starts, page, heads, width, g, order, n_pages):
    """Pages whose unwritten places hold NaN, as a fresh pool might."""
    k = torch.full((heads, n_pages, page, width), float("nan"), dtype=torch.bfloat16)
    at = 0
    for s, n in zip(starts, q_lens):
        blocks = (s + n + page - 1) // page
        rows = torch.full((heads, blocks * page, width), float("nan"), dtype=torch.bfloat16)
        rows[:, :s + n] = (torch.randn(heads, s + n, width, generator=g) * 0.5).to(torch.bfloat16)
        k[:, order[at:at + blocks]] = rows.view(heads, blocks, page, width)
        at += blocks
    return k.cuda()


@pytest.mark.parametrize("H, Hkv, da, db, dv, shared, page, extra", [
    (16, 1, 512, 64, 512, True, 16, {}),                                  # the widest latent: part of Q in tensor memory, two CTAs a tile
    (16, 1, 512, 0, 512, True, 64, {}),                                   # no rotated part: every chunk is a value chunk of some CTA
    (8, 1, 256, 64, 256, True, 8, {"sinks": True}),
    (12, 1, 64, 8, 64, True, 32, {"window": 100}),                        # a key row that ends inside a chunk, heads that do not divide 128
    (8, 4, 0, 128, 128, False, 16, {"window": 70, "sinks": True}),        # values of their own, two CTAs to an SM
    (3, 1, 0, 192, 320, False, 16, {"chunk": 37}),                        # not taken (values of 320): the rule has to say so
    (8, 2, 0, 64, 192, False, 128, {"chunk": 96}),                        # pages wider than a key tile
    (16, 8, 0, 64, 128, False, 16, {"chunk": 200, "softcap": 30.0, "maps": 2, "out_f32": True}),
    (16, 4, 0, 128, 128, False, 16, {"chunk": 150, "talk": True}),        # 512 value columns: two CTAs
    (6, 2, 0, 24, 64, False, 16, {"chunk": 64, "talk": True}),
])
def test_against_the_cuda_core_kernel(H, Hkv, da, db, dv, shared, page, extra):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H * 1000 + da + dv)
    per = 128 // (H // Hkv)                                                # tokens of a wide tile
    q_lens, starts = [per, 1, 2 * per + 3, 64, max(1, per // 2)], [0, 1001, 129, 64 - 1, 640]
    n_pages = sum((s + n + page - 1) // page for s, n in zip(starts, q_lens))
    order = torch.randperm(n_pages, generator=g).tolist()
    tables, at = [], 0
    for s, n in zip(starts, q_lens):
        k = (s + n + page - 1) // page
        tables.append(order[at:at + k])
        at += k
    ctx = helpers.make_context(q_lens, starts, [tables])
    maps = extra.get("maps", 1)
    k_pages = _pages(q_lens, starts, page, Hkv, da + db, g, order, n_pages)
    v_pages = k_pages[..., :dv] if shared else _pages(q_lens, starts, page, Hkv // maps, dv, g, order, n_pages)
    qa = torch.randn(H * ctx.T, da, generator=g).to(torch.bfloat16).cuda() if da else None
    qb = torch.randn(H * ctx.T, db, generator=g).to(torch.bfloat16).cuda() if db else None
    talk = torch.randn(H, H, generator=g).cuda() if extra.get("talk") else None
    common = dict(window=extra.get("window"), chunk=extra.get("chunk"), out_head_major=shared, softcap=extra.get("softcap", 0.0), maps=maps,
                  out_f32=extra.get("out_f32", False), talk=talk, sinks=torch.randn(H, generator=g).cuda() if extra.get("sinks") else None)
    scale = (da + db) ** -0.5
    tokens = ops.attention_flex_wide_tokens(max(q_lens), H, Hkv, da, db, dv, talk is not None, shared, page, scale)
    if dv == 320:
        assert tokens == 0
        return
    assert tokens == per
    assert ops.attention_flex_wide_tokens(1, 2 * Hkv, Hkv, da, db, dv, False, shared, page, scale) == 0     # decode steps stay where they were
    args = (qa, qb, shared, k_pages, v_pages, ctx.block_tables[0], ctx.req_of_token, ctx.positions, H, scale)
    clean = [torch.nan_to_num(t) for t in (k_pages, v_pages)]
    want = ops.attention_flex(qa.float() if da else None, qb, shared, clean[0], clean[0][..., :dv] if shared else clean[1], *args[5:], **common)
    longest = max(s + n for s, n in zip(starts, q_lens))
    for max_context in (0, longest):                                       # 0: one key range; else fixed ranges, merged
        got = ops.attention_flex(*args, wide_tiles=ctx.query_tiles(tokens), max_context=max_context, **common)
        assert got.dtype == want.dtype and got.shape == want.shape and bool(torch.isfinite(got).all())
        # two bfloat16 results of the same bfloat16 operands: half an ulp each (2^-9 of a value); weights carry 16 bits, their
        # exponentials 21
        diff, size = (got.float() - want.float()).abs().max().item(), want.float().abs().max().item()
        rel = ((got.float() - want.float()).norm() / want.float().norm()).item()
        assert diff < 1e-2 * size and rel < 4e-3, f"max_context {max_context}: {diff / size:.3e}, {rel:.3e}"
    assert ops.tc_status() == 0


def test_every_row_sees_its_last_value_product():
    """From one key tile to seven, two CTAs to an SM, launched again and again: a row that comes late to ask for the last product
    has to see that it is done (a wait by a parity two products old would run out, leave a status and store nothing)."""
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(5)
    H, Hkv, hd, page = 8, 2, 64, 16
    q_lens, starts = [32] * 48, [(64 * i) % 448 for i in range(48)]
    n_pages = sum((s + n + page - 1) // page for s, n in zip(starts, q_lens))
    order, tables, at = torch.randperm(n_pages, generator=g).tolist(), [], 0
    for s, n in zip(starts, q_lens):
        tables.append(order[at:at + (s + n + page - 1) // page])
        at += len(tables[-1])
    ctx = helpers.make_context(q_lens, starts, [tables])
    k, v = (_pages(q_lens, starts, page, Hkv, hd, g, order, n_pages) for _ in range(2))
    q = torch.randn(H * ctx.T, hd, generator=g).to(torch.bfloat16).cuda()
    tiles = ctx.query_tiles(ops.attention_flex_wide_tokens(32, H, Hkv, 0, hd, hd, False, False, page, 0.125))
    run = lambda: ops.attention_flex(None, q, False, k, v, ctx.block_tables[0], ctx.req_of_token, ctx.positions, H, 0.125, wide_tiles=tiles, max_context=512)
    first = run()
    assert bool(torch.isfinite(first).all())
    for _ in range(200):
        assert torch.equal(run(), first)
    assert ops.tc_status() == 0


@pytest.mark.parametrize("H, Hkv", [(96, 8), (112, 8)])                   # a mixing matrix that fits 48 KB, or does not
def test_mixed_heads_of_any_number(H, Hkv):
    from quench6k_b200 import ops
    g = torch.Generator().manual_seed(H)
    T, hd, dv, page, chunk = 21, 64, 64, 16, 8
    ctx = helpers.make_context([T], [0], [[[1, 0]]])
    k, v = (torch.randn(Hkv, 2, page, n, generator=g).to(torch.bfloat16).cuda() for n in (hd, dv))
    q = torch.randn(T * H, hd, generator=g).to(torch.bfloat16).cuda()
    talk = (torch.randn(H, H, generator=g) * H ** -0.5).cuda()
    run = lambda **tiles: ops.attention_flex(None, q, False, k, v, ctx.block_tables[0], ctx.req_of_token, ctx.positions, H, 0.125, chunk=chunk, talk=talk, max_context=T, **tiles)
    pos = torch.arange(T, device="cuda")
    seen = (pos[:, None] >= pos) & (pos[:, None] // chunk == pos // chunk)
    rows = [x[:, [1, 0]].reshape(Hkv, -1, x.shape[-1])[:, :T].double().repeat_interleave(H // Hkv, 0) for x in (k, v)]
    w = torch.softmax((torch.einsum("thd,hjd->htj", q.view(T, H, hd).double(), rows[0]) * 0.125).masked_fill(~seen, float("-inf")), -1)
    want = torch.einsum("hgtj,hjd->thd", talk.double()[:, :, None, None] * w[None], rows[1]).reshape(T, H * dv)
    for got in (run(tiles=ctx.query_tiles(ops.attention_flex_tile_tokens(H, Hkv))), run(wide_tiles=ctx.query_tiles(ops.attention_flex_tc_tile_tokens(H, Hkv)))):
        assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8          # a rounding to bfloat16 (2^-9), weights of 16 bits
