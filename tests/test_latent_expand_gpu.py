"""Latent attention of prompt portions on keys and values expanded from the latents they see, against the absorbed form over the same pages and against
float64: portions that end inside a tile, several requests, positions before them, page sizes, a sink, no rotated part; pages and rows nobody may read hold NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _context(lens, starts, table):
    from quench6k_b200.engine.batch import StepContext
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).to(DEV)
    T, R = sum(lens), len(lens)
    return StepContext(T=T, R=R, token_ids=i32([0] * T), positions=i32([s + i for s, n in zip(starts, lens) for i in range(n)]),
                       req_of_token=i32([r for r, n in enumerate(lens) for _ in range(n)]), q_start=i32([sum(lens[:i]) for i in range(R + 1)]), pos_start=i32(starts),
                       slot_ids=i32(list(range(R))), block_tables=[table], logit_rows=i32([]), n_logit_rows=0, q_lens=list(lens), pos_starts=list(starts),
                       slots=list(range(R)), max_context=max(s + n for s, n in zip(starts, lens)), max_q_len=max(lens))


@pytest.mark.parametrize("H, dim, rd, vd, rank, page, lens, starts, sinks", [
    (4, 128, 64, 128, 256, 16, [130], [0], False), (4, 128, 64, 128, 512, 4, [1, 127, 129], [300, 64, 0], True), (3, 64, 32, 64, 128, 64, [200, 65], [63, 1000], False),
    (8, 32, 0, 64, 96, 8, [257], [15], True), (2, 128, 64, 128, 256, 16, [64], [4000], False)])
def test_expanded_against_absorbed_and_float64(monkeypatch, H, dim, rd, vd, rank, page, lens, starts, sinks):
    from quench6k_b200 import ops
    from quench6k_b200.parts.base import MIXERS, LayerCache, Runtime, make_part
    from quench6k_b200.spec import PartSpec
    D, scale = 192, (dim + rd) ** -0.5
    g = torch.Generator().manual_seed(H * rank + lens[0])
    rnd = lambda *s, std=0.05: (torch.randn(s, generator=g) * std).to(torch.bfloat16).to(DEV)
    weights = {"q_proj.weight": rnd(H * (dim + rd), D, std=0.1), "kv_down_proj.weight": rnd(rank + rd, D), "kv_norm.weight": torch.ones(rank), "k_up_proj.weight": rnd(H * dim, rank),
               "v_up_proj.weight": rnd(H * vd, rank), "o_proj.weight": rnd(D, H * vd), "sinks": torch.randn(H, generator=g)}
    pos = PartSpec("rope", {"head_dim": rd, "theta": 10000.0, "rotary_dim": rd}) if rd else PartSpec("none", {"head_dim": 0})
    mixer = make_part(MIXERS, "mixer", PartSpec("latent_attention", dict(num_heads=H, head_dim=dim, rot_dim=rd, v_dim=vd, kv_rank=rank, scale=scale, eps=1e-6, pos=pos, sinks=sinks)),
                      hidden_size=D)
    mixer.bind(lambda name: weights[name], Runtime(torch.device(DEV), torch.bfloat16))
    assert mixer.w_ukv is not None
    blocks = [-(-(s + n) // page) for s, n in zip(starts, lens)]
    order = torch.randperm(sum(blocks) + 3, generator=g).tolist()
    table = torch.full((len(lens), max(blocks)), 0, dtype=torch.int32)
    for r in range(len(lens)):
        table[r, :blocks[r]] = torch.tensor(order[sum(blocks[:r]):sum(blocks[:r + 1])])
    table = table.to(DEV)
    fresh = torch.full((1, sum(blocks) + 3, page, rank + rd), float("nan"), dtype=torch.bfloat16, device=DEV)
    for r, s in enumerate(starts):
        for p in range(s):
            fresh[0, table[r, p // page], p % page] = rnd(rank + rd, std=1.0) if p % 7 == 0 else 0.5
    x = rnd(sum(lens), D, std=1.0)
    results = {}
    for form in (True, False):
        monkeypatch.setattr(type(mixer), "expands", lambda self, ctx, form=form: form)
        k = fresh.clone()
        results[form] = mixer.forward(x, _context(lens, starts, table), LayerCache(0, k, k[..., :rank], page), None, torch.empty((sum(lens), D), device=DEV))
        if results[form].dim() == 3:
            results[form] = results[form].sum(0)
    # float64 over the pages as they were left
    q = (x.double() @ weights["q_proj.weight"].double().T).view(-1, H, dim + rd)
    _, qr = ops.latent_prep(torch.cat([q.float().reshape(len(x), -1), torch.zeros(len(x), rank + rd, device=DEV)], 1).contiguous(), H, dim, rd, rank, None, 1e-6,
                            *(mixer.pos.rotary_table()[:2] if rd else (None, 0)), _context(lens, starts, table).positions, _context(lens, starts, table).req_of_token, table, page, k.clone(),
                            write=False)
    at, outs = 0, []
    for r, (s, n) in enumerate(zip(starts, lens)):
        rows = torch.stack([k[0, table[r, p // page], p % page] for p in range(s + n)]).double()
        seen = torch.arange(s, s + n, device=DEV)[:, None] >= torch.arange(s + n, device=DEV)[None]
        heads = []
        for h in range(H):
            up = lambda name, w: rows[:, :rank] @ weights[name][h * w:(h + 1) * w].double().T
            sc = q[at:at + n, h, :dim] @ up("k_up_proj.weight", dim).T
            if rd:
                sc = sc + qr.view(H, -1, rd)[h, at:at + n].double() @ rows[:, rank:].T
            sc = (sc * scale).masked_fill(~seen, float("-inf"))
            if sinks:
                sc = torch.cat([sc, weights["sinks"][h].double().to(DEV).expand(n, 1)], 1)
            heads.append(torch.softmax(sc, -1)[:, :s + n] @ up("v_up_proj.weight", vd))
        outs.append(torch.cat(heads, -1))
        at += n
    want = torch.cat(outs) @ weights["o_proj.weight"].double().T
    off = {form: float((y.double() - want).norm() / want.norm()) for form, y in results.items()}
    assert off[True] <= 1e-2 and off[True] <= 1.1 * off[False] + 1e-4, off             # bfloat16 operands: about 3e-3, and no more than the form before
    assert ops.tc_status() == 0


def test_the_rule_leaves_recorded_steps_and_decoded_tokens_alone():
    from quench6k_b200.parts.latent_attention import EXPAND_BYTES, LatentAttention
    from types import SimpleNamespace as NS
    part = NS(w_ukv=1, H=16, dim=128, rd=64, vd=128, rank=512)
    takes = lambda lens, starts, replayed=False: LatentAttention.expands(part, NS(replayed=replayed, q_lens=lens, max_q_len=max(lens), pos_starts=starts, plans={}))
    assert takes([2048], [0]) and takes([130], [4096]) and takes([600, 500], [0, 16000])
    assert not takes([2048], [0], True) and not takes([1] * 8, [40] * 8) and not takes([63], [0]) and not takes([130], [16000])
    rows = EXPAND_BYTES // (2 * (512 + 16 * 320))
    assert takes([2048], [rows - 2048 - 64]) and not takes([2048], [rows - 2048 + 64])


def _layer_and_context(lens, starts, page=16, H=4, rank=256):
    from quench6k_b200.parts.base import MIXERS, LayerCache, Runtime, make_part
    from quench6k_b200.spec import PartSpec
    D, dim, rd, vd = 192, 128, 64, 128
    g = torch.Generator().manual_seed(sum(lens))
    rnd = lambda *s, std=0.05: (torch.randn(s, generator=g) * std).to(torch.bfloat16).to(DEV)
    weights = {"q_proj.weight": rnd(H * (dim + rd), D, std=0.1), "kv_down_proj.weight": rnd(rank + rd, D), "kv_norm.weight": torch.ones(rank), "k_up_proj.weight": rnd(H * dim, rank),
               "v_up_proj.weight": rnd(H * vd, rank), "o_proj.weight": rnd(D, H * vd)}
    mixer = make_part(MIXERS, "mixer", PartSpec("latent_attention", dict(num_heads=H, head_dim=dim, rot_dim=rd, v_dim=vd, kv_rank=rank, scale=192 ** -0.5, eps=1e-6,
                                                                         pos=PartSpec("rope", {"head_dim": rd, "theta": 10000.0, "rotary_dim": rd}))), hidden_size=D)
    mixer.bind(lambda name: weights[name], Runtime(torch.device(DEV), torch.bfloat16))
    blocks = [-(-(s + n) // page) for s, n in zip(starts, lens)]
    table = torch.zeros((len(lens), max(blocks)), dtype=torch.int32)
    for r in range(len(lens)):
        table[r, :blocks[r]] = torch.arange(sum(blocks[:r]), sum(blocks[:r + 1]))
    k = rnd(1, sum(blocks), page, rank + rd, std=1.0)
    x, out = rnd(sum(lens), D, std=1.0), torch.empty((sum(lens), D), device=DEV)
    ctx = _context(lens, starts, table.to(DEV))
    run = lambda ctx: mixer.forward(x, ctx, LayerCache(0, k, k[..., :rank], page), None, out)
    return mixer, ctx, run


def test_a_new_context_uploads_nothing_for_the_rows_it_expands():
    """What an expanding step needs of its requests is on the device already: the tiles of its queries are all that goes up."""
    import copy

    from torch.utils._python_dispatch import TorchDispatchMode
    mixer, ctx, run = _layer_and_context([300, 1, 130], [1000, 64, 0])

    class Uploads(TorchDispatchMode):
        count = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            if func in (torch.ops.aten._to_copy.default, torch.ops.aten.copy_.default):
                src = args[1] if func is torch.ops.aten.copy_.default else args[0]
                Uploads.count += out.is_cuda and not src.is_cuda
            return out

    assert mixer.expands(ctx)
    run(ctx)                                                            # tensors that the process keeps are made
    fresh = copy.copy(ctx)
    fresh.plans, fresh.made = {}, set()
    with Uploads():
        run(fresh)
    assert Uploads.count <= 1


@pytest.mark.parametrize("lens, starts", [([64], [0]), ([1, 63, 65, 200], [128, 1, 0, 500]), ([1] * 33 + [70] + [2] * 40, [9 * i for i in range(74)])])
def test_rows_and_blocks_of_every_request(lens, starts):
    """Requests side by side, more than a warp looks at together: every row is the latent of its request and position, the rows between are zeros."""
    from quench6k_b200 import ops
    H, dim, rd, vd, rank, page = 2, 32, 8, 64, 64, 4
    reach = [s + n for s, n in zip(starts, lens)]
    need = [-(-c // page) for c in reach]
    g = torch.Generator().manual_seed(len(lens))
    order = torch.randperm(sum(need), generator=g, dtype=torch.int32)
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    for r in range(len(lens)):
        table[r, :need[r]] = order[sum(need[:r]):sum(need[:r + 1])]
    pages = torch.randn(1, sum(need), page, rank + rd, generator=g).to(torch.bfloat16)
    w = (torch.randn(H * (dim + vd), rank, generator=g) * 0.1).to(torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    k, v, blocks = ops.latent_expanded(pages.to(DEV), reach, i32([sum(lens[:i]) for i in range(len(lens) + 1)]), i32(starts), table.to(DEV), w.to(DEV), H, dim, rd)
    counts = [-(-c // 64) for c in reach]
    assert k.shape == (H, sum(counts), 64, dim + rd) and v.shape == (H, sum(counts), 64, vd)
    first = [sum(counts[:r]) for r in range(len(lens))]
    assert blocks.tolist() == [[f + min(i, n - 1) for i in range(max(counts))] for f, n in zip(first, counts)]
    want = torch.zeros(sum(counts) * 64, rank + rd)
    for r, c in enumerate(reach):
        for p in range(c):
            want[first[r] * 64 + p] = pages[0, table[r, p // page], p % page].float()
    for h in range(H):
        up = (want[:, :rank].double() @ w[h * (dim + vd):(h + 1) * (dim + vd)].double().T)
        assert torch.equal(k[h, :, :, dim:].reshape(-1, rd).float().cpu(), want[:, rank:])
        got = torch.cat([k[h, :, :, :dim], v[h]], -1).reshape(-1, dim + vd).double().cpu()
        # a sum of 64 products of FP32, rounded to bfloat16
        assert bool(((got - up).abs() <= up.abs() * 2.0 ** -8 + 1e-5).all())
    assert ops.tc_status() == 0


def test_where_the_expanded_rows_find_no_memory_the_step_is_absorbed(monkeypatch):
    """The step then gives the bits of the absorbed form, which needs no such rows.  The failure is the host's: the call that allocates them raises."""
    from quench6k_b200 import ops
    mixer, ctx, run = _layer_and_context([300], [100])
    assert mixer.expands(ctx)

    def no_room(*a, **k):
        raise torch.OutOfMemoryError("out of memory, says the test")

    with monkeypatch.context() as m:
        m.setattr(ops, "latent_expanded", no_room)
        got = run(ctx).clone()
    absorbed = _layer_and_context([300], [100])
    monkeypatch.setattr(type(absorbed[0]), "expands", lambda self, ctx: False)
    assert torch.equal(got, absorbed[2](absorbed[1])) and ops.tc_status() == 0
