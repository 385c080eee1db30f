"""Which steps the flexible attention layers give to the tcgen05 kernel: those, and only those, that the mma.sync kernel would run otherwise
(its query and weights are rounded alike), with pages that copies of whole boxes can address.  No GPU: the rule reads sizes and strides."""
import pytest
import torch

from quench6k_b200 import ops


def _pages(heads, page, width, n=3):
    return torch.empty((heads, n, page, width), dtype=torch.bfloat16)


@pytest.mark.parametrize("H, Hkv, da, db, dv, page", [(16, 1, 512, 64, 512, 16), (32, 1, 512, 64, 512, 16), (8, 1, 256, 64, 256, 8), (16, 4, 0, 128, 128, 16), (32, 1, 0, 64, 64, 128)])
def test_what_the_mma_kernel_would_run(H, Hkv, da, db, dv, page):
    k = _pages(Hkv, page, da + db)
    v = k[..., :dv] if da else _pages(Hkv, page, dv)
    tokens = 128 // (H // Hkv)
    wide = lambda n, k=k, v=v, scale=0.1: ops.attention_flex_wide(n, H, da, db, False, k, v, scale)
    assert wide(tokens) == tokens and wide((tokens + 1) // 2) == tokens and wide(tokens // 2 - 1) == 0
    assert wide(1) == 0                                                # a step of single tokens, whatever the group
    assert wide(tokens, scale=0.0) == 0 and wide(tokens, k=k.float(), v=v.float()) == 0
    if Hkv > 1:                                                        # heads that do not follow one another
        apart = torch.empty((3, Hkv, page, db), dtype=torch.bfloat16).transpose(0, 1)
        assert wide(tokens, k=apart) == 0
    off = torch.empty(k.numel() + 1, dtype=torch.bfloat16)[1:].view(k.shape)
    assert wide(tokens, k=off, v=off[..., :dv] if da else v) == 0      # pages that do not start on 16 bytes


@pytest.mark.parametrize("H, Hkv, da, db, dv", [
    (33, 1, 512, 64, 512), (64, 1, 512, 64, 512), (128, 1, 512, 64, 512), (128, 2, 0, 128, 128),        # a key head of more than 32 query heads
    (12, 1, 64, 8, 64), (6, 2, 0, 24, 64), (16, 4, 0, 72, 128),                                         # key rows that are no multiple of 16
    (8, 2, 0, 128, 576), (8, 2, 0, 128, 1024)])                                                         # values no decode kernel takes
def test_what_runs_on_cuda_cores_stays_there(H, Hkv, da, db, dv):
    k = _pages(Hkv, 16, da + db)
    v = k[..., :dv] if da else _pages(Hkv, 16, dv)
    assert not ops.attention_flex_mma_supported(H, Hkv, da + db, dv, k.stride(2), v.stride(2), db, bool(da))
    for n in (1, 2, 64, 2048):
        assert ops.attention_flex_wide(n, H, da, db, False, k, v, 0.1) == 0


@pytest.mark.parametrize("lens, context, taken", [
    ([64] + [1] * 32, 4000, False),                  # four key ranges on mma.sync, none on tcgen05
    ([128] + [1] * 32, 4000, True), ([40] + [1] * 4, 4000, True), ([2048] + [1] * 32, 4000, True), ([64] + [1] * 32, 200, True), ([64], 30000, True)])
def test_short_portions_beside_deep_requests(lens, context, taken):
    k = _pages(1, 16, 576)
    assert (ops.attention_flex_wide(max(lens), 16, 512, 64, False, k, k[..., :512], 0.1, lens, context) > 0) == taken
    assert ops.attention_flex_wide(max(lens), 16, 512, 64, False, k, k[..., :512], 0.1, lens, context, chunk=64) > 0        # chunks are never split


def test_windows_are_not_cut_into_ranges_of_the_whole_context():
    assert ops._wide_ranges(20, 16000, 512, 32) == (1, 0) and ops._wide_ranges(20, 16000, None, 32)[0] > 1 and ops._wide_ranges(20, 16000, 8192, 32)[0] > 1
