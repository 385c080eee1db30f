"""Which steps of portions of more than 64 tokens the selective scan walks in one pass, and which in segments: the form measured to be the faster one (us, bfloat16:
one pass, segments).  No GPU: the rule reads sizes."""
import pytest

from quench6k_b200 import ops


@pytest.mark.parametrize("lens, C, N, one_pass", [
    ([8192], 640, 16, False),                    # 362, 230
    ([8192], 768, 16, False),                    # 365, 264
    ([8192], 1024, 16, False),                   # 395, 364
    ([4096], 640, 16, False),                    # 184, 133
    ([4096], 768, 16, False),                    # 184, 150
    ([2048], 640, 16, True),                     # 94, 100
    ([4096], 1024, 16, True),                    # 185, 191
    ([2048], 1024, 16, True),                    # 94, 113
    ([2048], 4096, 16, True),                    # 146, 349
    ([4096], 2048, 9, True),                     # 202, 344
    ([8192], 2048, 9, True),                     # 403, 667
    ([1024], 640, 16, True),                     # 49, 86
    ([509], 1536, 9, True),                      # 29, 84
    ([682] * 3, 640, 16, True),                  # 36, 94
    ([256], 512, 16, False), ([2048], 64, 16, False)])
def test_one_pass_or_segments(lens, C, N, one_pass):
    segments = max(-(-n // 64) for n in lens)
    assert bool(ops.library().q6k_selective_scan_lanes_taken(sum(lens), len(lens), C, N, segments)) == one_pass
