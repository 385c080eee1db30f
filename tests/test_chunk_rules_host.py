"""Which steps the retention and delta layers walk in chunks: where that was measured to be the faster form.  No GPU: the rules read sizes."""
import pytest

from quench6k_b200 import ops


@pytest.mark.parametrize("lens, H, dk, chunked", [
    ([65], 16, 128, False), ([256], 16, 128, False), ([512], 16, 128, True), ([1024], 16, 128, True), ([130] + [1] * 32, 16, 128, False), ([65] + [1], 16, 128, False),
    ([512] + [1] * 8, 16, 128, True), ([200] * 8, 16, 128, False), ([1021, 851, 681], 16, 128, True), ([1024] * 2, 16, 64, False), ([512], 16, 64, True),
    ([400], 8, 256, False), ([1024], 8, 256, True), ([64] * 4, 16, 128, False), ([], 16, 128, False)])
def test_retention(lens, H, dk, chunked):
    assert ops.retention_chunks(lens, H, dk, dk) == chunked


@pytest.mark.parametrize("lens, H, chunked", [          # us, walked and by chunks on tensor cores
    ([1021] * 3, 16, True),                              # 204, 90
    ([300] * 3, 16, True),                               # 64, 40
    ([400] * 3, 8, True),                                # 60, 37
    ([2048], 8, True),                                   # 217, 37
    ([512] + [1] * 32, 16, True),                        # 120, 68
    ([320], 16, False),                                  # 37, 35
    ([128], 8, False),                                   # 17, 35
    ([65] + [1] * 32, 8, False)])                        # 21, 43
def test_retention_on_tensor_cores(lens, H, chunked):
    assert ops.retention_chunks(lens, H, 128, 128) == chunked


@pytest.mark.parametrize("lens, chunked", [([65], False), ([130], True), ([128] + [1] * 32, False), ([2048], True), ([512] + [1] * 32, True)])
def test_delta(lens, chunked):
    assert ops.gated_delta_chunks(max(lens), 4, 16, 128, 128, lens) == chunked
