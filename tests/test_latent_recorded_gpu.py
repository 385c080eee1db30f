"""A prompt portion through a latent attention layer takes one form, whether its shape comes for the first time (an eager pass), is recorded or replayed:
three requests with the same tokens get the same logits, bit for bit."""
import pytest
import torch

import helpers
import pedotar_configs
import pedotar_helpers

pytestmark = pytest.mark.gpu


# portions whose end fills the recording's table width (64 pages), so that every pass splits its keys alike
@pytest.mark.parametrize("page, start, portion", [(16, 894, 130), (16, 960, 64), (4, 0, 256)])
def test_a_portion_keeps_its_bits_when_its_shape_comes_again(tmp_path, page, start, portion):
    from quench6k_b200 import ops
    from quench6k_b200.engine import StepEntry
    from quench6k_b200.engine.runner import ModelRunner
    layer = pedotar_configs.latent(8, 128, 64, 128, 256, 10000.0, 192 ** -0.5)
    pedotar_helpers.make_folder(str(tmp_path), pedotar_configs.one_layer(layer, width=256, page=page), seed=5)
    runner = ModelRunner.from_folder(str(tmp_path), num_pages=3 * 64 + 8)
    assert runner.cuda_graphs and any(getattr(b.mixer, "w_ukv", None) is not None for b in runner.model.blocks)
    tokens = helpers.random_tokens(start + portion, 101, 3)
    got = []
    for rid in "abc":
        runner.add_request(rid)
        if start:
            runner.step([StepEntry(rid, tokens[:start], ())])          # more tokens than a recording takes: eager every time
        got.append(runner.step([StepEntry(rid, tokens[start:], (0, portion - 1))]).clone())
    assert runner.graph_captures == 1 and runner.graph_replays == 1
    assert torch.equal(got[0], got[1]) and torch.equal(got[1], got[2])
    assert ops.tc_status() == 0
