"""Which steps expand the latents they see.  No GPU: the rule reads sizes and positions."""
from types import SimpleNamespace as NS

from quench6k_b200.parts.latent_attention import LatentAttention


def _takes(lens, starts, replayed=False):
    part = NS(w_ukv=1, H=16, dim=128, rd=64, vd=128, rank=512)
    return LatentAttention.expands(part, NS(replayed=replayed, q_lens=lens, max_q_len=max(lens), pos_starts=starts, plans={}))


def test_a_step_whose_positions_the_host_does_not_know_is_absorbed():
    assert _takes([300], [0]) and not _takes([300], [])                # a StepContext may come without host copies of the positions
    assert _takes([300, 200], [0, 0]) and not _takes([300, 200], [0])
