"""d_head 64 prefill with an accumulator per softmax group: the hand-overs that depend on which group
an item's key tiles fall to, against the CPU oracle.  Tolerances as in test_prefill_gpu (fp16 O 2e-3,
LSE 1e-3, max abs)."""
import numpy as np
import pytest

from helpers import run_prefill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [1, 128, 129, 257, 400])
@pytest.mark.parametrize("causal", [True, False])
def test_many_items_per_cta(fa, dev, oracle, s, causal):
    """More items than SMs several times over; items of one tile leave one accumulator unused, and odd
    tile counts move the groups' roles from item to item."""
    bh, d = 460, 64
    q, k, v = (oracle.round_to(x, "f16") for x in oracle.normal_inputs(9100 + s, (bh, s, d)))
    o, lse = run_prefill(fa, dev, q, k, v, 0.125, causal)
    assert fa.device_status() == 0
    o_ref, l_ref = oracle.attention(q, k, v, 0.125, causal)
    assert np.abs(o - o_ref).max() < 2e-3
    assert np.abs(lse - l_ref).max() < 1e-3


@pytest.mark.parametrize("order", ["rising", "falling", "odd tiles high"])
def test_group_maxima_far_apart(fa, dev, oracle, order):
    """Tile maxima that differ by far more than the rescale threshold (2^8), within and between groups."""
    bh, s, d = 3, 1000, 64
    q, k, v = (oracle.round_to(x, "f16") for x in oracle.normal_inputs(9200, (bh, s, d)))
    q[..., 0], k[..., 0] = 4.0, 0.0
    tile = np.arange(s) // 128
    level = {"rising": tile, "falling": 8 - tile, "odd tiles high": (tile & 1) * 6}[order]
    k[..., 0] = level * 24.0                       # + 12 (17 in log2 units) in the exponent per level
    o, lse = run_prefill(fa, dev, q, k, v, 0.125, False)
    assert fa.device_status() == 0
    o_ref, l_ref = oracle.attention(q, k, v, 0.125, False)
    assert np.abs(o - o_ref).max() < 2e-3
    assert np.abs(lse - l_ref).max() < 1e-3


@pytest.mark.parametrize("dead_tile", [0, 1, 3])
def test_tile_of_minus_infinity_scores(fa, dev, oracle, dead_tile):
    """A key tile whose scores are all -inf weighs nothing, whichever group meets it first."""
    bh, s, d = 2, 500, 64
    q, k, v = (oracle.round_to(x, "f16") for x in oracle.normal_inputs(9300, (bh, s, d)))
    q[..., 0], k[..., 0] = 1.0, 0.0
    dead = np.arange(s) // 128 == dead_tile
    o_ref, l_ref = oracle.attention(q, k[:, ~dead], v[:, ~dead], 0.125, False)
    k[:, dead, 0] = -np.inf
    o, lse = run_prefill(fa, dev, q, k, v, 0.125, False)
    assert fa.device_status() == 0
    assert np.abs(o - o_ref).max() < 2e-3
    assert np.abs(lse - l_ref).max() < 1e-3
