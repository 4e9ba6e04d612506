"""Weight preparation: blocks that come back from closed operators, tensors too large for a layout map, a scratch limit
with no room for the tensors' bytes, uploads past the end of the staging buffer, and weights used from another context."""
import numpy as np
import pytest

from localfold_b200 import synthetic as syn
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import localfold_b200 as lf
    d = lf.Device(0)
    yield d
    d.close()


def _transition(dev, rows, c, hidden, seed, run_dev=None, check=True):
    import localfold_b200 as lf
    from localfold_b200 import _native as nat
    from localfold_b200.operators import TRANSITION_WEIGHT_ORDER
    d = syn.draw(seed)
    act = d.normal(rows, c)
    w = {"layerNormScale": 1 + d.normal(c, std=0.1), "layerNormOffset": d.normal(c, std=0.1), "firstWeight": d.linear(c, c, hidden),
         "firstBias": d.normal(hidden, std=0.1), "secondWeight": d.linear(hidden, hidden, c), "secondBias": d.normal(c, std=0.1)}
    prepared = lf.PreparedWeights(dev, nat.WEIGHTS_TRANSITION_AF2, {"channels": c, "hidden": hidden}, [w[k] for k in TRANSITION_WEIGHT_ORDER])
    given = {"activations": act, "rows": rows, "channels": c, "hiddenChannels": hidden, "weights": prepared}
    got = {p: lf.TransitionGpu(run_dev or dev).run(given, {"precision": p})["output"] for p in ("f32", "bf16")}
    prepared.close()
    want = oracle.transition_af2(act, w, hidden)
    assert oracle.relative_l2(got["f32"], want) <= 1e-5
    assert oracle.relative_l2(got["bf16"], want) <= 8e-3


def test_blocks_are_reused_by_later_operators(dev):
    for seed, (c, hidden) in enumerate([(128, 512), (64, 256), (128, 512), (72, 200), (128, 512), (13, 7)] * 2):
        _transition(dev, 37, c, hidden, 700 + seed)


def test_tensors_past_the_staging_buffer_and_past_a_layout_map(dev):
    _transition(dev, 5, 1024, 2304, 720)      # 18.9 MB: the staging buffer fills up in the middle of a tensor
    _transition(dev, 3, 1024, 8192, 721)      # 2^24 + elements: laid out on the host


def test_scratch_limit_without_room_for_the_tensors(dev):
    from localfold_b200 import _native as nat
    import localfold_b200 as lf
    other = lf.Device(0)
    other.limit_scratch(1 << 16)
    w = syn.af2_transition_weights(syn.draw(730), 128)
    prepared = lf.PreparedWeights(other, nat.WEIGHTS_TRANSITION_AF2, {"channels": 128, "hidden": 512},
                                  [w[k] for k in ("layerNormScale", "layerNormOffset", "firstWeight", "firstBias", "secondWeight", "secondBias")])
    act = syn.draw(731).normal(50, 128)
    got = lf.TransitionGpu(dev).run({"activations": act, "rows": 50, "channels": 128, "hiddenChannels": 512, "weights": prepared},
                                    {"precision": "bf16"})["output"]
    assert oracle.relative_l2(got, oracle.transition_af2(act, w, 512)) <= 8e-3
    prepared.close()
    other.close()


def test_weights_used_from_another_context_at_once(dev):
    import localfold_b200 as lf
    other = lf.Device(0)
    for seed in range(4):
        _transition(dev, 64, 384, 1536, 740 + seed, run_dev=other)
    other.close()


@pytest.mark.parametrize("n,c,more", [(20, 128, 1), (33, 64, 1)])
def test_first_float32_call_of_a_pair_stack(dev, n, c, more):
    """What the float32 mode derives from a stack's weights at its first call is one launch more (at 64 channels the transition's alone: the
    other operators run in float32 in either mode), also where two blocks share their weights; the results do not change."""
    import localfold_b200 as lf
    from localfold_b200.stack import PreparedPairBlock
    d = syn.draw(750 + n)
    pair, mask, w = d.normal(n, n, c), syn.residue_pair_mask(n, 0.1), syn.af2_pair_block_weights(d, c, c, 4)
    options = {"precision": "f32", "variance": "two-pass"}
    block = PreparedPairBlock(dev, w, c, c)
    stack = lf.PairStackGpu(dev).prepare([block, block], c, c)
    first, again = stack.run(pair, mask, options), stack.run(pair, mask, options)
    assert first["launches"] - again["launches"] == more
    assert np.array_equal(first["pair"], again["pair"])
    other = lf.Device(0)
    elsewhere = lf.PairStackGpu(other).prepare([block, block], c, c)
    assert np.array_equal(elsewhere.run(pair, mask, options)["pair"], again["pair"])
    block.close()
    other.close()
