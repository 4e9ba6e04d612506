"""The 16-bit attention core's two forms of work item - a query tile of two neighbouring batch rows, two neighbouring query tiles of one row - at the
sizes around the line between them (148 SMs) and at their edges: an odd last row, a row by itself, an odd last tile, partial tiles of queries and keys.

The bound: projections, gate, probabilities and products are rounded to fp16 (2^-12 relative each, six of them in a chain that averages out to
2.5 x 2^-12 = 6e-4 of an update's norm)."""
import numpy as np
import pytest

from localfold_b200 import synthetic as syn
from oracle import tier2_torch as t2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import localfold_b200 as lf
    d = lf.Device(0)
    yield d
    d.close()


# With a bias: up to 36 rows of 500 queries fill one round either way, 37 only as tiles, 38 neither; without one, 370 rows of two query tiles are five
# rounds and the last ones as tiles; one row is always tiles
@pytest.mark.parametrize("q,batch,transpose", [(256, 2, False), (250, 3, True), (129, 5, False), (500, 36, False), (500, 37, False), (511, 37, True), (500, 38, True),
                                               (700, 1, False), (200, 1, True), (1100, 9, False), (130, 370, False), (130, 371, True)])
@pytest.mark.parametrize("bias", [True, False])
def test_forms(dev, q, batch, transpose, bias):
    import localfold_b200 as lf
    d = syn.draw(9000 + q + batch)
    heads, c = 4, 128
    act = d.normal(batch * q, c)
    mask = (d.rng.random((q, batch) if transpose else (batch, q)) > 0.2).astype(np.float32)
    w = syn.af2_attention_weights(d, c, heads, 128, separate=True)
    pb = dict(w["pairBias"], source="separate", channels=128, activations=d.normal(q, q, 128)) if bias else None
    dev.profile(True)
    got = lf.AttentionGpu(dev).run({"activations": act, "mask": mask, "batch": batch, "queryLength": q, "channels": c, "heads": heads, "weights": w["attention"],
                                    "transpose": transpose, "pairBias": pb}, {"precision": "bf16", "variance": "two-pass"})["output"]
    launches = dev.profile_read()["attention"][1]
    dev.profile(False)
    assert launches == 1      # this core, not the float32 one
    want = np.asarray(t2.attention_af2(act, mask, batch, q, c, heads, w["attention"], transpose, pb), np.float64)
    got = np.asarray(got, np.float64).reshape(want.shape)
    assert np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want)
