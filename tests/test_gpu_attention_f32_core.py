"""The float32 attention core at the edges of its tiles: query counts around the groups of 16 and the key tiles of 32,
head widths on either side of every instance (whole and broken groups of four and eight), rows whose reference has to
be raised (their first keys masked, large logits later), fully masked rows, both orientations."""
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


@pytest.mark.parametrize("q,batch,heads,dim,transpose,bias", [
    (1, 3, 2, 8, False, True), (15, 2, 1, 5, False, True), (16, 5, 2, 16, True, False), (17, 4, 4, 32, False, True),
    (31, 3, 2, 24, True, True), (32, 2, 8, 8, False, False), (33, 40, 2, 13, False, True), (127, 3, 4, 16, True, True),
    (128, 2, 2, 41, False, True), (129, 2, 1, 64, False, True), (145, 1, 16, 24, False, True), (64, 300, 4, 32, False, True)])
def test_attention_core_edges(dev, q, batch, heads, dim, transpose, bias):
    import localfold_b200 as lf
    d = syn.draw(2000 + q)
    c = heads * dim
    act = d.normal(batch * q, c)
    mask = (d.rng.random((q, batch) if transpose else (batch, q)) > 0.25).astype(np.float32)
    first = mask[:, 0] if transpose else mask[0]
    first[:min(q, 40)] = 0                 # the first tile of batch row 0 is masked: its reference is raised later, or no key is left
    w = syn.af2_attention_weights(d, c, heads, 32, separate=True)
    att = dict(w["attention"], queryWeight=w["attention"]["queryWeight"] * 6, keyWeight=w["attention"]["keyWeight"] * 6)
    pb = None
    if bias:
        pb = dict(w["pairBias"], source="separate", channels=32, activations=d.normal(q, q, 32))
        pb["projectionWeight"] = pb["projectionWeight"] * 8
    given = {"activations": act, "mask": mask, "batch": batch, "queryLength": q, "channels": c, "heads": heads, "weights": att,
             "transpose": transpose, "pairBias": pb}
    got = lf.AttentionGpu(dev).run(given, {"precision": "f32"})["output"]
    want = oracle.attention_af2(act, mask, batch, q, c, heads, att, transpose, pb)
    assert np.isfinite(got).all()
    assert oracle.relative_l2(got, want) <= 1e-5
