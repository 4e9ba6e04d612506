"""The mma.sync attention core (float32 mode, and 16-bit mode at head widths other than 4 x 32) at the edges of its tiles: query counts around the groups of 16 and the key tiles of 32,
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
    (128, 2, 2, 44, False, True), (37, 2, 2, 41, False, True), (129, 2, 1, 64, False, True), (145, 1, 16, 24, False, True), (64, 300, 4, 32, False, True)])
@pytest.mark.parametrize("precision,tol", [("f32", 1e-5), ("bf16", 8e-3)])
def test_attention_core_edges(dev, q, batch, heads, dim, transpose, bias, precision, tol):
    import localfold_b200 as lf
    d = syn.draw(2000 + q)
    c = heads * dim
    act = d.normal(batch * q, c)
    mask = (d.rng.random((q, batch) if transpose else (batch, q)) > 0.25).astype(np.float32)
    first = mask[:, 0] if transpose else mask[0]
    first[:min(q, 40)] = 0                 # the first tile of batch row 0 is masked: its reference is raised later, or no key is left
    pc = 128 if precision == "bf16" else 32
    big = 6 if precision == "f32" else 2
    w = syn.af2_attention_weights(d, c, heads, pc, separate=True)
    att = dict(w["attention"], queryWeight=w["attention"]["queryWeight"] * big, keyWeight=w["attention"]["keyWeight"] * big)
    pb = None
    if bias:
        pb = dict(w["pairBias"], source="separate", channels=pc, activations=d.normal(q, q, pc))
        pb["projectionWeight"] = pb["projectionWeight"] * (big + 2)
    given = {"activations": act, "mask": mask, "batch": batch, "queryLength": q, "channels": c, "heads": heads, "weights": att,
             "transpose": transpose, "pairBias": pb}
    got = lf.AttentionGpu(dev).run(given, {"precision": precision})["output"]
    want = oracle.attention_af2(act, mask, batch, q, c, heads, att, transpose, pb)
    assert np.isfinite(got).all()
    assert oracle.relative_l2(got, want) <= tol


@pytest.mark.parametrize("n,heads,dim,transpose,af3", [(20, 4, 16, False, False), (33, 4, 16, True, False), (47, 12, 32, True, True), (16, 3, 8, True, True), (65, 2, 24, False, True)])
@pytest.mark.parametrize("precision,tol", [("f32", 1e-5), ("bf16", 8e-3)])
def test_bias_from_the_normalised_input(dev, n, heads, dim, transpose, af3, precision, tol):
    """Triangle attention at widths other than 128: the bias columns ride in the projection, in either orientation."""
    import localfold_b200 as lf
    d = syn.draw(2100 + n)
    c = heads * dim
    pair = d.normal(n, n, c)
    mask = (d.rng.random((n, n)) > 0.2).astype(np.float32)
    if af3:
        w = syn.af3_grid_attention_weights(d, c, heads, dim)
        for swap in (False, True):
            got = lf.Af3GridSelfAttentionGpu(dev).run(pair, mask, {"n": n, "channels": c, "transpose": transpose}, w, {"swapTransposedBias": swap},
                                                      {"precision": precision})["output"]
            assert oracle.relative_l2(got, oracle.grid_attention_af3(pair, mask, w, transpose, swap)) <= tol
    else:
        w = syn.af2_attention_weights(d, c, heads, c)
        pb = dict(w["pairBias"], source="normalized-input")
        got = lf.AttentionGpu(dev).run({"activations": pair, "mask": mask, "batch": n, "queryLength": n, "channels": c, "heads": heads,
                                        "weights": w["attention"], "transpose": transpose, "pairBias": pb}, {"precision": precision})["output"]
        assert oracle.relative_l2(got, oracle.attention_af2(pair, mask, n, n, c, heads, w["attention"], transpose, pb)) <= tol
