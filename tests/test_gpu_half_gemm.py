"""16-bit mode's plain GEMM (tiles of 128 x 256 x 64, epilogue shares of 32 x 64) at the edges of its tiles, in each of its output layouts: fp16 rows and
float32 rows (transition), attention pieces in both orientations (MSA attention of 32-wide heads), sums grouped per pair
(outer product mean of 32 channels)."""
import numpy as np
import pytest

from localfold_b200 import synthetic as syn
from oracle import oracle

pytestmark = pytest.mark.gpu
TOL = 8e-3


@pytest.fixture(scope="module")
def dev():
    import localfold_b200 as lf
    d = lf.Device(0)
    yield d
    d.close()


@pytest.mark.parametrize("rows,c,hidden", [(1, 8, 8), (31, 64, 256), (128, 72, 264), (129, 136, 120), (300, 256, 1024), (257, 384, 4160)])
def test_transition(dev, rows, c, hidden):
    import localfold_b200 as lf
    d = syn.draw(4000 + rows)
    act = d.normal(rows, c)
    w = {"layerNormScale": 1 + d.normal(c, std=0.1), "layerNormOffset": d.normal(c, std=0.1), "firstWeight": d.linear(c, c, hidden),
         "firstBias": d.normal(hidden, std=0.1), "secondWeight": d.linear(hidden, hidden, c), "secondBias": d.normal(c, std=0.1)}
    got = lf.TransitionGpu(dev).run({"activations": act, "rows": rows, "channels": c, "hiddenChannels": hidden, "weights": w}, {"precision": "bf16"})["output"]
    assert oracle.relative_l2(got, oracle.transition_af2(act, w, hidden)) <= TOL


@pytest.mark.parametrize("q,batch,heads,transpose,bias", [(1, 3, 8, False, False), (7, 5, 12, True, False), (31, 2, 8, False, True), (33, 130, 8, True, False),
                                                          (127, 2, 8, False, True), (129, 3, 8, True, False), (257, 2, 12, False, True),
                                                          (260, 1, 8, False, True), (300, 3, 8, False, True)])
def test_attention_pieces(dev, q, batch, heads, transpose, bias):
    import localfold_b200 as lf
    d = syn.draw(4100 + q)
    c = heads * 32
    act = d.normal(batch * q, c)
    mask = (d.rng.random((q, batch) if transpose else (batch, q)) > 0.2).astype(np.float32)
    w = syn.af2_attention_weights(d, c, heads, 128, separate=True)
    pb = dict(w["pairBias"], source="separate", channels=128, activations=d.normal(q, q, 128)) if bias else None
    got = lf.AttentionGpu(dev).run({"activations": act, "mask": mask, "batch": batch, "queryLength": q, "channels": c, "heads": heads,
                                    "weights": w["attention"], "transpose": transpose, "pairBias": pb}, {"precision": "bf16"})["output"]
    want = oracle.attention_af2(act, mask, batch, q, c, heads, w["attention"], transpose, pb)
    assert oracle.relative_l2(got, want) <= TOL


@pytest.mark.parametrize("S,n", [(1, 1), (63, 3), (65, 9), (130, 33)])
def test_outer_product_mean(dev, S, n):
    import localfold_b200 as lf
    d = syn.draw(4200 + n)
    msa, mask = d.normal(S, n, 64), (d.rng.random((S, n)) > 0.2).astype(np.float32)
    mask[0] = 1
    w = syn.af2_opm_weights(d, 64, 32, 128)
    got = lf.OuterProductMeanGpu(dev).run({"activations": msa, "mask": mask, "sequences": S, "length": n, "cM": 64, "cOuter": 32, "cZ": 128, "weights": w},
                                          {"precision": "bf16"})["output"]
    assert oracle.relative_l2(got, oracle.outer_product_mean_af2(msa, mask, w, 32, 128)) <= TOL
