"""Float32 mode through the split-operand GEMM at the edges of its tiles (128 x 128 x 64): rows, columns and inner lengths
around them, widths that are not whole groups of eight, contractions past one accumulation chunk of 64 - and no less
accurate than a float32 product: the error against float64 stays below that of float32 rounding of every operand."""
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


@pytest.mark.parametrize("rows,c,hidden", [(1, 8, 8), (127, 64, 256), (128, 128, 512), (129, 136, 120), (300, 65, 129), (257, 384, 640), (40, 512, 1100)])
@pytest.mark.parametrize("af3", [False, True])
def test_transition_edges(dev, rows, c, hidden, af3):
    import localfold_b200 as lf
    from localfold_b200 import _native as nat
    from localfold_b200.operators import TRANSITION_AF3_ORDER
    d = syn.draw(3000 + rows)
    act = d.normal(rows, c)
    if af3:
        w = {"inputLayerNormScale": 1 + d.normal(c, std=0.1), "inputLayerNormOffset": d.normal(c, std=0.1),
             "transition1": d.linear(c, c, 8 * c), "transition2": d.linear(4 * c, 4 * c, c)}
        got = lf.Af3TransitionGpu(dev).run(act, {"rows": rows, "channels": c, "factor": 4}, w, {"precision": "f32"})["output"]
        want = oracle.transition_af3(act, w, 4)
    else:
        w = {"layerNormScale": 1 + d.normal(c, std=0.1), "layerNormOffset": d.normal(c, std=0.1), "firstWeight": d.linear(c, c, hidden),
             "firstBias": d.normal(hidden, std=0.1), "secondWeight": d.linear(hidden, hidden, c), "secondBias": d.normal(c, std=0.1)}
        got = lf.TransitionGpu(dev).run({"activations": act, "rows": rows, "channels": c, "hiddenChannels": hidden, "weights": w},
                                        {"precision": "f32"})["output"]
        want = oracle.transition_af2(act, w, hidden)
    assert np.isfinite(got).all()
    assert oracle.relative_l2(got, want) <= 1e-6


@pytest.mark.parametrize("n,c,incoming", [(1, 8, False), (63, 16, True), (64, 32, False), (65, 24, True), (127, 8, False), (129, 16, True), (200, 12, False), (530, 8, False), (530, 8, True), (70, 72, False), (33, 136, True)])
@pytest.mark.parametrize("precision,tol", [("f32", 2e-6), ("bf16", 8e-3)])
def test_triangle_edges(dev, n, c, incoming, precision, tol):
    import localfold_b200 as lf
    d = syn.draw(3100 + n)
    z, mask, w = d.normal(n, n, c), syn.residue_pair_mask(n, 0.1 if n > 1 else 0.0), syn.af2_triangle_weights(d, c, c)
    op = (lf.TriangleMultiplicationIncomingGpu if incoming else lf.TriangleMultiplicationOutgoingGpu)(dev)
    got = op.run({"shape": {"length": n, "cZ": c, "cHidden": c}, "z": z, "mask": mask, "weights": w}, {"precision": precision})["output"]
    want = oracle.trimul_af2(z, mask, w, c, incoming=incoming)
    assert oracle.relative_l2(got, want) <= tol


@pytest.mark.parametrize("S,n,cm,heads,dim", [(1, 1, 16, 2, 8), (3, 31, 64, 8, 8), (130, 33, 64, 8, 8), (17, 129, 40, 3, 12), (9, 65, 24, 2, 5)])
def test_msa_averaging_edges(dev, S, n, cm, heads, dim):
    import localfold_b200 as lf
    msa, pair, mask, _, w = syn.af3_msa_block(3200 + n, S=S, n=n, cm=cm, cz=32, msa_heads=heads, msa_dim=dim)
    if n > 1:
        mask[:, -1] = 0                 # a token that no sequence covers
    got = lf.Af3MsaAttentionGpu(dev).run(msa, mask, pair, {"sequences": S, "tokens": n, "msaChannels": cm, "pairChannels": 32},
                                         w["msaAttention1"], {"precision": "f32"})["output"]
    want = oracle.msa_attention_af3(msa, mask, pair, w["msaAttention1"])
    assert oracle.relative_l2(got, want) <= 2e-6


@pytest.mark.parametrize("S,n,c,heads,dim", [(1, 1, 8, 1, 8), (7, 5, 64, 8, 8), (300, 9, 40, 3, 20), (33, 17, 600, 2, 32)])
def test_global_attention_edges(dev, S, n, c, heads, dim):
    import localfold_b200 as lf
    d = syn.draw(3300 + S)
    act = d.normal(S, n, c)
    mask = (d.rng.random((S, n)) > 0.3).astype(np.float32)
    w = syn.af2_global_attention_weights(d, c, heads, dim)
    got = lf.GlobalColumnAttentionGpu(dev).run({"activations": act, "mask": mask, "sequences": S, "length": n, "channels": c, "weights": w},
                                               {"precision": "f32"})["output"]
    want = oracle.global_column_attention_af2(act, mask, w)
    assert np.isfinite(got).all()
    assert oracle.relative_l2(got, want) <= 1e-5
