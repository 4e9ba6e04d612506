"""What the float32 GEMM's epilogues write for the operators: triangle planes (groups of 16 channels, runs of eight pairs that do or
do not straddle pair rows), the end of an operator with a residual, a factor, transposed rows, four channels at a time or one by one.
float32 sums of a few hundred terms: 1e-6, as measured twice over (1.6e-7 to 4.5e-7)."""
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


def _with_biases(d, w):
    """The same weights with biases that are not zero."""
    return {k: d.rng.normal(size=v.shape).astype(np.float32) if "Bias" in k else v for k, v in w.items()}


def _relative(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("n,c,hidden,incoming", [(1, 16, 16, False), (7, 15, 15, True), (8, 17, 17, False), (31, 23, 16, True), (32, 32, 48, False), (33, 31, 64, True),
                                                 (40, 4, 8, False), (127, 24, 24, False), (136, 20, 129, True), (129, 40, 30, False)])
def test_triangle_update(dev, n, c, hidden, incoming):
    import localfold_b200 as lf
    d = syn.draw(7000 + n)
    z, mask, w = d.normal(n, n, c), (d.rng.random((n, n)) > 0.2).astype(np.float32), _with_biases(d, syn.af2_triangle_weights(d, c, hidden))
    mask[0, 0] = 1
    op = (lf.TriangleMultiplicationIncomingGpu if incoming else lf.TriangleMultiplicationOutgoingGpu)(dev)
    got = op.run({"shape": {"length": n, "cZ": c, "cHidden": hidden}, "z": z, "mask": mask, "weights": w}, {"precision": "f32", "variance": "two-pass"})["output"]
    assert _relative(got, t2.trimul_af2(z, mask, w, incoming=incoming)) <= 1e-6


@pytest.mark.parametrize("rows,c,residual", [(1, 5, False), (130, 33, True), (257, 66, False), (128, 128, True)])
def test_transition(dev, rows, c, residual):
    import localfold_b200 as lf
    d = syn.draw(7100 + rows)
    act, w = d.normal(rows, c), _with_biases(d, syn.af2_transition_weights(d, c))
    got = lf.TransitionGpu(dev).run({"activations": act, "rows": rows, "channels": c, "hiddenChannels": 4 * c, "weights": w},
                                    {"precision": "f32", "variance": "two-pass", "residual": residual})["output"]
    assert _relative(got, t2.transition_af2(act, w) + (act if residual else 0)) <= 1e-6


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("n,heads,dim", [(31, 1, 5), (65, 3, 22), (97, 4, 16)])
def test_attention_with_a_residual(dev, n, heads, dim, transpose):
    import localfold_b200 as lf
    d = syn.draw(7200 + n)
    c = heads * dim
    act, mask = d.normal(n, n, c), np.ones((n, n), np.float32)
    w = syn.af2_attention_weights(d, c, heads, c)
    pb = dict(w["pairBias"], source="normalized-input")
    got = lf.AttentionGpu(dev).run({"activations": act, "mask": mask, "batch": n, "queryLength": n, "channels": c, "heads": heads, "weights": w["attention"],
                                    "transpose": transpose, "pairBias": pb}, {"precision": "f32", "variance": "two-pass", "residual": True})["output"]
    want = t2.attention_af2(act, mask, n, n, c, heads, w["attention"], transpose, pb)
    assert _relative(got, act.astype(np.float64) + want) <= 1e-6
