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


# ---- device tensors updated in place: the last GEMM adds to them, a launch less than from host arrays, whose result goes to another buffer ----

OPTIONS = {"precision": "f32", "variance": "two-pass", "residual": True}


def _in_place(run, act, mask):
    import torch
    x = torch.from_numpy(act).cuda()
    here, there = run(x, torch.from_numpy(mask).cuda(), x), run(act, mask, None)
    assert here["launches"] == there["launches"] - 1
    return x.cpu().numpy()


@pytest.mark.parametrize("n,c,hidden", [(1, 16, 16), (31, 20, 24), (40, 64, 64), (129, 4, 30)])
def test_triangle_update_in_place(dev, n, c, hidden):
    import localfold_b200 as lf
    d = syn.draw(7600 + n)
    z, mask, w = d.normal(n, n, c), (d.rng.random((n, n)) > 0.2).astype(np.float32), _with_biases(d, syn.af2_triangle_weights(d, c, hidden))
    mask[0, 0] = 1
    op, shape = lf.TriangleMultiplicationOutgoingGpu(dev), {"length": n, "cZ": c, "cHidden": hidden}
    got = _in_place(lambda z, mask, out: op.run({"shape": shape, "z": z, "mask": mask, "weights": w}, OPTIONS, out=out), z, mask)
    assert _relative(got, z + t2.trimul_af2(z, mask, w)) <= 1e-6


@pytest.mark.parametrize("rows,c", [(1, 8), (130, 36), (257, 64)])
def test_transition_in_place(dev, rows, c):
    import localfold_b200 as lf
    d = syn.draw(7700 + rows)
    act, w = d.normal(rows, c), _with_biases(d, syn.af2_transition_weights(d, c))
    given = {"rows": rows, "channels": c, "hiddenChannels": 4 * c, "weights": w}
    got = _in_place(lambda act, _, out: lf.TransitionGpu(dev).run(dict(given, activations=act), OPTIONS, out=out), act, np.ones(1, np.float32))
    assert _relative(got, act + t2.transition_af2(act, w)) <= 1e-6


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("batch,q,heads,dim", [(3, 31, 1, 8), (65, 33, 2, 22), (97, 97, 4, 32)])
def test_attention_in_place(dev, batch, q, heads, dim, transpose):
    import localfold_b200 as lf
    d, c = syn.draw(7800 + q), heads * dim
    act, mask = d.normal(batch * q, c), np.ones((q, batch) if transpose else (batch, q), np.float32)
    w = _with_biases(d, syn.af2_attention_weights(d, c, heads)["attention"])
    given = {"batch": batch, "queryLength": q, "channels": c, "heads": heads, "weights": w, "transpose": transpose}
    got = _in_place(lambda act, mask, out: lf.AttentionGpu(dev).run(dict(given, activations=act, mask=mask), OPTIONS, out=out), act, mask)
    assert _relative(got, act + t2.attention_af2(act, mask, batch, q, c, heads, w, transpose)) <= 1e-6


# ---- a gate that is not a number: one channel of the gating weights ----


def _spoiled(w, name, channel):
    w = dict(w, **{name: w[name].copy()})
    w[name][..., channel] = np.nan
    return w


@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("c", [24, 64, 128])
def test_gates_of_the_triangle_pass_a_nan_on(dev, c, precision):
    import localfold_b200 as lf
    d, n = syn.draw(7300 + c), 40
    z, mask, w = d.normal(n, n, c), np.ones((n, n), np.float32), syn.af2_triangle_weights(d, c, c)

    def nans(name, channel):
        got = lf.TriangleMultiplicationOutgoingGpu(dev).run({"shape": {"length": n, "cZ": c, "cHidden": c}, "z": z, "mask": mask, "weights": _spoiled(w, name, channel)},
                                                            {"precision": precision, "variance": "two-pass"})["output"]
        return np.isnan(got)

    nan = nans("linearGBias", 5)
    assert nan[..., 5].all() and not np.delete(nan, 5, -1).any()
    for name in ("linearAGBias", "linearBGBias"):      # a channel of a contraction operand: all of it, so every pair's centre LayerNorm
        assert nans(name, 7).all()


@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("q,heads,dim", [(24, 2, 8), (97, 4, 16), (96, 4, 32), (40, 8, 32), (33, 3, 22)])
def test_gates_of_the_attention_pass_a_nan_on(dev, q, heads, dim, precision):
    import localfold_b200 as lf
    d, c = syn.draw(7400 + q), heads * dim
    w = syn.af2_attention_weights(d, c, heads)["attention"]
    got = lf.AttentionGpu(dev).run({"activations": d.normal(q, q, c), "mask": np.ones((q, q), np.float32), "batch": q, "queryLength": q, "channels": c, "heads": heads,
                                    "weights": _spoiled(w, "gatingBias", 3)}, {"precision": precision, "variance": "two-pass"})["output"]
    assert np.isnan(got).all()


@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_gates_of_global_attention_and_averaging_pass_a_nan_on(dev, precision):
    import localfold_b200 as lf
    d, s, n = syn.draw(7500), 20, 33
    act, mask = d.normal(s, n, 64), np.ones((s, n), np.float32)
    w = _spoiled(syn.af2_global_attention_weights(d, 64, 8, 8), "gatingBias", 3)
    assert np.isnan(lf.GlobalColumnAttentionGpu(dev).run({"activations": act, "mask": mask, "sequences": s, "length": n, "channels": 64, "weights": w},
                                                         {"precision": precision})["output"]).all()
    w = syn.af3_msa_attention_weights(d, 64, 128, 8, 8)
    w["gatingQuery"] = w["gatingQuery"].copy()
    w["gatingQuery"].reshape(-1)[3] = np.nan
    got = lf.Af3MsaAttentionGpu(dev).run(act, mask, d.normal(n, n, 128), {"sequences": s, "tokens": n, "msaChannels": 64, "pairChannels": 128}, w,
                                         {"precision": precision})["output"]
    assert np.isnan(got).all()
