"""What 16-bit mode rounds at widths the fused 128-channel kernels do not take: of a triangle update only a, b and the
stored product x, of an attention whose heads the tcgen05 core does not take nothing.  The float64 evaluation of the triangle
update here rounds exactly those, so what is left between it and the GPU is float32 arithmetic and the values that land on
the other side of a rounding boundary because of it."""
import numpy as np
import pytest
import torch

from localfold_b200 import synthetic as syn
from oracle import tier2_torch as t2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import localfold_b200 as lf
    d = lf.Device(0)
    yield d
    d.close()


def _relative(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def _triangle_with_16_bit_contraction(z, mask, w, incoming):
    def half(v):
        return v.to(torch.float16).to(t2.F64)

    def lin(x, k):
        return x @ t2.T(w[f"linear{k}Weight"]).T + t2.T(w[f"linear{k}Bias"])

    n = z.shape[0]
    scale = 2.0 ** -int(0.5 * np.log2(n))
    zn = t2.ln(t2.T(z), w["layerNormInWeight"], w["layerNormInBias"])
    m = t2.T(mask)[..., None]
    a, b = half(lin(zn, "AP") * torch.sigmoid(lin(zn, "AG")) * m), half(lin(zn, "BP") * torch.sigmoid(lin(zn, "BG")) * m)
    x = torch.einsum("kjc,kic->ijc", a, b) if incoming else torch.einsum("ikc,jkc->ijc", a, b)
    x = half(x * scale) / scale
    xn = t2.ln(x, w["layerNormOutWeight"], w["layerNormOutBias"])
    return (lin(xn, "Z") * torch.sigmoid(lin(zn, "G"))).numpy()


# float32 errors of 3e-7 put about one value in a thousand on the other side of a boundary 2^-10.5 apart: 2e-5 each from a and b, 4e-5
# from x, 5e-5 together.  One more tensor in fp16 (2^-11 / sqrt(3) at most, 2e-4 on average) is well outside.
@pytest.mark.parametrize("n,c,incoming", [(20, 64, False), (65, 24, True), (33, 136, True), (130, 64, True), (129, 16, False), (40, 256, False), (530, 8, False)])
def test_triangle_update_rounds_its_contraction_only(dev, n, c, incoming):
    import localfold_b200 as lf
    d = syn.draw(5000 + n)
    z, mask, w = d.normal(n, n, c), syn.residue_pair_mask(n, 0.1), syn.af2_triangle_weights(d, c, c)
    op = (lf.TriangleMultiplicationIncomingGpu if incoming else lf.TriangleMultiplicationOutgoingGpu)(dev)
    got = op.run({"shape": {"length": n, "cZ": c, "cHidden": c}, "z": z, "mask": mask, "weights": w}, {"precision": "bf16", "variance": "two-pass"})["output"]
    assert _relative(got, _triangle_with_16_bit_contraction(z, mask, w, incoming)) <= 1e-4


# Heads that the tcgen05 core (groups of four heads of 32, no bias from the normalised input beside 128 channels) does not take run in
# float32 in either mode: the float32 mode's bound.
@pytest.mark.parametrize("q,heads,dim,transpose,own_bias", [(20, 4, 16, False, True), (65, 8, 8, True, True), (47, 12, 32, True, True), (129, 3, 24, False, True),
                                                            (33, 8, 8, False, False), (130, 4, 16, True, False)])
def test_attention_of_other_heads_is_float32(dev, q, heads, dim, transpose, own_bias):
    import localfold_b200 as lf
    d = syn.draw(5100 + q)
    c = heads * dim
    act, mask = d.normal(q, q, c), (d.rng.random((q, q)) > 0.2).astype(np.float32)
    w = syn.af2_attention_weights(d, c, heads, c)
    pb = dict(w["pairBias"], source="normalized-input") if own_bias else None
    got = lf.AttentionGpu(dev).run({"activations": act, "mask": mask, "batch": q, "queryLength": q, "channels": c, "heads": heads, "weights": w["attention"],
                                    "transpose": transpose, "pairBias": pb}, {"precision": "bf16", "variance": "two-pass"})["output"]
    assert _relative(got, t2.attention_af2(act, mask, q, q, c, heads, w["attention"], transpose, pb)) <= 1e-5
