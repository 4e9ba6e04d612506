"""Device tensors that do not start on a 16-byte (or, as bfloat16, 32-byte) boundary: a view into a larger allocation.  The
fused kernels do not take them; the calls do, through the general path, in every operator and mode."""
import numpy as np
import pytest

from localfold_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import torch

    import localfold_b200 as lf
    d = lf.Device(0, stream=torch.cuda.current_stream().cuda_stream)
    yield d
    d.close()


def _at(value, offset, dtype="float32"):
    """A contiguous device tensor `offset` elements past an allocation's start."""
    import torch
    host = torch.from_numpy(np.ascontiguousarray(value, np.float32)).to(getattr(torch, dtype))
    room = torch.zeros(host.numel() + 64, dtype=host.dtype, device="cuda")
    out = room[offset:offset + host.numel()].view(host.shape)
    out.copy_(host)
    return out


def _relative(got, want):
    got, want = got.double(), want.double()
    return float((got - want).norm() / want.norm())


# (the two paths differ by what 16-bit mode rounds, at most the mode's 8e-3 an update, a bfloat16 result by one more rounding)
PLACES = [("float32", 1), ("float32", 2), ("bfloat16", 1), ("bfloat16", 8)]


def _check(run, value, dtype, offset, tol=8e-3):
    """run(tensor, residual) on the same values aligned and not, into a new tensor and added in place."""
    want = run(_at(value, 0, dtype), False)
    got = run(_at(value, offset, dtype), False)
    assert _relative(got, want) <= tol
    want, got = run(_at(value, 0, dtype), True), run(_at(value, offset, dtype), True)
    assert _relative(got, want) <= tol


@pytest.mark.parametrize("dtype,offset", PLACES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("c", [128, 64])
def test_triangle_update(dev, c, precision, dtype, offset):
    import localfold_b200 as lf
    n = 33
    d = syn.draw(6000 + c)
    z, mask, w = d.normal(n, n, c), _at(syn.residue_pair_mask(n, 0.1), 1), syn.af2_triangle_weights(d, c, c)

    def run(t, residual):
        out = t if residual else _at(np.zeros((n, n, c)), offset, dtype)
        given = {"shape": {"length": n, "cZ": c, "cHidden": c}, "z": t, "mask": mask, "weights": w}
        lf.TriangleMultiplicationOutgoingGpu(dev).run(given, {"precision": precision, "variance": "two-pass", "residual": residual}, out=out)
        return out.clone()
    _check(run, z, dtype, offset)


@pytest.mark.parametrize("dtype,offset", PLACES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("c,heads,source", [(128, 4, "own"), (64, 4, "own"), (256, 8, "separate"), (256, 8, None)])
def test_attention(dev, c, heads, source, precision, dtype, offset):
    import localfold_b200 as lf
    n = 35
    d = syn.draw(6100 + c + heads)
    act, mask = d.normal(n, n, c), _at((d.rng.random((n, n)) > 0.2).astype(np.float32), 3)
    w = syn.af2_attention_weights(d, c, heads, 128 if source == "separate" else c, separate=source == "separate")
    pair = d.normal(n, n, 128)

    def run(t, residual):
        out = t if residual else _at(np.zeros((n, n, c)), offset, dtype)
        pb = None
        if source == "own":
            pb = dict(w["pairBias"], source="normalized-input")
        elif source == "separate":
            pb = dict(w["pairBias"], source="separate", channels=128, activations=_at(pair, t.storage_offset(), dtype))
        lf.AttentionGpu(dev).run({"activations": t, "mask": mask, "batch": n, "queryLength": n, "channels": c, "heads": heads, "weights": w["attention"],
                                  "transpose": source is None, "pairBias": pb}, {"precision": precision, "variance": "two-pass", "residual": residual}, out=out)
        return out.clone()
    _check(run, act, dtype, offset)


@pytest.mark.parametrize("dtype,offset", PLACES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
@pytest.mark.parametrize("c", [128, 256, 72])
def test_transition(dev, c, precision, dtype, offset):
    import localfold_b200 as lf
    d = syn.draw(6200 + c)
    w = syn.af2_transition_weights(d, c)
    act = d.normal(300, c)

    def run(t, residual):
        out = t if residual else _at(np.zeros((300, c)), offset, dtype)
        lf.TransitionGpu(dev).run({"activations": t, "rows": 300, "channels": c, "hiddenChannels": 4 * c, "weights": w},
                                  {"precision": precision, "variance": "two-pass", "residual": residual}, out=out)
        return out.clone()
    _check(run, act, dtype, offset)


@pytest.mark.parametrize("dtype,offset", PLACES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_outer_product_mean(dev, precision, dtype, offset):
    import localfold_b200 as lf
    S, n = 9, 21
    d = syn.draw(6300)
    msa, mask = _at(d.normal(S, n, 64), 1), _at(np.ones((S, n)), 1)
    w = syn.af2_opm_weights(d, 64, 32, 128)

    def run(t, residual):
        lf.OuterProductMeanGpu(dev).run({"activations": msa, "mask": mask, "sequences": S, "length": n, "cM": 64, "cOuter": 32, "cZ": 128, "weights": w},
                                        {"precision": precision, "variance": "two-pass", "residual": residual}, out=t)
        return t.clone()
    _check(run, d.normal(n, n, 128), dtype, offset)


@pytest.mark.parametrize("dtype,offset", PLACES)
@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_pair_stack(dev, precision, dtype, offset):
    import localfold_b200 as lf
    n = 33
    pair, mask, weights = syn.af2_pair_block(6400, n, masked_tail=0.1)
    stack = lf.PairStackGpu(dev).prepare(weights, 128, 128)
    got, want = _at(pair, offset, dtype), _at(pair, 0, dtype)
    for t in (got, want):
        stack.run(t, _at(mask, 1), {"precision": precision, "variance": "two-pass"})
    assert _relative(got, want) <= (6e-3 if dtype == "bfloat16" else 2e-3)      # a block's bounds
    stack.close()
