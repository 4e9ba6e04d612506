"""The float32 attention core on tcgen05 (heads of 8, 16 and 32 channels, enough logits to pay): query counts around the tiles of 128 queries and
32 keys, batch rows that do not fill a group of four, more items than blocks, both orientations, rows whose reference has to be
raised, fully masked rows; and that what is not finite stays in its batch row.

The bound is the float32 mode's: logits of size 100 come with errors of 100 x 2^-24 x a few, which the exponentials pass on; with
weights of the usual size the error is below 5e-7."""
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


def _relative(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def _case(q, batch, heads, dim, transpose, bias, big=1):
    d = syn.draw(6000 + q)
    c = heads * dim
    act = d.normal(batch * q, c)
    mask = (d.rng.random((q, batch) if transpose else (batch, q)) > 0.25).astype(np.float32)
    w = syn.af2_attention_weights(d, c, heads, 32, separate=True)
    att = dict(w["attention"], queryWeight=w["attention"]["queryWeight"] * big, keyWeight=w["attention"]["keyWeight"] * big)
    pb = None
    if bias:
        pb = dict(w["pairBias"], source="separate", channels=32, activations=d.normal(q, q, 32))
        pb["projectionWeight"] = pb["projectionWeight"] * (big + 2)
    return {"activations": act, "mask": mask, "batch": batch, "queryLength": q, "channels": c, "heads": heads, "weights": att, "transpose": transpose,
            "pairBias": pb}


def _want(g):
    return t2.attention_af2(g["activations"], g["mask"], g["batch"], g["queryLength"], g["channels"], g["heads"], g["weights"], g["transpose"], g["pairBias"])


# every one of these goes to the tcgen05 kernel (attention3_wins)
SIZES = [(94, 131, 4, 16, False, True), (96, 97, 4, 32, True, True), (97, 99, 4, 32, False, False), (127, 130, 4, 16, True, False), (128, 66, 4, 32, False, True),
         (200, 129, 8, 8, False, True), (160, 131, 8, 8, True, False), (203, 40, 4, 32, True, True), (256, 70, 8, 16, False, True), (385, 41, 4, 16, True, True),
         (131, 161, 4, 32, False, True), (32, 885, 4, 32, True, True)]      # 32 channels with two and six items a block, of several key tiles and of one


@pytest.mark.parametrize("q,batch,heads,dim,transpose,bias", SIZES)
def test_attention_core_edges(dev, q, batch, heads, dim, transpose, bias):
    import localfold_b200 as lf
    given = _case(q, batch, heads, dim, transpose, bias)
    got = lf.AttentionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass"})["output"]
    assert _relative(got, _want(given)) <= 1e-6


@pytest.mark.parametrize("q,batch,heads,dim,transpose,bias", [SIZES[1], SIZES[3], SIZES[5], SIZES[9]])
def test_raised_references_and_masked_rows(dev, q, batch, heads, dim, transpose, bias):
    import localfold_b200 as lf
    given = _case(q, batch, heads, dim, transpose, bias, big=6)
    by_row = given["mask"].T if transpose else given["mask"]
    by_row[0, :40] = 0           # the first tile of a row is masked: its reference is raised from near -1e9
    by_row[1] = 0                # no key is left
    by_row[2, 33:] = 0
    got = lf.AttentionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass"})["output"]
    assert np.isfinite(got).all()
    assert _relative(got, _want(given)) <= 1e-5


def test_these_sizes_run_this_kernel(dev):
    import localfold_b200 as lf
    import torch
    calls = [_case(*size) for size in SIZES] + [_square(*size)[0] for size in SQUARES]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for given in calls:
            lf.AttentionGpu(dev).run(given, {"precision": "f32"})
    names = [e.name for e in prof.events()]
    assert sum("attention3_kernel" in name for name in names) == len(calls)
    assert not any("mma_attention" in name for name in names)


# the pair bias as columns of the projection: 97 is one item a block, 203 are three
SQUARES = [(97, 4, 32, True), (203, 4, 32, False), (200, 4, 16, True), (202, 8, 8, False)]


def _square(n, heads, dim, transpose):
    d, c = syn.draw(6200 + n), heads * dim
    w = syn.af2_attention_weights(d, c, heads, c)
    return {"activations": d.normal(n * n, c), "mask": (d.rng.random((n, n)) > 0.25).astype(np.float32), "batch": n, "queryLength": n, "channels": c, "heads": heads,
            "weights": w["attention"], "transpose": transpose, "pairBias": dict(w["pairBias"], source="normalized-input")}, d


@pytest.mark.parametrize("n,heads,dim,transpose", SQUARES)
def test_bias_from_the_normalised_input(dev, n, heads, dim, transpose):
    import localfold_b200 as lf
    given, d = _square(n, heads, dim, transpose)
    given["pairBias"]["projectionWeight"] = given["pairBias"]["projectionWeight"] * 3
    got = lf.AttentionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass"})["output"]
    assert _relative(got, _want(given)) <= 1e-6


@pytest.mark.parametrize("n", [98, 131])
@pytest.mark.parametrize("transpose,swap", [(False, False), (True, False), (True, True)])
def test_bias_of_the_transposed_dialects(dev, n, transpose, swap):
    import localfold_b200 as lf
    d = syn.draw(6300 + n)
    pair, mask, w = d.normal(n, n, 128), (d.rng.random((n, n)) > 0.25).astype(np.float32), syn.af3_grid_attention_weights(d, 128, 4, 32)
    got = lf.Af3GridSelfAttentionGpu(dev).run(pair, mask, {"n": n, "channels": 128, "transpose": transpose}, w, {"swapTransposedBias": swap}, {"precision": "f32"})["output"]
    assert _relative(got, t2.grid_attention_af3(pair, mask, w, transpose, swap)) <= 1e-6


def test_what_is_not_finite_stays_in_its_row(dev):
    import localfold_b200 as lf
    given = _case(97, 99, 4, 32, False, False)
    clean = lf.AttentionGpu(dev).run(given, {"precision": "f32"})["output"].reshape(99, 97, -1)
    given["activations"].reshape(99, 97, -1)[6, 96] = np.inf      # a row between others of its group, the key a partial tile ends on
    got = lf.AttentionGpu(dev).run(given, {"precision": "f32"})["output"].reshape(99, 97, -1)
    rest = np.arange(99) != 6
    assert np.isnan(got[6]).any() and np.array_equal(got[rest], clean[rest])


# Runs of keys (first, one behind the last) with logits of +-8e4 or +-2.4e5, a query each: up across 65536 behind the first key tile; from below
# -65536 back to the others' size and up; up twice beyond 65536; below it where the reference is not theirs.  Three neighbouring lanes, another warp.
FAR = {3: [(40, 41, 8e4)], 4: [(0, 35, -8e4), (70, 71, 8e4)], 5: [(33, 34, 8e4), (66, 67, 2.4e5)], 37: [(0, 33, -2.4e5), (64, 90, -8e4)]}


@pytest.mark.parametrize("q,batch,heads,dim,transpose,bias", [SIZES[0], SIZES[1], SIZES[5]])
def test_queries_with_far_logits_leave_the_others_alone(dev, q, batch, heads, dim, transpose, bias):
    import localfold_b200 as lf
    given = _case(q, batch, heads, dim, transpose, bias)
    given["mask"][:] = 1
    # Pair rows of +1 and -1 in equal numbers have mean 0 exactly, so their last four channels are 0 after the LayerNorm; rows of +-8 in two of these
    # channels and nothing else have +-4 there.
    pair = np.zeros((q, q, 32), np.float32)
    pair[..., :28] = syn.draw(6100 + q).rng.permuted(np.tile(np.repeat(np.float32([1, -1]), 14), (q, q, 1)), axis=-1)
    for query, runs in FAR.items():
        for first, last, logit in runs:
            pair[query, first:last] = 0
            at = 30 if abs(logit) == 8e4 else 28
            pair[query, first:last, at:at + 2] = np.float32([8, -8]) * np.sign(logit)
    given["pairBias"]["activations"] = pair
    given["pairBias"]["projectionWeight"][28:] = np.float32([3e4, -3e4, 1e4, -1e4])[:, None]
    got, want = lf.AttentionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass"})["output"], _want(given)
    by_query = (lambda x: x.reshape(q, batch, -1).swapaxes(0, 1)) if transpose else (lambda x: x.reshape(batch, q, -1))
    got, want = by_query(got), by_query(want)
    ordinary = ~np.isin(np.arange(q), list(FAR))
    assert _relative(got[:, ordinary], want[:, ordinary]) <= 1e-6
    assert _relative(got[:, ~ordinary], want[:, ~ordinary]) <= 1e-6      # each of them ends on one key or on ordinary ones
