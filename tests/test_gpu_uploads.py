"""Weights that another context of the GPU prepares (Device.uploads) while this one computes: the calls that use them wait for them,
whichever thread and device object runs them, and closing in any order is clean."""
import threading

import numpy as np
import pytest

from localfold_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _run(dev, blocks, n):
    import localfold_b200 as lf
    d = syn.draw(8000 + n)
    state = {"pair": d.normal(n, n, 128), "single": d.normal(n, 384), "pairMask": np.ones((n, n), np.float32), "seqMask": np.ones(n, np.float32), "tokens": n}
    out = lf.Af3PairformerStackGpu(dev).run(state, blocks, {"swapTransposedBias": True}, {"precision": "bf16", "variance": "fast"})
    return out["pair"], out["single"]


def test_stacks_of_several_threads_and_devices():
    import localfold_b200 as lf
    d = syn.draw(8100)
    blocks = [syn.af3_pairformer_block_weights(d, 128, 384, 4, 16) for _ in range(3)]
    dev = lf.Device(0)
    want = {n: _run(dev, blocks, n) for n in (17, 64)}
    got = {}

    def work(key, n):
        own = lf.Device(0)
        got[key] = _run(own, blocks, n)
        own.close()

    threads = [threading.Thread(target=work, args=((n, k), n)) for n in want for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (n, _), result in got.items():
        assert all(np.array_equal(a, b) for a, b in zip(result, want[n]))
    assert len(got) == 4
    dev.limit_scratch(1 << 30)
    dev.release_scratch()
    assert all(np.array_equal(a, b) for a, b in zip(_run(dev, blocks, 17), want[17]))
    dev.close()


def test_weights_outlive_the_devices_that_prepared_them():
    import localfold_b200 as lf
    d = syn.draw(8150)
    pair, mask, w = d.normal(40, 40, 128), np.ones((40, 40), np.float32), syn.af2_pair_block_weights(d)
    first, dev = lf.Device(0), lf.Device(0)
    stack = lf.PairStackGpu(dev).prepare([w], 128, 128, first.uploads())
    want = {p: stack.run(pair, mask, {"precision": p, "variance": "two-pass"})["pair"] for p in ("bf16", "f32")}
    again = lf.PairStackGpu(dev).prepare([w], 128, 128, first.uploads())
    first.close()      # the weights' contexts go, then the one that uses them, then the weights
    for p in want:
        assert np.array_equal(again.run(pair, mask, {"precision": p, "variance": "two-pass"})["pair"], want[p])
    dev.close()
    stack.close()
    again.close()


def test_a_scratch_limit_and_the_launch_count_cover_the_weights():
    """A device counts the launches of one that prepares its weights itself; a limit leaves it one arena."""
    import localfold_b200 as lf
    d = syn.draw(8200)
    blocks = [syn.af3_pairformer_block_weights(d, 128, 384, 4, 16) for _ in range(2)]
    counts, results = [], []
    for limit in (0, 1 << 30):
        dev = lf.Device(0)
        dev.limit_scratch(limit)
        before = dev.launch_count()
        results.append(_run(dev, blocks, 33))
        counts.append(dev.launch_count() - before)
        assert (dev.uploads() is dev) == (limit != 0)
        dev.limit_scratch(1 << 30)
        assert dev.uploads() is dev
        results.append(_run(dev, blocks, 33))
        dev.limit_scratch(0)
        assert dev.uploads() is not dev
        dev.close()
    assert counts[0] == counts[1]
    assert all(np.array_equal(a, b) for r in results[1:] for a, b in zip(r, results[0]))
