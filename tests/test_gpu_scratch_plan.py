"""What a call is planned to need is what it takes: under a limit of exactly the scratch that it used, the same call runs, whether its float32
result leaves with the last GEMM (in place, aligned) or by a pass of its own (off a 16-byte boundary, another buffer's residual)."""
import numpy as np
import pytest

from localfold_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _tensor(values, offset):
    import torch
    buf = torch.empty(values.size + 4, device="cuda")
    view = buf[offset:offset + values.size].view(values.shape)
    view.copy_(torch.from_numpy(values))
    return view


def _triangle(lf, dev, d, place, n=96, c=64):
    act = place(d.normal(n, n, c))
    w, mask = syn.af2_triangle_weights(d, c, c), _tensor(np.ones((n, n), np.float32), 0)
    return act, lambda out: lf.TriangleMultiplicationOutgoingGpu(dev).run({"shape": {"length": n, "cZ": c, "cHidden": c}, "z": act, "mask": mask, "weights": w},
                                                                          {"precision": "f32", "residual": True}, out=out)


def _attention(lf, dev, d, place, n=70, heads=4, dim=16):
    c = heads * dim
    act = place(d.normal(n, n, c))
    w, mask = syn.af2_attention_weights(d, c, heads, c), _tensor(np.ones((n, n), np.float32), 0)
    given = {"activations": act, "mask": mask, "batch": n, "queryLength": n, "channels": c, "heads": heads, "weights": w["attention"], "transpose": True,
             "pairBias": dict(w["pairBias"], source="normalized-input")}
    return act, lambda out: lf.AttentionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass", "residual": True}, out=out)


def _transition(lf, dev, d, place, rows=5000, c=64):
    act = place(d.normal(rows, c))
    w = syn.af2_transition_weights(d, c)
    given = {"activations": act, "rows": rows, "channels": c, "hiddenChannels": 4 * c, "weights": w}
    return act, lambda out: lf.TransitionGpu(dev).run(given, {"precision": "f32", "variance": "two-pass", "residual": True}, out=out)


def _global(lf, dev, d, place, s=60, n=50, c=64):
    act = place(d.normal(s, n, c))
    given = {"activations": act, "mask": _tensor(np.ones((s, n), np.float32), 0), "sequences": s, "length": n, "channels": c,
             "weights": syn.af2_global_attention_weights(d, c, 8, 8)}
    return act, lambda out: lf.GlobalColumnAttentionGpu(dev).run(given, {"residual": True}, out=out)


def _average(lf, dev, d, place, s=60, n=50):
    act = place(d.normal(s, n, 64))
    mask, pair, w = _tensor(np.ones((s, n), np.float32), 0), _tensor(d.normal(n, n, 128), 0), syn.af3_msa_attention_weights(d, 64, 128, 8, 8)
    shape = {"sequences": s, "tokens": n, "msaChannels": 64, "pairChannels": 128}
    return act, lambda out: lf.Af3MsaAttentionGpu(dev).run(act, mask, pair, shape, w, {"residual": True}, out=out)


def _stack(lf, dev, d, place, n=40, c=128):      # a host array
    act = d.normal(n, n, c)
    stack = lf.PairStackGpu(dev).prepare([syn.af2_pair_block_weights(d, c, c, 4)], c, c)
    return act, lambda out: stack.run(act, np.ones((n, n), np.float32), {"precision": "f32", "variance": "two-pass"})


@pytest.mark.parametrize("offset,apart", [(0, False), (1, False), (0, True)])
@pytest.mark.parametrize("op", [_triangle, _attention, _transition, _global, _average, _stack])
def test_a_limit_of_what_a_call_takes(op, offset, apart):
    import localfold_b200 as lf
    import torch
    results, limit = [], 0
    for _ in range(2):
        dev = lf.Device(0)
        dev.limit_scratch(limit)
        act, call = op(lf, dev, syn.draw(9000), lambda values: _tensor(values, offset))
        out = None if op is _stack else torch.empty_like(act) if apart else act
        used = call(out)
        dev.synchronize()
        results.append(used["pair"] if op is _stack else out.cpu().numpy())
        limit = used["memory"]["peakBytes"]
        dev.close()
    assert np.array_equal(results[0], results[1])


def test_the_arena_stays_within_its_limit():
    """The room an arena gets to grow into ends at the limit (what the driver hands out is whole pieces of 2 MiB)."""
    import localfold_b200 as lf
    import torch
    dev, limit = lf.Device(0), 512 << 20
    dev.limit_scratch(limit)
    dev.synchronize()
    free = torch.cuda.mem_get_info()[0]
    dev.reserve(limit)
    assert 0 <= free - torch.cuda.mem_get_info()[0] - limit <= 2 << 20
    with pytest.raises(MemoryError):
        dev.reserve(limit + 1)
    dev.close()
