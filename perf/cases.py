"""Performance cases of the pair stack and the operators around it.

Each case is one call (or one short loop of calls) that a structure-prediction program makes through the package's
public classes: single operators, the AF2 pair stack in its storage and precision options, the template stack, whole
Evoformer and extra-MSA blocks, the AF3 pairformer and MSA stacks.  Activations are N(0, 1), weights N(0, 1/fan_in),
as everywhere in this repository; lengths are those of the benchmark and the tests, and odd ones like real chains.
"""
import math
import random

import numpy as np
import torch

import localfold_b200 as lf
from localfold_b200 import synthetic as syn

C_M, C_Z, C_S, C_OUTER, C_EXTRA = 256, 128, 384, 32, 64
MSA_HEADS, PAIR_HEADS, SINGLE_HEADS = 8, 4, 16


def listed():
    return [
        # the smallest call: one triangle update of a short chain, device tensors, launch latency counts
        {"name": "tri_out_n64", "family": "op", "op": "triangle_outgoing", "n": 64, "precision": "bf16", "tail": 0.0},
        # a first call of the library: numpy arrays, the default precision (baseline configuration 0)
        {"name": "pair_n64_f32_host", "family": "pair", "n": 64, "blocks": 1, "precision": "f32", "store": "f32", "space": "host",
         "template": False, "tail": 0.0},
        # the float32 mode on an ordinary chain of odd length, pair resident, padded residues masked
        {"name": "pair_n203_f32", "family": "pair", "n": 203, "blocks": 1, "precision": "f32", "store": "f32", "space": "device",
         "template": False, "tail": 0.05},
        # the benchmark's shorter length, 16-bit mode, two blocks of the stack in one call
        {"name": "pair_n384", "family": "pair", "n": 384, "blocks": 2, "precision": "bf16", "store": "f32", "space": "device",
         "template": False, "tail": 0.0},
        # a bf16 pair stream (half the memory) at a ragged length, padded residues masked
        {"name": "pair_n701_bf16_stream", "family": "pair", "n": 701, "blocks": 1, "precision": "bf16", "store": "bf16", "space": "device",
         "template": False, "tail": 0.05},
        # the benchmark's workload: one block at the largest length
        {"name": "pair_n2048", "family": "pair", "n": 2048, "blocks": 1, "precision": "bf16", "store": "f32", "space": "device",
         "template": False, "tail": 0.0},
        # the template pair stack: 64 channels, attentions first, two blocks
        {"name": "template_n384", "family": "pair", "n": 384, "blocks": 2, "precision": "bf16", "store": "f32", "space": "device",
         "template": True, "tail": 0.0},
        # AF3 pairformer blocks with a single track from an int5 bundle's tensors (baseline configuration 2's shape)
        {"name": "pairformer_n384_int5", "family": "pairformer", "n": 384, "blocks": 4, "weights": "int5"},
        # one whole Evoformer block at the baseline's configuration 1
        {"name": "evoformer_s128_n256", "family": "evoformer", "sequences": 128, "n": 256, "precision": "bf16"},
        # ... and at the shape of the reference's published per-block figure
        {"name": "evoformer_s512_n825", "family": "evoformer", "sequences": 512, "n": 825, "precision": "bf16"},
        # one extra-MSA block: a deep alignment at 64 channels, global column attention
        {"name": "extra_msa_s1024_n256", "family": "extra_msa", "sequences": 1024, "n": 256, "precision": "bf16"},
        # one AF3 MSA block: pair-weighted averaging, outer product, pair updates
        {"name": "af3_msa_s512_n384", "family": "af3_msa", "sequences": 512, "n": 384, "blocks": 1},
    ]


OPS = ("triangle_outgoing", "triangle_incoming", "attention_start", "attention_end", "transition")


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random):
    family = rng.choice(("op", "pair", "pair", "pair_f32", "template", "pairformer", "evoformer", "evoformer", "extra_msa", "af3_msa"))
    if family == "op":
        return {"family": "op", "op": rng.choice(OPS), "n": _log_int(rng, 16, 512), "precision": "bf16", "tail": rng.choice((0.0, 0.05))}
    if family == "pair":
        return {"family": "pair", "n": _log_int(rng, 64, 1536), "blocks": 1, "precision": "bf16", "store": rng.choice(("f32", "f32", "bf16")),
                "space": "device", "template": False, "tail": rng.choice((0.0, 0.05))}
    if family == "pair_f32":
        return {"family": "pair", "n": _log_int(rng, 24, 320), "blocks": 1, "precision": "f32", "store": "f32",
                "space": rng.choice(("host", "device")), "template": False, "tail": rng.choice((0.0, 0.05))}
    if family == "template":
        return {"family": "pair", "n": _log_int(rng, 64, 480), "blocks": 2, "precision": "bf16", "store": "f32", "space": "device",
                "template": True, "tail": rng.choice((0.0, 0.05))}
    if family == "pairformer":
        return {"family": "pairformer", "n": _log_int(rng, 48, 768), "blocks": rng.randint(1, 4), "weights": rng.choice(("int5", "f32"))}
    if family == "evoformer":
        return {"family": "evoformer", "sequences": _log_int(rng, 32, 512), "n": _log_int(rng, 64, 640), "precision": "bf16"}
    if family == "extra_msa":
        return {"family": "extra_msa", "sequences": _log_int(rng, 96, 1536), "n": _log_int(rng, 48, 320), "precision": "bf16"}
    return {"family": "af3_msa", "sequences": _log_int(rng, 32, 768), "n": _log_int(rng, 64, 480), "blocks": 1}


# ---------------------------------------------------------------------------
# inputs


def _normal(generator, *shape):
    return torch.randn(*shape, generator=generator, device="cuda", dtype=torch.float32)


def _pair_mask(n, tail):
    return torch.from_numpy(syn.residue_pair_mask(n, tail)).cuda()


def _gapped_mask(generator, sequences, n, gaps):
    """An alignment with a fraction of gaps; its first row is whole."""
    mask = (torch.rand(sequences, n, generator=generator, device="cuda") >= gaps).float()
    mask[0] = 1
    return mask


def _row_mask(generator, sequences, n, share):
    """Whole rows masked, as at the end of a padded alignment."""
    rows = torch.ones(sequences, device="cuda")
    rows[torch.randperm(sequences, generator=generator, device="cuda")[: int(round(sequences * share))]] = 0
    return rows[:, None].repeat(1, n).contiguous()


def _int5(rng, shape, std):
    """A tensor as an int5 bundle stores it: groups of 32 five-bit codes, an fp16 scale and zero point for each."""
    count = int(np.prod(shape))
    groups = -(-count // 32)
    body = rng.bytes(groups * 20) + b"\0"
    body += b"\0" * (-len(body) % 4)
    reach = std * math.sqrt(3.0) * (1 + 0.1 * rng.random(groups))
    scales, zeros = (2 * reach / 31).astype(np.float16), (-reach).astype(np.float16)
    return lf.EncodedTensor(body + scales.tobytes() + zeros.tobytes(), len(body), len(body) + scales.nbytes, count, shape)


def _encode(weights, rng):
    """The linear weights of a block as int5 tensors, its norms, biases and whole numbers as they are."""
    out = {}
    for key, value in weights.items():
        if isinstance(value, dict):
            out[key] = _encode(value, rng)
        elif isinstance(value, np.ndarray) and value.ndim >= 2:
            out[key] = _int5(rng, value.shape, float(value.reshape(-1)[:4096].std()))
        else:
            out[key] = value
    return out


def _op_state(case, g, d):
    n, opts = case["n"], {"precision": case["precision"], "variance": "two-pass"}
    z, mask, op = _normal(g, n, n, C_Z), _pair_mask(n, case["tail"]), case["op"]
    device = lf.TriangleMultiplicationOutgoingGpu().device
    if op.startswith("triangle"):
        from localfold_b200.operators import prepare_triangle_weights
        runner = (lf.TriangleMultiplicationOutgoingGpu if op == "triangle_outgoing" else lf.TriangleMultiplicationIncomingGpu)(device)
        given = {"shape": {"length": n, "cZ": C_Z, "cHidden": C_Z}, "z": z, "mask": mask,
                 "weights": prepare_triangle_weights(device, syn.af2_triangle_weights(d, C_Z, C_Z), C_Z, C_Z)}
    elif op.startswith("attention"):
        from localfold_b200.operators import prepare_attention_weights
        w = syn.af2_attention_weights(d, C_Z, PAIR_HEADS, C_Z)
        bias = dict(w["pairBias"], source="normalized-input")
        runner = lf.AttentionGpu(device)
        given = {"activations": z, "mask": mask, "batch": n, "queryLength": n, "channels": C_Z, "heads": PAIR_HEADS,
                 "transpose": op == "attention_end", "pairBias": bias,
                 "weights": prepare_attention_weights(device, w["attention"], C_Z, PAIR_HEADS, bias)}
    else:
        from localfold_b200 import _native
        from localfold_b200.operators import TRANSITION_WEIGHT_ORDER
        w = syn.af2_transition_weights(d, C_Z)
        runner = lf.TransitionGpu(device)
        given = {"activations": z, "rows": n * n, "channels": C_Z, "hiddenChannels": 4 * C_Z,
                 "weights": lf.PreparedWeights(device, _native.WEIGHTS_TRANSITION_AF2, {"channels": C_Z, "hidden": 4 * C_Z},
                                               [w[k] for k in TRANSITION_WEIGHT_ORDER])}
    return {"runner": runner, "given": given, "options": opts}


def _pair_state(case, g, d):
    n, c = case["n"], 64 if case["template"] else C_Z
    stack = lf.PairStackGpu()
    stack.prepare([syn.af2_pair_block_weights(d, c, c, PAIR_HEADS, 4) for _ in range(case["blocks"])], c, c)
    pair, mask = _normal(g, n, n, c), _pair_mask(n, case["tail"])
    if case["store"] == "bf16":
        pair = pair.to(torch.bfloat16)
    if case["space"] == "host":
        pair, mask = pair.cpu().numpy(), mask.cpu().numpy()
    options = {"precision": case["precision"], "variance": "two-pass"}
    if case["template"]:
        options["order"] = "template"
    return {"stack": stack, "pair": pair, "mask": mask, "options": options}


def _pairformer_state(case, g, d, seed):
    n = case["n"]
    blocks = [syn.af3_pairformer_block_weights(d, C_Z, C_S, PAIR_HEADS, SINGLE_HEADS) for _ in range(case["blocks"])]
    if case["weights"] == "int5":
        rng = np.random.default_rng(seed)
        blocks = [_encode(b, rng) for b in blocks]
    state = {"pair": _normal(g, n, n, C_Z), "single": _normal(g, n, C_S), "pairMask": _pair_mask(n, 0.0),
             "seqMask": torch.ones(n, device="cuda"), "tokens": n}
    return {"runner": lf.Af3PairformerStackGpu(), "state": state, "blocks": blocks, "dialect": {"swapTransposedBias": True},
            "options": {"precision": "bf16", "variance": "fast"}}


def _evoformer_state(case, g, d):
    S, n, extra = case["sequences"], case["n"], case["family"] == "extra_msa"
    cm = C_EXTRA if extra else C_M
    w = {"msaRowAttention": syn.af2_attention_weights(d, cm, MSA_HEADS, C_Z, separate=True),
         "msaTransition": syn.af2_transition_weights(d, cm), "outerProductMean": syn.af2_opm_weights(d, cm, C_OUTER, C_Z)}
    if extra:
        w["msaColumnGlobalAttention"] = syn.af2_global_attention_weights(d, cm, MSA_HEADS, cm // MSA_HEADS)
    else:
        w["msaColumnAttention"] = syn.af2_attention_weights(d, cm, MSA_HEADS)
    w.update(syn.af2_pair_block_weights(d, C_Z, C_Z, PAIR_HEADS))
    runner = (lf.ExtraMsaStackGpu if extra else lf.EvoformerStackGpu)()
    given = {"sequences": S, "length": n, "cM": cm, "cZ": C_Z, "cOuter": C_OUTER, "triangleHidden": C_Z,
             "msa": _normal(g, S, n, cm), "pair": _normal(g, n, n, C_Z), "pairMask": _pair_mask(n, 0.0),
             "msaMask": _gapped_mask(g, S, n, 0.15) if extra else _row_mask(g, S, n, 0.1),
             "blockWeights": [lf.PreparedMsaBlock(runner.device, w, cm, C_Z, C_OUTER, C_Z)]}
    return {"runner": runner, "given": given, "options": {"precision": case["precision"], "variance": "two-pass"}}


def _af3_msa_state(case, g, d):
    S, n = case["sequences"], case["n"]
    state = {"msa": _normal(g, S, n, C_EXTRA), "pair": _normal(g, n, n, C_Z), "msaMask": _gapped_mask(g, S, n, 0.2),
             "pairMask": _pair_mask(n, 0.0), "sequences": S, "tokens": n}
    blocks = [syn.af3_msa_block_weights(d, C_EXTRA, C_Z, C_OUTER) for _ in range(case["blocks"])]
    return {"runner": lf.Af3MsaStackGpu(), "state": state, "blocks": blocks,
            "dialect": {"swapTransposedBias": False, "msaUpdateBeforeOuterProduct": False}, "options": {"precision": "bf16", "variance": "fast"}}


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    d = syn.draw(seed)
    family = case["family"]
    if family == "op":
        made = _op_state(case, g, d)
    elif family == "pair":
        made = _pair_state(case, g, d)
    elif family == "pairformer":
        made = _pairformer_state(case, g, d, seed)
    elif family == "af3_msa":
        made = _af3_msa_state(case, g, d)
    else:
        made = _evoformer_state(case, g, d)
    made["family"] = family
    return made


def run(state):
    family = state["family"]
    if family == "op":
        return state["runner"].run(state["given"], state["options"])["output"]
    if family == "pair":                  # device tensors are updated in place, numpy arrays come back as a new array
        return state["stack"].run(state["pair"], state["mask"], state["options"])["pair"]
    if family == "pairformer":
        out = state["runner"].run(state["state"], state["blocks"], state["dialect"], state["options"])
        return {"pair": out["pair"], "single": out["single"]}
    if family == "af3_msa":
        out = state["runner"].run(state["state"], state["blocks"], state["dialect"], state["options"])
        return {"msa": out["msa"], "pair": out["pair"]}
    out = state["runner"].run(state["given"], state["options"])
    return {"msa": out["msa"], "pair": out["pair"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _triangle_flops(n, c):
    return 2.0 * n * n * c * (4 * c + 2 * c) + 2.0 * n ** 3 * c


def _attention_flops(n, c, heads):
    return 2.0 * n * n * c * (5 * c + heads) + 4.0 * n ** 3 * c


def _transition_flops(rows, c, swiglu):
    return 2.0 * rows * c * 4 * c * (3 if swiglu else 2)


def _pair_block_flops(n, c, swiglu=False):
    return 2 * _triangle_flops(n, c) + 2 * _attention_flops(n, c, PAIR_HEADS) + _transition_flops(n * n, c, swiglu)


def _opm_flops(S, n, cm):
    return 2.0 * S * n * cm * 2 * C_OUTER + 2.0 * S * (n * C_OUTER) ** 2 + 2.0 * n * n * C_OUTER ** 2 * C_Z


def work(case):
    family, n = case["family"], case["n"]
    pairs = float(n) * n
    if family == "op":
        op = case["op"]
        flops = (_triangle_flops(n, C_Z) if op.startswith("triangle") else _attention_flops(n, C_Z, PAIR_HEADS) if op.startswith("attention")
                 else _transition_flops(n * n, C_Z, False))
        return {"bytes": pairs * (2 * C_Z * 4 + (0 if op == "transition" else 4)), "flops": flops}
    if family == "pair":
        c, width = 64 if case["template"] else C_Z, 2 if case["store"] == "bf16" else 4
        return {"bytes": pairs * (2 * c * width + 4), "flops": case["blocks"] * _pair_block_flops(n, c)}
    if family == "pairformer":
        single = 2.0 * n * C_S * 5 * C_S + 4.0 * pairs * C_S + 2.0 * pairs * C_Z * SINGLE_HEADS + _transition_flops(n, C_S, True)
        weights = 4.0e6 * (0.625 + 0.125 if case["weights"] == "int5" else 4)      # about 4 million weights a block
        return {"bytes": pairs * (2 * C_Z * 4 + 4) + 2.0 * n * C_S * 4 + case["blocks"] * weights,
                "flops": case["blocks"] * (_pair_block_flops(n, C_Z, True) + single)}
    S = case["sequences"]
    rows = float(S) * n
    cm = C_M if family == "evoformer" else C_EXTRA
    moved = 2 * rows * cm * 4 + rows * 4 + pairs * (2 * C_Z * 4 + 4)
    if family == "af3_msa":
        averaging = 2.0 * rows * cm * 3 * cm + 2.0 * pairs * C_Z * MSA_HEADS + 2.0 * S * pairs * cm
        flops = averaging + _transition_flops(rows, cm, True) + _opm_flops(S, n, cm) + _pair_block_flops(n, C_Z, True)
        return {"bytes": moved, "flops": case["blocks"] * flops}
    row = 2.0 * rows * cm * 5 * cm + 4.0 * S * pairs * cm + 2.0 * pairs * C_Z * MSA_HEADS
    if family == "evoformer":
        column = 2.0 * rows * cm * 5 * cm + 4.0 * n * float(S) * S * cm
    else:        # one key and value head for all, a mean query a column
        column = 2.0 * rows * cm * (2 * cm + 2 * cm // MSA_HEADS) + 4.0 * rows * cm
    return {"bytes": moved, "flops": row + column + _transition_flops(rows, cm, False) + _opm_flops(S, n, cm) + _pair_block_flops(n, C_Z)}


def tolerance(case):
    """float32 mode: the repository's bound for one block.  16-bit mode: fp16 operands into float32 sums, read against
    the operator's own output, or against a running pair of unit size; a bf16 pair stream rounds at every update."""
    if case.get("precision") == "f32":
        return {"rel": 1e-5}
    if case.get("store") == "bf16":
        return {"rel": 6e-3}
    return {"rel": 4e-3 if case["family"] == "op" else 2e-3}
