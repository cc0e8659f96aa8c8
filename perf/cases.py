"""The framework's workloads for performance measurements: what its users have it do, through the
public entry points, from the smallest call to the largest.

A case is a dict of plain values with a ``kind``:

* ``linear``    one ``HLQLinear`` call on ``rows`` rows of activations;
* ``layer``     the seven projections of a decoder layer, one ``HLQLinear`` call each (prompt processing
                and batched decoding of a model that keeps its own glue);
* ``group``     the projections of ``layers`` layers as one ``HLQGroup`` launch;
* ``decode``    one token of a ``TPDecoder`` (decode chain, one CUDA graph per step);
* ``quantize``  fit and assignment of a whole weight (``pseudo_quantize_device``).

Weights, scales and activations have the distributions of the benchmark: planes Bernoulli(0.5),
alpha = |N(0, 0.02)|, z ~ N(0, 0.01), x ~ N(0, 1).
"""
import torch

from elutq_b200.decoder import DecoderConfig, TPDecoder
from elutq_b200.format import ExportedLinear, pseudo_quantize_device
from elutq_b200.linear import HLQGroup, HLQLinear, HLQWeight

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
FIT_ITERS = 10


def listed():
    return [
        # the smallest call: one token through a 4096-wide projection (latency and launch cost)
        {"name": "linear_1row_w2", "kind": "linear", "rows": 1, "n": 4096, "k": 4096, "bits": 2, "g": 128,
         "dtype": "fp16", "bias": False},
        # the lm_head of one decoded token, always quantized to 4 bits
        {"name": "lm_head_1row_w4", "kind": "linear", "rows": 1, "n": 128256, "k": 4096, "bits": 4, "g": 128,
         "dtype": "fp16", "bias": False},
        # batch-1 products of four Llama-3-8B layers in one launch: the weight stream itself
        {"name": "group_1row_w2", "kind": "group", "rows": 1, "layers": 4, "hidden": 4096, "ffn": 14336, "kv": 1024,
         "bits": 2, "g": 128},
        # decoding sixteen sequences together at 3 bits, four layers in one launch
        {"name": "group_16rows_w3", "kind": "group", "rows": 16, "layers": 4, "hidden": 4096, "ffn": 14336,
         "kv": 1024, "bits": 3, "g": 128},
        # a layer's projections for a batch of four sequences, call by call
        {"name": "layer_4rows_w3", "kind": "layer", "rows": 4, "hidden": 4096, "ffn": 14336, "kv": 1024, "bits": 3,
         "g": 128, "dtype": "fp16"},
        # a small batch on a 4-bit weight with a bias
        {"name": "linear_8rows_w4", "kind": "linear", "rows": 8, "n": 4096, "k": 4096, "bits": 4, "g": 64,
         "dtype": "fp16", "bias": True},
        # a short prompt, or a large decode batch, through a layer
        {"name": "layer_48rows_w3", "kind": "layer", "rows": 48, "hidden": 4096, "ffn": 14336, "kv": 1024, "bits": 3,
         "g": 128, "dtype": "fp16"},
        # odd sizes: rows, output and input channels that fill no tile
        {"name": "linear_333rows_ragged", "kind": "linear", "rows": 333, "n": 1000, "k": 1536, "bits": 3, "g": 64,
         "dtype": "bf16", "bias": True},
        # a 2048-token prompt through a Llama-2-13B layer
        {"name": "layer_2048rows_w2", "kind": "layer", "rows": 2048, "hidden": 5120, "ffn": 13824, "kv": 5120,
         "bits": 2, "g": 64, "dtype": "bf16"},
        # one token of a Llama-3-8B-shaped decoder at context 2048 (half of its 32 layers: all do the same work)
        {"name": "decode_8b", "kind": "decode", "hidden": 4096, "ffn": 14336, "layers": 16, "heads": 32, "kv_heads": 8,
         "vocab": 128256, "bits": 2, "g": 128, "ctx": 2048},
        # one token of a Llama-3-70B-shaped decoder (8 of its 80 layers)
        {"name": "decode_70b", "kind": "decode", "hidden": 8192, "ffn": 28672, "layers": 8, "heads": 64, "kv_heads": 8,
         "vocab": 128256, "bits": 2, "g": 128, "ctx": 2048},
        # the quantizer on one 4096-wide weight
        {"name": "quantize_w2", "kind": "quantize", "n": 4096, "k": 4096, "bits": 2, "g": 128},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("linear", "linear", "layer", "layer", "group", "decode", "quantize"))
    bits, g = rng.choice((2, 2, 3, 3, 4)), rng.choice((32, 64, 128))
    if kind == "linear":
        # rows over the whole range; shapes on and off the tiles
        return {"kind": kind, "rows": rng.choice((1, _log(rng, 2, 16), _log(rng, 17, 256), _log(rng, 257, 2048))),
                "n": _log(rng, 512, 16384), "k": g * _log(rng, 512 // g, 14336 // g), "bits": bits, "g": g,
                "dtype": rng.choice(("fp16", "bf16")), "bias": rng.random() < 0.3}
    if kind == "layer":
        hidden = 512 * rng.randint(4, 10)
        return {"kind": kind, "rows": rng.choice((1, _log(rng, 2, 16), _log(rng, 17, 256), _log(rng, 257, 2048))),
                "hidden": hidden, "ffn": 128 * rng.randint(hidden // 64, hidden * 27 // 1280),
                "kv": 128 * rng.randint(2, hidden // 128), "bits": bits, "g": g, "dtype": rng.choice(("fp16", "bf16"))}
    if kind == "group":
        hidden = 512 * rng.randint(2, 8)
        return {"kind": kind, "rows": rng.randint(1, 16), "layers": rng.randint(1, 4), "hidden": hidden,
                "ffn": 128 * rng.randint(hidden // 64, hidden * 7 // 256), "kv": 128 * rng.randint(1, hidden // 256),
                "bits": bits, "g": g}
    if kind == "decode":
        kv_heads = rng.choice((2, 4, 8))
        heads = kv_heads * rng.choice((4, 8))
        return {"kind": kind, "hidden": heads * 128, "ffn": 128 * rng.randint(heads * 2, heads * 7 // 2),
                "layers": rng.randint(2, 5), "heads": heads, "kv_heads": kv_heads, "vocab": 8 * _log(rng, 512, 16032),
                "bits": rng.choice((2, 3)), "g": rng.choice((64, 128)), "ctx": _log(rng, 64, 4096)}
    return {"kind": kind, "n": _log(rng, 64, 4096), "k": g * _log(rng, 512 // g, 4096 // g), "bits": bits, "g": g}


def _shapes(case):
    """(n, k) of the projections q, k, v, o, gate, up, down of one layer."""
    h, f, kv = case["hidden"], case["ffn"], case["kv"]
    return [(h, h), (kv, h), (kv, h), (h, h), (f, h), (f, h), (h, f)]


def _export(gen, n, k, bits, g, bias=False):
    planes = torch.randint(0, 256, (bits, n, k // 8), dtype=torch.uint8, device="cuda", generator=gen)
    scale = (torch.randn((bits, n, k // g), device="cuda", generator=gen) * 0.02).abs().half()
    zero = (torch.randn((n, k // g), device="cuda", generator=gen) * 0.01).half()
    b = (torch.randn((n,), device="cuda", generator=gen)).half() if bias else None
    return ExportedLinear(planes, scale, zero, b, g)


def _k_of(case, k):
    """Input channels padded up to whole groups (an exported weight has whole groups only)."""
    return -(-k // case["g"]) * case["g"]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        lin = HLQLinear.from_exported(_export(gen, case["n"], case["k"], case["bits"], case["g"], case["bias"]),
                                      max_batch=case["rows"])
        x = torch.randn((case["rows"], case["k"]), device="cuda", generator=gen).to(DTYPES[case["dtype"]])
        return {"case": case, "linears": [lin], "xs": [x]}
    if kind == "layer":
        lins, by_k, xs = [], {}, []
        for n, k in _shapes(case):
            k = _k_of(case, k)
            lins.append(HLQLinear.from_exported(_export(gen, n, k, case["bits"], case["g"]), max_batch=case["rows"]))
            if len(lins) == 4 or k not in by_k:      # o reads the attention's output, not the layer's input
                x = torch.randn((case["rows"], k), device="cuda", generator=gen).to(DTYPES[case["dtype"]])
                xs.append(x)
                if len(lins) != 4:
                    by_k[k] = x
            else:
                xs.append(by_k[k])
        return {"case": case, "linears": lins, "xs": xs}
    if kind == "group":
        weights, xs, ys = [], [], []
        for _ in range(case["layers"]):
            for n, k in _shapes(case):
                k = _k_of(case, k)
                weights.append(HLQWeight.from_export(_export(gen, n, k, case["bits"], case["g"])))
                xs.append(torch.randn((case["rows"], k), device="cuda", generator=gen).half())
                ys.append(torch.zeros((case["rows"], n), dtype=torch.float16, device="cuda"))
        group = HLQGroup(weights, max_m=case["rows"])
        group.bind(xs, ys)
        return {"case": case, "group": group}
    if kind == "decode":
        cfg = DecoderConfig(case["hidden"], case["ffn"], case["layers"], case["heads"], case["kv_heads"], 128,
                            case["vocab"], bits=case["bits"], groupsize=case["g"], ctx=case["ctx"])
        # every tensor of the decoder has a seed of its own, counted up from this one
        dec = TPDecoder(cfg, torch.device("cuda", 0), seed=seed * 4096, chain=True)
        # The random weights' mean is not zero and would carry the stream out of fp16's range within a few
        # layers; norm gains of either sign (and of a quarter in front of the MLP) keep it at a model's values.
        gains = [(layer[name], size) for layer in dec.layers for name, size in (("ln1", 1.0), ("ln2", 0.25))]
        for gain, size in gains + [(dec.norm, 1.0)]:
            gain.mul_(size * (torch.randint(0, 2, gain.shape, device="cuda", generator=gen) * 2 - 1))
        pos = cfg.ctx - 1
        rows = [dec.kv_rows(layer, name, pos, pos + 1) for layer in dec.layers for name in ("kc", "vc")]
        return {"case": case, "decoder": dec, "graph": dec.capture(1 + seed % (cfg.vocab - 1)), "kv": rows}
    w = torch.randn((case["n"], case["k"]), device="cuda", generator=gen) * 0.02
    return {"case": case, "w": w}


def run(state):
    kind = state["case"]["kind"]
    if kind in ("linear", "layer"):
        return [lin(x) for lin, x in zip(state["linears"], state["xs"])]
    if kind == "group":
        return state["group"].forward(state["case"]["rows"])
    if kind == "decode":
        dec = state["decoder"]
        state["graph"].replay()
        # The chosen token is left out: the largest of the fp16 logits are often equal, and then two correct
        # sums pick different ones.  Its value and all logits are here, and the cache rows the token added.
        return {"logits": dec.logits, "largest": dec.next_value, "hidden": dec.hidden_after_step(), "kv": state["kv"]}
    return pseudo_quantize_device(state["w"], state["case"]["bits"], state["case"]["g"], FIT_ITERS)


def _linear_bytes(n, k, bits, g):
    return bits * n * k // 8 + 2 * (bits + 1) * n * (k // g)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": _linear_bytes(n, k, case["bits"], case["g"]) + 2 * m * (n + k) + (2 * n if case["bias"] else 0),
                "flops": 2 * m * n * k}
    if kind in ("layer", "group"):
        m = case["rows"]
        shapes = [(n, _k_of(case, k)) for n, k in _shapes(case)]
        total = sum(_linear_bytes(n, k, case["bits"], case["g"]) + 2 * m * n for n, k in shapes)
        # x of q/k/v, of o, of gate/up and of down for the group; the layer's q/k/v and gate/up share theirs
        total += 2 * m * (sum(k for _, k in shapes) if kind == "group" else 2 * shapes[0][1] + (
            shapes[6][1] if shapes[6][1] != shapes[0][1] else 0))
        flops = 2 * m * sum(n * k for n, k in shapes)
        layers = case.get("layers", 1)
        return {"bytes": layers * total, "flops": layers * flops}
    if kind == "decode":
        h, f, q, kv = case["hidden"], case["ffn"], case["heads"] * 128, case["kv_heads"] * 128
        shapes = [(q, h), (kv, h), (kv, h), (h, q), (f, h), (f, h), (h, f)]
        layer = sum(_linear_bytes(n, k, case["bits"], case["g"]) for n, k in shapes) + 2 * 2 * kv * case["ctx"]
        return {"bytes": case["layers"] * layer + _linear_bytes(case["vocab"], h, 4, 128) + 2 * case["vocab"],
                "flops": 2 * case["layers"] * (sum(n * k for n, k in shapes) + 2 * q * case["ctx"]) + 2 * case["vocab"] * h}
    n, k, q, g = case["n"], case["k"], case["bits"], case["g"]
    # in: w; out: the reconstruction, one byte per bit, scales and offsets.  Per iteration a weight is
    # compared with 2^q values and enters q + 1 sums.
    return {"bytes": n * k * (4 + 4 + q) + 4 * n * (k // g) * (q + 1),
            "flops": FIT_ITERS * n * k * (2 * 2 ** q + q + 1)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("linear", "layer", "group"):
        # against a product in 64 bits: 1.7e-3 in bf16, 3e-4 in fp16 (weights and results rounded once each)
        return {"rel": 7e-3, "max": 0.02} if case.get("dtype") == "bf16" else {"rel": 1.2e-3, "max": 0.005}
    if kind == "decode":
        return {"rel": 1e-2, "max": 0.04}     # against the launch-per-op decoder 2.6e-3, run to run 1.8e-3
    # fits agree to 1e-7; a weight halfway between two values may go to either, which moves it by a step
    return {"rel": 1e-3, "max": 0.9, "differ": 1e-4}
