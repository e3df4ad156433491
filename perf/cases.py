"""The work that a user of this package has it do, as timed cases through the public entry points.

Kinds of case:

* ``decode``   a serving step: ``E8LatticeLinear`` on 1 to 16 rows without gradients
* ``block``    decode of transformer blocks with ``ops.GroupedGemv``: q/k/v, o, gate/up and down as one launch each
* ``prefill``  ``E8LatticeLinear`` on a batch of prompt tokens without gradients
* ``train``    fine-tuning step of a layer with an adapter: forward, then the gradients of x and of both adapter factors
* ``pack``     a dense weight to codes and scales with the format's packer
* ``unpack``   codes and scales back to a dense weight

Activations are normal with a few channels 20 times larger than the rest, as transformer activations have them;
weights are normal with a standard deviation of 1 / sqrt(in_features).
"""

import importlib
import math

import torch

pkg = importlib.import_module("ojasx-open-source-cuda_b200")

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_BYTES = {"bf16": 2, "f16": 2, "f32": 4}
_PACKERS = {1.0: "RootE8LatticePacker", 1.5: "TernaryE8LatticePacker", 2.0: "E8LatticePacker"}


def _layer(name, kind, rows, k, n, bits=1.5, group=32, dtype="bf16", bias=False, hadamard=False, rank=0):
    c = {"kind": kind, "rows": rows, "k": k, "n": n, "bits": bits, "group": group, "dtype": dtype, "bias": bias,
         "hadamard": hadamard, "rank": rank}
    return dict(c, name=name) if name else c


def _weight(name, kind, n, k, bits, group, dtype):
    c = {"kind": kind, "n": n, "k": k, "bits": bits, "group": group, "dtype": dtype}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one token through a key/value projection of an 8B model: the smallest call there is, latency counts
        _layer("decode_kv_row1", "decode", 1, 4096, 1024),
        # sixteen sequences through the down projection of an 8B model
        _layer("decode_down_rows16", "decode", 16, 14336, 4096),
        # E8LatticeLinear(in, out) as it is without further arguments: 2.0 bits, one scale per 8 weights, a bias
        _layer("decode_default_row1", "decode", 1, 4096, 4096, bits=2.0, group=8, bias=True),
        # the smallest format on a large model's gate projection, eight sequences
        _layer("decode_1bit_rows8", "decode", 8, 8192, 28672, bits=1.0),
        # a fine-tuned layer at inference: rotated weights, adapter of rank 16
        _layer("decode_adapter_rows4", "decode", 4, 4096, 4096, dtype="f16", hadamard=True, rank=16),
        # four blocks of an 8B model, one token: the serving loop
        {"name": "block_8b_row1", "kind": "block", "rows": 1, "hidden": 4096, "kv": 1024, "inter": 14336, "layers": 4, "dtype": "bf16"},
        # a prompt of 2048 tokens through the gate projection of an 8B model
        _layer("prefill_gate_2048", "prefill", 2048, 4096, 14336),
        # a short prompt of odd length, features that are multiples of 32 but not of 256 (as many small models have them)
        _layer("prefill_ragged_333", "prefill", 333, 2912, 2000, bits=1.5, bias=True),
        # fine-tuning as pack_model_e8 sets it up (2.0 bits, groups of 32) with an adapter of rank 16
        _layer("train_down_1024", "train", 1024, 14336, 4096, bits=2.0, rank=16),
        # packing a large model's weight in its checkpoint's type
        _weight("pack_ternary_70b_gate", "pack", 28672, 8192, 1.5, 32, "f16"),
        # packing into the smallest format
        _weight("pack_1bit_8b", "pack", 4096, 4096, 1.0, 32, "bf16"),
        # back to the default type; odd sizes, so groups run across rows and the last one is padded
        _weight("unpack_2bit_odd", "unpack", 4001, 3003, 2.0, 8, "f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _features(rng, lo, hi, step):
    return max(step, _log(rng, lo, hi) // step * step)


# no drawn case has more multiply-adds than the listed case of its kind (or weights, where they are what counts)
_MOST = {"decode": 16 * 8192 * 28672, "prefill": 2048 * 4096 * 14336, "train": 1024 * 14336 * 4096}
_MOST_RAGGED = 333 * 2912 * 2000


def _draw_layer(rng, kind):
    bits = rng.choice([1.5, 1.5, 2.0, 1.0])
    group = rng.choice([32, 32, 32, 8])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    lo, hi = {"decode": (1, 16), "prefill": (17, 4096), "train": (32, 2048)}[kind]
    # features: mostly multiples of 256, as large models have them, else of 32
    ragged = kind != "train" and rng.random() < 0.25
    step = 32 if ragged else 256
    while True:
        rows, k, n = _log(rng, lo, hi), _features(rng, 512, 16384, step), _features(rng, 256, 28672, 8 if ragged else 64)
        if rows * k * n <= (_MOST_RAGGED if ragged and kind == "prefill" else _MOST[kind]) and k * n <= 8192 * 28672:
            break
    rank = rng.choice([8, 16, 32]) if kind == "train" or rng.random() < 0.2 else 0
    return _layer(None, kind, rows, k, n, bits, group, dtype, rng.random() < 0.3, rng.random() < 0.2, rank)


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "train", "block", "pack", "pack", "unpack"])
    if kind in ("decode", "prefill", "train"):
        return _draw_layer(rng, kind)
    if kind == "block":
        hidden = _features(rng, 1024, 6144, 256)
        inter = _features(rng, 2 * hidden, 4 * hidden, 256)
        return {"kind": kind, "rows": _log(rng, 1, 16), "hidden": hidden, "kv": hidden // rng.choice([1, 4]), "inter": inter,
                "layers": rng.randint(1, 2), "dtype": rng.choice(["bf16", "bf16", "f16"])}
    bits = rng.choice([1.5, 1.5, 2.0, 1.0])
    most = 28672 * 8192 if bits != 1.0 or kind == "unpack" else 14336 * 4096
    odd = rng.random() < 0.3
    while True:
        n, k = _log(rng, 256, 28672), _log(rng, 512, 16384)
        if not odd:
            n, k = max(64, n // 64 * 64), max(256, k // 256 * 256)
        if n * k <= most:
            break
    return _weight(None, kind, n, k, bits, rng.choice([32, 32, 8]), rng.choice(["bf16", "f16", "f32"]))


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype).mul_(std)


def _activations(g, rows, k, dtype):
    x = _randn(g, rows, k)
    x[:, torch.randint(0, k, (max(1, k // 512),), generator=g, device="cuda")] *= 20.0
    return x.to(dtype)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind, dt = case["kind"], _DTYPES[case["dtype"]]
    with torch.no_grad():
        if kind == "block":
            return _prepare_block(case, g, dt)
        n, k = case["n"], case["k"]
        w = _randn(g, n, k, std=k ** -0.5, dtype=dt)
        if kind in ("pack", "unpack"):
            packer = getattr(pkg, _PACKERS[case["bits"]])
            if kind == "pack":
                return {"kind": kind, "call": lambda: packer.pack(w, case["group"])[:2]}
            packed, scales, shape = packer.pack(w, case["group"])
            return {"kind": kind, "call": lambda: packer.unpack(packed, scales, shape, dt)}
        dense = torch.nn.utils.skip_init(torch.nn.Linear, k, n, bias=case["bias"], device="cuda", dtype=dt)
        dense.weight.copy_(w)
        if case["bias"]:
            dense.bias.copy_(_randn(g, n, std=0.1))
        layer = pkg.E8LatticeLinear.from_linear(dense, rank=case["rank"], group_size=case["group"], bitrate=case["bits"],
                                                use_hadamard=case["hadamard"])
        if case["rank"]:
            layer.lora_A.copy_(_randn(g, k, case["rank"], std=k ** -0.5))
            layer.lora_B.copy_(_randn(g, case["rank"], n, std=0.02))
        layer.requires_grad_(False)
        x = _activations(g, case["rows"], k, dt)
        if kind != "train":
            return {"kind": kind, "layer": layer.eval(), "x": x}
        layer.lora_A.requires_grad_(True)
        layer.lora_B.requires_grad_(True)
        return {"kind": kind, "layer": layer, "x": x.requires_grad_(True), "gy": _randn(g, case["rows"], n, std=0.01).to(dt)}


def _prepare_block(case, g, dt):
    m, h, kv, inter = case["rows"], case["hidden"], case["kv"], case["inter"]

    def matrix(n, k):
        packed, scales, _ = pkg.TernaryE8LatticePacker.pack(_randn(g, n, k, std=k ** -0.5, dtype=dt), 32)
        return packed, scales, n, k

    def buffer(n):
        return torch.empty(m, n, dtype=dt, device="cuda")

    def group(x, ys, mats):
        return pkg.ops.GroupedGemv([(x, p, s, None, y) for y, (p, s, _, _) in zip(ys, mats)], [(n, k) for _, _, n, k in mats],
                                   static_weights=True)

    x, launches, out = _activations(g, m, h, dt), [], []
    for _ in range(case["layers"]):
        q, key, val, a, gate, up, y = buffer(h), buffer(kv), buffer(kv), buffer(h), buffer(inter), buffer(inter), buffer(h)
        launches += [group(x, [q, key, val], [matrix(h, h), matrix(kv, h), matrix(kv, h)]), group(q, [a], [matrix(h, h)]),
                     group(a, [gate, up], [matrix(inter, h), matrix(inter, h)]), group(up, [y], [matrix(h, inter)])]
        out += [key, val, gate, y]
        x = y
    return {"kind": "block", "launches": launches, "out": out}


def run(state):
    kind = state["kind"]
    if kind == "block":
        for launch in state["launches"]:
            launch()
        return state["out"]
    if kind in ("pack", "unpack"):
        return state["call"]()
    layer = state["layer"]
    if kind == "train":
        y = layer(state["x"])
        return [y, *torch.autograd.grad(y, [state["x"], layer.lora_A, layer.lora_B], state["gy"])]
    with torch.no_grad():
        return layer(state["x"])


def _group(bits, group):
    return max(16, group) if bits == 1.5 else group


def _packed(n, k, bits, group):
    return n * k * bits / 8 + n * k / _group(bits, group) * 2


def work(case):
    kind, e = case["kind"], _BYTES[case["dtype"]]
    if kind == "block":
        m, h, kv, inter = case["rows"], case["hidden"], case["kv"], case["inter"]
        shapes = [(h, h), (kv, h), (kv, h), (h, h), (inter, h), (inter, h), (h, inter)]
        ends = [(h, h + 2 * kv), (h, h), (h, 2 * inter), (inter, h)]
        return {"bytes": case["layers"] * (sum(_packed(n, k, 1.5, 32) for n, k in shapes) + sum(m * e * (i + o) for i, o in ends)),
                "flops": case["layers"] * sum(2 * m * n * k for n, k in shapes)}
    n, k = case["n"], case["k"]
    packed = _packed(n, k, case["bits"], case["group"])
    if kind in ("pack", "unpack"):
        return {"bytes": n * k * e + packed, "flops": 0}
    m, r = case["rows"], case["rank"]
    adapter = r * (n + k)
    if kind == "train":                        # x, dY, the adapter in; y, dX, the adapter's gradients out; the weights in each direction
        return {"bytes": 2 * packed + e * (2 * m * (n + k) + 2 * adapter), "flops": 4 * m * n * k + 6 * m * adapter}
    return {"bytes": packed + e * (m * (n + k) + adapter + (n if case["bias"] else 0)), "flops": 2 * m * (n * k + adapter)}


def tolerance(case):
    if case["kind"] in ("pack", "unpack"):
        return "exact"
    # one rounding to the 16-bit output; several of them where an adapter or a chain of layers is in between
    chain = case["kind"] in ("block", "train") or case["rank"] > 0
    if case["dtype"] == "bf16":
        return {"rel": 1e-2 if chain else 5e-3}
    return {"rel": 2e-3 if chain else 1e-3}
