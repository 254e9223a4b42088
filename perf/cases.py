"""The work that programs built on this package have it do, as cases that can be timed.

Every case goes through the public entry points of ``fp6_marlin_b200`` the way a user's program calls
them: ``mul`` (b200 and reference layouts), ``mul_fused``, ``W46Linear``, ``make_w46_weight`` on the GPU and
the host codec ``quantize`` / ``prepacking`` / ``dequantize``.  Shapes are those of the benchmark
configurations (square layers, the Llama-2-7B and Llama-2-70B layer sets) or generic ones; activations are
N(0, 1), weights N(0, 0.02) with the FP6 columns scaled by 8, as in ``fp6_marlin_b200.synth``.
"""
import math

import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200.synth import algorithmic_bytes

MAX_FLOPS = 2 * 4096 * 16384 * 16384          # of the largest listed case


def _mul(name, m, k, n, qc=256, group=128, layout="b200"):
    case = {"kind": "mul", "m": m, "k": k, "n": n, "qc": qc, "group": group, "layout": layout}
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # one token of one sequence through an attention output projection: latency, launches and host time count
        _mul("mul 4096x4096 m1", 1, 4096, 4096),
        # small-batch decode on a square layer, the benchmark's headline shape
        _mul("mul 8192x8192 m16", 16, 8192, 8192),
        # the four projections of one Llama-2-7B decoder block for five sequences, with the fused neighbours:
        # a chain of short dependent GEMMs, the inner loop of token generation
        {"name": "7B block m5", "kind": "block", "m": 5, "hidden": 4096, "inter": 11008, "qc": 256},
        # the largest decode layer: the Llama-2-70B gate / up projection, a quarter of a gigabyte of weights
        _mul("mul 8192x57344 m16", 16, 8192, 57344),
        # continuous batching: a few dozen sequences through the 7B qkv projection
        _mul("mul 4096x12288 m48", 48, 4096, 12288),
        # a larger serving batch, not a multiple of any tile, through the 7B down projection
        _mul("mul 11008x4096 m100", 100, 11008, 4096),
        # a short prompt batch through the module wrapper: feature order restored, bias added
        {"name": "linear 4096->4096 3x67", "kind": "linear", "m": 67, "batch": 3, "k": 4096, "n": 4096, "qc": 256, "group": 128, "bias": True},
        # a prompt of odd length through the 7B gate / up projection
        _mul("mul 4096x22016 m777", 777, 4096, 22016),
        # compute-bound prefill, the largest shape of the prefill sweep that is run at every length
        _mul("mul 16384x16384 m4096", 4096, 16384, 16384),
        # the drop-in call: tensors packed the reference's way, one scale per output channel
        _mul("mul reference layout m8", 8, 4096, 4096, 256, -1, "reference"),
        # loading a model: quantise and pack one 7B gate projection on the GPU
        {"name": "pack 4096x11008", "kind": "pack", "k": 4096, "n": 11008, "qc": 256, "group": 128},
        # the reference's own preparation calls on host tensors, for a block of FP6 columns
        {"name": "host codec 4096x1024", "kind": "codec", "k": 4096, "n": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, of):
    return max(1, round(_log_int(rng, lo, hi) / of)) * of


def _fp6_columns(rng, n):
    # none, the usual widths, widths that leave both regions with a ragged last strip, or all columns
    pick = rng.random()
    if pick < 0.15:
        return -1
    if pick < 0.6:
        return rng.choice([128, 256, 512])
    if pick < 0.92:
        return 8 * rng.randint(1, 96)
    return n


def draw(rng):
    pick = rng.random()
    if pick < 0.58:
        while True:
            m, k, n = _log_int(rng, 1, 4096), _multiple(rng, 1024, 16384, 128), _multiple(rng, 1024, 28672, 256)
            if 2 * m * k * n <= MAX_FLOPS:
                return _mul(None, m, k, n, _fp6_columns(rng, n), -1 if rng.random() < 0.15 else 128)
    if pick < 0.68:
        m, k, n = _log_int(rng, 1, 256), _multiple(rng, 1024, 8192, 256), _multiple(rng, 1024, 8192, 256)
        return _mul(None, m, k, n, 64 * rng.randint(1, n // 64) if rng.random() < 0.3 else 256, -1, "reference")
    if pick < 0.80:
        return {"kind": "block", "m": _log_int(rng, 1, 512), "hidden": _multiple(rng, 1024, 8192, 256),
                "inter": _multiple(rng, 2816, 14336, 256), "qc": rng.choice([128, 256, 512])}
    if pick < 0.88:
        return {"kind": "linear", "m": _log_int(rng, 1, 600), "batch": rng.randint(1, 4), "k": _multiple(rng, 1024, 4096, 128),
                "n": _multiple(rng, 1024, 6144, 256), "qc": rng.choice([128, 256, 320]), "group": 128, "bias": rng.random() < 0.5}
    if pick < 0.95:
        return {"kind": "pack", "k": _multiple(rng, 1024, 8192, 128), "n": _multiple(rng, 1024, 14336, 256),
                "qc": rng.choice([128, 256, 512]), "group": 128}
    return {"kind": "codec", "k": _multiple(rng, 1024, 8192, 256), "n": _multiple(rng, 256, 1024, 256)}


def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def _activations(gen, *shape):
    return torch.randn(shape, generator=gen, dtype=torch.float32, device=gen.device).half()


def _weight(gen, k, n, qc):
    w = torch.randn((k, n), generator=gen, dtype=torch.float16, device=gen.device)
    w *= 0.02
    if qc > 0:
        w[:, n - qc:] *= 8.0
    return w


def _packed(gen, k, n, qc, group):
    return fm.make_w46_weight(_weight(gen, k, n, qc), qc, group, keep_dequantized=False, quant_device="cuda")


def _workspace(n):
    return torch.zeros(max(n // 128 * 16, 1), dtype=torch.int32, device="cuda")


def _reference_packed(gen, k, n, qc):
    # every bit pattern is a valid code; scales of the size that N(0, 0.02) weights have
    words = (k * (n - qc) // 2 + k * qc * 3 // 4) // 4
    B = torch.randint(-2**31, 2**31, (words,), generator=gen, dtype=torch.int64, device="cuda").to(torch.int32)
    s = (torch.rand(n, generator=gen, device="cuda") * 0.004 + 0.008).half()
    return B, s


def _empty(m, n):
    return torch.empty((m, n), dtype=torch.float16, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "codec":
        gen = _gen(seed, "cpu")
        x, s = fm.fake_quantize_fp6(_weight(gen, case["k"], case["n"], case["n"]))
        return {"kind": kind, "x": x.contiguous(), "s": s[:1].expand(case["n"]).contiguous()}
    gen = _gen(seed)
    if kind == "pack":
        return {"kind": kind, "w": _weight(gen, case["k"], case["n"], case["qc"]), "qc": case["qc"], "group": case["group"]}
    if kind == "linear":
        k, n = case["k"], case["n"]
        w = torch.randn((n, k), generator=gen, dtype=torch.float16, device="cuda") * 0.02
        w[torch.randperm(n, generator=gen, device="cuda")[: case["qc"]]] *= 8.0
        bias = _activations(gen, n) if case["bias"] else None
        layer = fm.W46Linear(w, case["qc"], case["group"], bias, quant_device="cuda").cuda()
        return {"kind": kind, "layer": layer, "x": _activations(gen, case["batch"], case["m"], k)}
    if kind == "block":
        m, h, i, qc = case["m"], case["hidden"], case["inter"], case["qc"]
        gate, up = (_weight(gen, h, i, qc // 2) for _ in range(2))
        return {"kind": kind, "qc": qc, "workspace": _workspace(max(3 * h, 2 * i)),
                "x": _activations(gen, m, h), "attended": _activations(gen, m, h),
                "w_qkv": _packed(gen, h, 3 * h, qc, 128), "w_o": _packed(gen, h, h, qc, 128),
                "w_gate_up": fm.make_gate_up_weight(gate, up, qc, 128, quant_device="cuda")[0],
                "w_down": _packed(gen, i, h, qc, 128),
                "qkv": _empty(m, 3 * h), "x1": _empty(m, h), "act": _empty(m, i), "x2": _empty(m, h)}
    m, k, n = case["m"], case["k"], case["n"]
    state = {"kind": kind, "A": _activations(gen, m, k), "C": _empty(m, n), "workspace": _workspace(n), "qc": case["qc"],
             "options": {"group_size": case["group"], "layout": case["layout"]}}
    if case["layout"] == "reference":
        state["B"], state["s"] = _reference_packed(gen, k, n, case["qc"])
    else:
        w = _packed(gen, k, n, case["qc"], case["group"])
        state["B"], state["s"] = w.B, w.s
    return state


def run(state):
    kind = state["kind"]
    if kind == "mul":
        fm.mul(state["A"], state["B"], state["C"], state["s"], state["workspace"], state["qc"], **state["options"])
        return state["C"]
    if kind == "block":
        qc, ws = state["qc"], state["workspace"]
        w = state["w_qkv"]
        fm.mul(state["x"], w.B, state["qkv"], w.s, ws, qc, group_size=128, layout="b200")
        w = state["w_o"]
        fm.mul_fused(state["attended"], w.B, state["x1"], w.s, ws, qc, epilogue="residual", residual=state["x"], group_size=128)
        w = state["w_gate_up"]
        fm.mul_fused(state["x1"], w.B, state["act"], w.s, ws, qc, epilogue="silu_mul", group_size=128)
        w = state["w_down"]
        fm.mul_fused(state["act"], w.B, state["x2"], w.s, ws, qc, epilogue="residual", residual=state["x1"], group_size=128)
        return [state["qkv"], state["x1"], state["act"], state["x2"]]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "pack":
        w = fm.make_w46_weight(state["w"], state["qc"], state["group"], keep_dequantized=False, quant_device="cuda")
        return [w.B, w.s]
    codes = fm.quantize(state["x"])
    n, k = state["s"].numel(), state["x"].numel() // state["s"].numel()
    stream = codes.view(n, k * 3 // 16)
    return [codes, fm.prepacking(stream), fm.dequantize(stream, state["s"])]


def work(case):
    kind = case["kind"]
    if kind == "codec":
        values = case["k"] * case["n"]
        return {"bytes": values * (2 + 0.75) + values * 1.5 + values * (0.75 + 2), "flops": values}
    if kind == "pack":
        k, n, qc = case["k"], case["n"], case["qc"]
        return {"bytes": 2 * k * n + algorithmic_bytes(0, k, n, qc, case["group"]), "flops": k * n}
    if kind == "block":
        m, h, i, qc = case["m"], case["hidden"], case["inter"], case["qc"]
        layers = [(h, 3 * h), (h, h), (h, 2 * i), (i, h)]
        nbytes = sum(algorithmic_bytes(m, k, n, qc, 128) for k, n in layers) + 2 * m * (2 * h - i)   # residuals read, half of gate / up written
        return {"bytes": nbytes, "flops": sum(2 * m * k * n for k, n in layers)}
    m = case["m"] * case.get("batch", 1)
    nbytes = algorithmic_bytes(m, case["k"], case["n"], case["qc"], case["group"])
    return {"bytes": nbytes + (2 * case["n"] if case.get("bias") else 0), "flops": 2 * m * case["k"] * case["n"]}


def tolerance(case):
    if case["kind"] in ("pack", "codec"):
        return "exact"
    # results are fp16 (half an ulp is 2.4e-4 on average over a binade) of fp32 sums; INT4 weights times their group
    # scale may be rounded to fp16 before the sums, which adds as much again.  The block chains three of them.
    return {"rel": 2e-3 if case["kind"] == "block" else 1e-3}
