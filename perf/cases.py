"""The packed linears as an engine calls them, at the sizes and in the forms it calls them.

Rows: one conditioning vector (the adaLN modulation), a short or ragged text prompt, and the image tokens of a
512 x 512 (1024 rows), 1024 x 1024 (4096) or 2048 x 2048 (16384) picture, with any number of rows between them for other
picture sizes, cropped prompts and stacked batches. Matrices: the 3072-wide block (qkv 9216, out 3072, fc1 12288, fc2
from 12288), its modulation (18432 x 3072), the 4096-wide block of the drop-in engine, and other sizes the operators
take (n a multiple of 32, k of 64 or 256). Float16 or float32 activations and results, packed or byte-wide weights, with
and without a bias. A case is a dict of plain values; `kind` says which entry points it goes through:

  linear      one record through `linear`, the dispatcher
  block       the four linears of one 3072-wide block through `linear`
  engine      the seven linears of one block of the drop-in engine (q, k, v share an input, gate and up share one) and
              the SwiGLU between them, fused into the quantiser of the last
  mlp         fc1, GELU fused into the quantiser of fc2, fc2
  modulation  the modulation linears of several blocks against one conditioning vector, in one call
  dropin      activation quantisation or conversion and a GEMM by the engine's four native symbols
"""
import importlib
import math

import torch

qi = importlib.import_module("qwen-image-cplus_b200")  # the folder's name has a hyphen

W4A16, W4A4 = qi.SCHEME_W4A16, qi.SCHEME_W4A4_H256
HIDDEN = 3072                 # the block of `block` and `mlp`; fc1 and fc2 are four times as wide
ENGINE, ENGINE_MLP = 4096, 12288
BLOCK_SHAPES = ((3 * HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (4 * HIDDEN, HIDDEN), (HIDDEN, 4 * HIDDEN))
NAMED_SHAPES = BLOCK_SHAPES + ((6 * HIDDEN, HIDDEN), (ENGINE, ENGINE), (ENGINE_MLP, ENGINE), (ENGINE, ENGINE_MLP))
LARGEST = 16384 * sum(n * k for n, k in BLOCK_SHAPES)  # multiply-adds of the largest listed case


def listed():
    return [
        # one block's adaLN modulation: a single row against a wide matrix, the smallest call and a very frequent one
        {"name": "modulation", "kind": "linear", "scheme": W4A16, "m": 1, "n": 6 * HIDDEN, "k": HIDDEN, "x": "f16", "y": "f16", "bias": True, "wide": False},
        # the same for all 60 blocks of a denoising step, which share the conditioning vector
        {"name": "modulation of a step", "kind": "modulation", "m": 1, "n": 6 * HIDDEN, "k": HIDDEN, "count": 60},
        # a handful of rows against a deep matrix (the pair of a guided step with its extra tokens), in the engine's float32
        {"name": "few rows", "kind": "linear", "scheme": W4A16, "m": 5, "n": ENGINE, "k": ENGINE_MLP, "x": "f32", "y": "f32", "bias": False, "wide": False},
        # a short, ragged text prompt through one linear of each scheme
        {"name": "prompt w4a16", "kind": "linear", "scheme": W4A16, "m": 77, "n": 4 * HIDDEN, "k": HIDDEN, "x": "f16", "y": "f16", "bias": True, "wide": False},
        {"name": "prompt w4a4", "kind": "linear", "scheme": W4A4, "m": 77, "n": 3 * HIDDEN, "k": HIDDEN, "x": "f16", "y": "f16", "bias": True, "wide": True},
        # one attention projection of a 512 x 512 picture
        {"name": "projection 1024", "kind": "linear", "scheme": W4A16, "m": 1024, "n": HIDDEN, "k": HIDDEN, "x": "f16", "y": "f16", "bias": True, "wide": False},
        # the drop-in engine at 512 x 512: one linear by its own symbols on nibble-packed codes, then a whole block
        {"name": "dropin w4a4 1024", "kind": "dropin", "scheme": W4A4, "m": 1024, "n": ENGINE_MLP, "k": ENGINE},
        {"name": "engine block 1024", "kind": "engine", "m": 1024, "wide": True},
        # the MLP of a 1024 x 1024 picture with its activation fused
        {"name": "mlp 4096", "kind": "mlp", "m": 4096},
        # a block of a 1024 x 1024 picture under each scheme, and of a 2048 x 2048 picture, the largest
        {"name": "block w4a16 4096", "kind": "block", "scheme": W4A16, "m": 4096},
        {"name": "block w4a4 4096", "kind": "block", "scheme": W4A4, "m": 4096},
        {"name": "block w4a4 16384", "kind": "block", "scheme": W4A4, "m": 16384},
    ]


def _spread(rng, low, high):
    """A whole number of low..high, evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "linear", "linear", "block", "engine", "mlp", "modulation", "dropin"))
    scheme = rng.choice((W4A16, W4A4))
    if kind == "linear":
        n, k = rng.choice(NAMED_SHAPES)
        if rng.random() < 0.5:
            step = 64 if scheme == W4A16 else 256
            n, k = 32 * _spread(rng, 16, 576), step * _spread(rng, 512 // step, 12288 // step)
        m = min(_spread(rng, 1, 16384), LARGEST // (n * k))
        return {"kind": kind, "scheme": scheme, "m": m, "n": n, "k": k, "x": rng.choice(("f16", "f32")), "y": rng.choice(("f16", "f32")),
                "bias": rng.random() < 0.5, "wide": scheme == W4A4 and rng.random() < 0.7}
    if kind == "block":
        return {"kind": kind, "scheme": scheme, "m": _spread(rng, 16, 8192)}
    if kind == "engine":
        return {"kind": kind, "m": _spread(rng, 16, 4096), "wide": rng.random() < 0.7}
    if kind == "mlp":
        return {"kind": kind, "m": _spread(rng, 16, 8192)}
    if kind == "modulation":
        return {"kind": kind, "m": rng.choice((1, 1, 2)), "n": 32 * _spread(rng, 64, 576), "k": 64 * _spread(rng, 16, 64), "count": _spread(rng, 2, 120)}
    n, k = rng.choice(((ENGINE, ENGINE), (ENGINE_MLP, ENGINE), (ENGINE, ENGINE_MLP)))
    return {"kind": kind, "scheme": scheme, "m": 128 * _spread(rng, 1, 32), "n": n, "k": k}


# ---- inputs ------------------------------------------------------------------------------------------------------

DTYPES = {"f16": torch.float16, "f32": torch.float32}
CODES = {"f16": qi.DTYPE_F16, "f32": qi.DTYPE_F32}


class _Maker:
    def __init__(self, seed):
        self.random = torch.Generator(device="cuda")
        self.random.manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, device="cuda", generator=self.random)

    def uniform(self, low, high, *shape):
        return torch.rand(*shape, device="cuda", generator=self.random) * (high - low) + low

    def activations(self, m, k, dtype="f16"):
        """Normal values, one channel in a hundred twenty times as large."""
        channels = torch.where(self.uniform(0.0, 1.0, k) < 0.01, 20.0, 1.0)
        return (self.normal(m, k) * channels).to(DTYPES[dtype])

    def conditioning(self, m, k):
        return torch.nn.functional.silu(self.normal(m, k)).half()

    def record(self, scheme, n, k, bias=False, wide=False):
        """What quantising normal weights of deviation 0.02 gives: codes of a bell shape, one scale (and minimum) for 64 of them."""
        scales = self.uniform(0.9, 1.1, n, k // 64)
        if scheme == W4A4:
            codes, zeros = (self.normal(n, k) * 2.7).round_().clamp_(-7, 7), None
            scales = (scales * (0.02 / 2.7)).half()
        else:
            codes = (self.normal(n, k) * 3.1 + 7.5).round_().clamp_(0, 15)
            scales = (scales * (0.02 / 3.1)).half()
            zeros = (scales.float() * self.uniform(-7.8, -7.2, n, k // 64)).half()
        codes = codes.to(torch.int8).bitwise_and_(15).view(torch.uint8)
        packed = codes[:, 0::2] | (codes[:, 1::2] << 4)
        widened = None
        if wide:  # once for each matrix, when it is loaded
            widened = torch.empty(n, k, dtype=torch.uint8, device="cuda")
            _ok(qi.w4a4_widen_codes_ex(packed, widened, n, k))
        return qi.PackedLinear(scheme, n, k, packed, scales, zeros, self.normal(n) * 0.01 if bias else None, weights_wide=widened)


def _ok(status):
    if status != 0:
        raise RuntimeError(f"status {status}")


def _work(m, k):
    """The activation arena an engine keeps, for inputs up to k wide."""
    return qi.LinearWork(torch.empty(m, k // 2, dtype=torch.uint8, device="cuda"), torch.empty(m, k // 64, dtype=torch.float16, device="cuda"),
                         torch.empty(m, k, dtype=torch.float16, device="cuda"), torch.empty(m, k, dtype=torch.uint8, device="cuda"))


def _result(m, n, dtype):
    return torch.zeros(m, n, dtype=DTYPES[dtype], device="cuda")


def prepare(case, seed):
    make, kind, m = _Maker(seed), case["kind"], case["m"]
    state = {"case": case}
    if kind == "linear":
        n, k = case["n"], case["k"]
        state["record"] = make.record(case["scheme"], n, k, case["bias"], case["wide"])
        state["x"] = make.conditioning(m, k).to(DTYPES[case["x"]]) if m <= 2 else make.activations(m, k, case["x"])
        state["work"], state["y"] = _work(m, k), _result(m, n, case["y"])
    elif kind == "block":
        state["records"] = [make.record(case["scheme"], n, k, bias=True, wide=case["scheme"] == W4A4) for n, k in BLOCK_SHAPES]
        attention_in, attention_out, mlp_in = (make.activations(m, HIDDEN) for _ in range(3))
        hidden = torch.nn.functional.gelu(make.normal(m, 4 * HIDDEN), approximate="tanh").half()
        state["xs"] = [attention_in, attention_out, mlp_in, hidden]
        state["work"], state["ys"] = _work(m, 4 * HIDDEN), [_result(m, n, "f16") for n, _ in BLOCK_SHAPES]
    elif kind == "engine":
        shapes = {"q": (ENGINE, ENGINE), "k": (ENGINE, ENGINE), "v": (ENGINE, ENGINE), "o": (ENGINE, ENGINE),
                  "gate": (ENGINE_MLP, ENGINE), "up": (ENGINE_MLP, ENGINE), "down": (ENGINE, ENGINE_MLP)}
        state["records"] = {role: make.record(W4A4, n, k, wide=case["wide"]) for role, (n, k) in shapes.items()}
        state["xs"] = {role: make.activations(m, ENGINE, "f32") for role in ("q", "o", "gate")}
        state["ys"] = {role: _result(m, n, "f32") for role, (n, _) in shapes.items()}
        work = _work(m, ENGINE_MLP)
        state["work"] = work if case["wide"] else qi.LinearWork(work.codes, work.code_scales, work.halves)
    elif kind == "mlp":
        state["records"] = [make.record(W4A4, n, k, bias=True, wide=True) for n, k in BLOCK_SHAPES[2:]]
        state["x"], state["work"] = make.activations(m, HIDDEN), _work(m, 4 * HIDDEN)
        state["hidden"], state["y"] = _result(m, 4 * HIDDEN, "f32"), _result(m, HIDDEN, "f16")
    elif kind == "modulation":
        n, k = case["n"], case["k"]
        state["records"] = [make.record(W4A16, n, k, bias=True) for _ in range(case["count"])]
        state["x"], state["ys"] = make.conditioning(m, k), torch.zeros(case["count"], m, n, dtype=torch.float16, device="cuda")
        state["items"] = qi.gemv_items([(r.weights, r.scales, r.zeros, r.bias, y) for r, y in zip(state["records"], state["ys"])])
    else:
        n, k = case["n"], case["k"]
        state["record"], state["x"] = make.record(case["scheme"], n, k), make.activations(m, k, "f32")
        state["work"], state["y"] = _work(m, k), _result(m, n, "f32")
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind, m = case["kind"], case["m"]
    if kind == "linear":
        _ok(qi.linear(state["record"], state["work"], state["x"], state["y"], m, input_dtype=CODES[case["x"]], output_dtype=CODES[case["y"]]))
        return state["y"]
    if kind == "block":
        for record, x, y in zip(state["records"], state["xs"], state["ys"]):
            _ok(qi.linear(record, state["work"], x, y, m, input_dtype=qi.DTYPE_F16, output_dtype=qi.DTYPE_F16))
        return state["ys"]
    if kind == "engine":
        records, work, xs, ys = state["records"], state["work"], state["xs"], state["ys"]
        for role, source in (("q", "q"), ("k", "q"), ("v", "q"), ("o", "o"), ("gate", "gate"), ("up", "gate")):
            _ok(qi.linear(records[role], work, xs[source], ys[role], m, reuse_input=role != source))
        _ok(qi.w4a4_swiglu_quantize_ex(ys["gate"], ys["up"], work.codes, work.code_scales, work.wide, m, ENGINE_MLP))
        _ok(qi.linear(records["down"], work, ys["gate"], ys["down"], m, reuse_input=True))
        return ys
    if kind == "mlp":
        (fc1, fc2), work = state["records"], state["work"]
        _ok(qi.linear(fc1, work, state["x"], state["hidden"], m, input_dtype=qi.DTYPE_F16))
        _ok(qi.w4a4_gelu_quantize_ex(state["hidden"], work.codes, work.code_scales, work.wide, m, 4 * HIDDEN))
        _ok(qi.linear(fc2, work, state["hidden"], state["y"], m, reuse_input=True, output_dtype=qi.DTYPE_F16))
        return state["hidden"], state["y"]
    if kind == "modulation":
        _ok(qi.w4a16_gemv_grouped_ex(state["x"], state["items"][0], qi.DTYPE_F16, case["n"], m, case["n"], case["k"]))
        return state["ys"]
    record, work, n, k = state["record"], state["work"], case["n"], case["k"]
    if case["scheme"] == W4A4:
        _ok(qi.w4a4_quantize_activations(state["x"], work.codes, work.code_scales, m, k))
        _ok(qi.w4a4_gemm(work.codes, work.code_scales, record.weights, record.scales, state["y"], m, n, k))
    else:
        _ok(qi.f32_to_f16(state["x"], work.halves, m * k))
        _ok(qi.w4a16_gemm(work.halves, record.weights, record.scales, record.zeros, state["y"], m, n, k))
    return state["y"]


# ---- what a pass cannot do without, and how far another implementation's results may be off ---------------------------


def _matrix_bytes(scheme, n, k):
    """Packed codes and scales; the byte-wide copy some cases hold says no more than the packed codes do."""
    return n * k / 2 + n * k / 64 * (4 if scheme == W4A16 else 2)


def work(case):
    kind, m = case["kind"], case["m"]
    size = {"f16": 2, "f32": 4}
    if kind == "linear":
        n, k = case["n"], case["k"]
        return {"bytes": m * k * size[case["x"]] + _matrix_bytes(case["scheme"], n, k) + m * n * size[case["y"]] + (4 * n if case["bias"] else 0),
                "flops": 2.0 * m * n * k}
    if kind == "block":
        return {"bytes": sum(2 * m * (n + k) + _matrix_bytes(case["scheme"], n, k) + 4 * n for n, k in BLOCK_SHAPES), "flops": 2.0 * m * sum(n * k for n, k in BLOCK_SHAPES)}
    if kind == "engine":
        shapes = 4 * [(ENGINE, ENGINE)] + 2 * [(ENGINE_MLP, ENGINE)] + [(ENGINE, ENGINE_MLP)]
        activations = 4 * m * (3 * ENGINE + 2 * ENGINE_MLP) + 4 * m * sum(n for n, _ in shapes)
        return {"bytes": activations + sum(_matrix_bytes(W4A4, n, k) for n, k in shapes), "flops": 2.0 * m * sum(n * k for n, k in shapes)}
    if kind == "mlp":
        wide = 4 * HIDDEN
        return {"bytes": 2 * m * HIDDEN + 2 * 4 * m * wide + 2 * m * HIDDEN + 2 * _matrix_bytes(W4A4, wide, HIDDEN) + 4 * (wide + HIDDEN), "flops": 4.0 * m * wide * HIDDEN}
    if kind == "modulation":
        n, k, count = case["n"], case["k"], case["count"]
        return {"bytes": 2 * m * k + count * (_matrix_bytes(W4A16, n, k) + 4 * n + 2 * m * n), "flops": 2.0 * m * n * k * count}
    n, k = case["n"], case["k"]
    return {"bytes": 4 * m * (n + k) + _matrix_bytes(case["scheme"], n, k), "flops": 2.0 * m * n * k}


def tolerance(case):
    """Activation codes are whole numbers that every implementation finds alike from the same activations; what differs is
    the order of the float32 sums (the tensor cores' own alignment included) and, where the result is float16, which way a
    value near a tie is rounded. In `engine` and `mlp` four-bit codes are made from such sums, and a sum near a tie may
    move a code."""
    kind = case["kind"]
    if kind in ("block", "modulation") or kind == "linear" and case["y"] == "f16":
        return {"rel": 1e-3, "max": 2e-3}
    if kind in ("engine", "mlp"):
        return {"rel": 1e-3, "max": 5e-2}
    return {"rel": 1e-5, "max": 1e-4} if case.get("scheme", W4A4) == W4A4 else {"rel": 3e-5, "max": 3e-4}
