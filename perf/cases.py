"""The calls that a training program makes of this package, as plain cases that can be timed and compared.

Four kinds of call carry the work of a low-precision training run:

* ``linear``   - one linear layer, forward and backward (or forward alone, as an evaluation pass runs it);
* ``moe``      - one expert-grouped linear, forward and backward, on a routed token buffer;
* ``quantize`` - quantise and dequantise one tensor, as weight de-oscillation and inspection tools do;
* ``gemm``     - quantise two operands and multiply them, the pair of public ops below the linear.

Every case is a dict of plain values.  Inputs have the distributions of the benchmark: activations
N(0, 1), weights N(0, 0.02), upstream gradients N(0, 1e-3).
"""
from __future__ import annotations

import math

import torch

from alto_b200 import grouped, mxfp4, mxfp8, nvfp4

DEVICE = "cuda"
STD = {"x": 1.0, "w": 0.02, "dy": 1e-3}


# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------
def _linear(recipe, m, k, n, backward=True, hadamard=0, sr=False, weight_2d=True):
    return {"op": "linear", "recipe": recipe, "m": m, "k": k, "n": n, "backward": backward, "hadamard": hadamard,
            "sr": sr, "weight_2d": weight_2d}


def _moe(recipe, experts, tokens, top_k, k, n, hadamard=0, sr=False):
    return {"op": "moe", "recipe": recipe, "experts": experts, "tokens": tokens, "top_k": top_k, "k": k, "n": n,
            "hadamard": hadamard, "sr": sr}


def _quantize(fmt, rows, cols, axis, blocks_2d, dtype):
    return {"op": "quantize", "format": fmt, "rows": rows, "cols": cols, "axis": axis, "blocks_2d": blocks_2d,
            "dtype": dtype}


def _gemm(recipe, m, k, n):
    return {"op": "gemm", "recipe": recipe, "m": m, "k": k, "n": n}


def listed():
    cases = {
        # a layer of a small or debugging model: every kernel is tiny, launches and host work count
        "linear_nvfp4_small": _linear("nvfp4", 256, 512, 384, hadamard=16, sr=True),
        # an evaluation pass on a short batch: weights quantised per call, no gradients
        "linear_nvfp4_eval_512": _linear("nvfp4", 512, 4096, 14336, backward=False, hadamard=16, sr=True),
        # the benchmark: Llama-3-8B MLP-up
        "linear_nvfp4_mlp_up": _linear("nvfp4", 8192, 4096, 14336, hadamard=16, sr=True),
        # Llama-3-8B key / value projection at batch 4 x 8192: many tokens, few output features
        "linear_nvfp4_kv_proj": _linear("nvfp4", 32768, 4096, 1024, hadamard=16, sr=True),
        # MLP-down with the MXFP4 recipe, a token count that fills no tile
        "linear_mxfp4_mlp_down": _linear("mxfp4", 8096, 14336, 4096, hadamard=16, sr=True),
        # Llama-3-8B attention output with MXFP8
        "linear_mxfp8_attn_out": _linear("mxfp8", 8192, 4096, 4096),
        # MLP-up with the two-level MXFP4 recipe
        "linear_two_level_mlp_up": _linear("mxfp4_two_level", 8192, 4096, 14336, hadamard=16, sr=True),
        # GPT-OSS-20B gate+up experts, the two-level MXFP4 recipe as its configuration writes it
        "moe_two_level_gate_up": _moe("mxfp4_two_level", 32, 16384, 4, 2880, 5760, hadamard=32, sr=True),
        # GPT-OSS-20B down experts on a short batch, MXFP8: few rows an expert
        "moe_mxfp8_down_short": _moe("mxfp8", 32, 2048, 4, 2880, 2880),
        # the first configuration: quantise both operands in 1-D blocks of 32, multiply
        "gemm_mxfp4_2048": _gemm("mxfp4", 2048, 2048, 2048),
        # de-oscillation's round trip of a master weight
        "quantize_nvfp4_weight": _quantize("nvfp4", 14336, 4096, -1, True, "float32"),
        # an odd number of rows, blocks along them left whole: inspection of an activation
        "quantize_mxfp8_rows_odd": _quantize("mxfp8_e5m2", 4099, 2880, -1, False, "bfloat16"),
    }
    return [{"name": name, **case} for name, case in cases.items()]


def _spread(rng, low, high, step):
    """A multiple of ``step`` in [low, high], even over its logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high, max(low, int(round(v / step)) * step))


_MAX_PRODUCT = 8192 * 4096 * 14336          # of m, k, n of the largest dense case
_MAX_ROUTED = 16384 * 4 * 2880 * 5760       # of routed rows, k, n of the largest expert case


def draw(rng):
    op = rng.choices(["linear", "moe", "quantize", "gemm"], [6, 3, 2, 1])[0]
    if op == "linear":
        recipe = rng.choice(["nvfp4", "nvfp4", "mxfp4", "mxfp8", "mxfp4_two_level"])
        k, n = _spread(rng, 256, 14336, 32), _spread(rng, 256, 14336, 32)
        m = _spread(rng, 32, 32768, 32)
        m = max(32, min(m, _MAX_PRODUCT // (k * n) // 32 * 32))
        fp4 = recipe != "mxfp8"
        return _linear(recipe, m, k, n, backward=rng.random() < 0.8, hadamard=16 if fp4 else 0,
                       sr=fp4 and rng.random() < 0.75, weight_2d=rng.random() < 0.75)
    if op == "moe":
        recipe = rng.choice(["nvfp4", "mxfp4", "mxfp8", "mxfp4_two_level"])
        k, n = _spread(rng, 256, 5760, 32), _spread(rng, 256, 5760, 32)
        top_k = rng.randint(1, 4)
        tokens = _spread(rng, 256, 16384, 32)
        tokens = max(256, min(tokens, _MAX_ROUTED // (k * n * top_k) // 32 * 32))
        fp4 = recipe != "mxfp8"
        return _moe(recipe, rng.choice([4, 8, 16, 32]), tokens, top_k, k, n,
                    hadamard=rng.choice([16, 32]) if fp4 else 0, sr=fp4)
    if op == "quantize":
        fmt = rng.choice(["nvfp4", "mxfp4", "mxfp8_e4m3", "mxfp8_e5m2"])
        axis = rng.choice([-1, -2])
        blocks_2d = axis == -1 and rng.random() < 0.4
        rows = _spread(rng, 64, 16384, 1 if axis == -1 and not blocks_2d else 32)
        return _quantize(fmt, rows, _spread(rng, 64, 8192, 32), axis, blocks_2d, rng.choice(["bfloat16", "float32"]))
    k, n = _spread(rng, 256, 8192, 32), _spread(rng, 256, 8192, 32)
    return _gemm(rng.choice(["mxfp4", "mxfp8"]), _spread(rng, 32, 8192, 32), k, n)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _normal(gen, shape, std, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=gen, device=DEVICE) * std).to(dtype)


def _route(gen, experts, tokens, top_k):
    """(destination row of every routed row, end of every expert's run): softmax top-k of N(0, 1) router
    logits, runs sorted by expert and padded to whole groups of 128 rows, as the grouped GEMMs want them."""
    logits = torch.randn(tokens, experts, generator=gen, device=DEVICE)
    expert = torch.topk(torch.softmax(logits, -1), top_k, dim=-1).indices.reshape(-1)
    counts = torch.bincount(expert, minlength=experts)
    padded = (counts + grouped.ALIGN_SIZE_M - 1) // grouped.ALIGN_SIZE_M * grouped.ALIGN_SIZE_M
    ends = torch.cumsum(padded, 0)
    order = torch.sort(expert, stable=True).values
    within = torch.arange(order.numel(), device=DEVICE) - (torch.cumsum(counts, 0) - counts)[order]
    return (ends - padded)[order] + within, ends.to(torch.int32)


def _buffer_rows(case):
    # the routed buffer has room for the worst padding, so its size does not depend on the routing
    return case["tokens"] * case["top_k"] + case["experts"] * grouped.ALIGN_SIZE_M


def _inputs(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    op = case["op"]
    if op == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"x": _normal(gen, (m, k), STD["x"]), "w": _normal(gen, (n, k), STD["w"]),
                "dy": _normal(gen, (m, n), STD["dy"]) if case["backward"] else None}
    if op == "moe":
        k, n, experts = case["k"], case["n"], case["experts"]
        rows, offs = _route(gen, experts, case["tokens"], case["top_k"])
        x = torch.zeros(_buffer_rows(case), k, dtype=torch.bfloat16, device=DEVICE)
        dy = torch.zeros(_buffer_rows(case), n, dtype=torch.bfloat16, device=DEVICE)
        x[rows] = _normal(gen, (rows.numel(), k), STD["x"])
        dy[rows] = _normal(gen, (rows.numel(), n), STD["dy"])
        return {"x": x, "w": _normal(gen, (experts, n, k), STD["w"]), "dy": dy, "offs": offs}
    if op == "quantize":
        return {"x": _normal(gen, (case["rows"], case["cols"]), STD["w"], getattr(torch, case["dtype"]))}
    return {"x": _normal(gen, (case["m"], case["k"]), STD["x"]), "w": _normal(gen, (case["n"], case["k"]), STD["x"])}


def prepare(case, seed):
    state = _inputs(case, seed)
    state.update(case=case, seed=seed)
    if case["op"] == "moe" or (case["op"] == "linear" and case["backward"]):
        state["x"].requires_grad_(True)
        state["w"].requires_grad_(True)
    return state


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _seed_draws(state):
    """Hadamard signs and stochastic rounding draw from two host generators.  A program that replays a step
    (recomputation of activations, a resumed run) sets them, and only then do two passes agree."""
    case = state["case"]
    if case["hadamard"]:
        nvfp4.HadamardFactory.configure(block_size=case["hadamard"], randomized=True, dtype=torch.float32,
                                        seed=state["seed"])
    if case["sr"]:
        torch.default_generator.manual_seed(state["seed"])


def _call_linear(state):
    case, x, w = state["case"], state["x"], state["w"]
    recipe, rht, sr, w2d = case["recipe"], case["hadamard"] > 0, case["sr"], case["weight_2d"]
    if recipe == "nvfp4":
        return nvfp4._to_nvfp4_then_scaled_mm(x, w, False, w2d, sr, use_outer_scale=True, use_hadamard=rht)
    if recipe == "mxfp8":
        return mxfp8._to_mxfp8_then_scaled_mm(x, w, "e4m3", False, False, w2d)
    return mxfp4._to_mxfp4_then_scaled_mm(x, w, False, w2d, sr, False, "none", rht,
                                          use_macro_block_scaling=recipe == "mxfp4_two_level")


def _call_moe(state):
    # experts hold their weights as [out, in] like a linear layer and hand a transposed view to the call
    case, x, w, offs = state["case"], state["x"], state["w"].transpose(-2, -1), state["offs"]
    recipe, rht, sr = case["recipe"], case["hadamard"] > 0, case["sr"]
    if recipe == "nvfp4":
        return grouped._quantize_then_nvfp4_scaled_grouped_mm(x, w, offs, False, True, sr, use_outer_scale=True,
                                                              use_hadamard=rht)
    if recipe == "mxfp8":
        return grouped._quantize_then_mxfp8_scaled_grouped_mm(x, w, offs, bwd_grad_format="e5m2")
    return grouped._quantize_then_mxfp_scaled_grouped_mm(x, w, offs, False, True, sr, False, rht, "none",
                                                         recipe == "mxfp4_two_level")


def _step(state, call):
    _seed_draws(state)
    if state["dy"] is None:
        with torch.no_grad():
            return call(state)
    y = call(state)
    dx, dw = torch.autograd.grad(y, (state["x"], state["w"]), state["dy"])
    return y.detach(), dx, dw


def _quantize_round_trip(state):
    case, x = state["case"], state["x"]
    fmt, axis, blocks_2d = case["format"], case["axis"], case["blocks_2d"]
    if fmt == "nvfp4":
        outer = torch.empty(1, dtype=torch.float32, device=x.device)
        codes, scales = nvfp4.convert_to_nvfp4(x, axis=axis, is_2d_block=blocks_2d, outer_scale=outer,
                                               update_outer_scale=True)
        back = nvfp4.convert_from_nvfp4(codes, scales, x.dtype, axis=axis, is_2d_block=blocks_2d, outer_scale=outer)
        return codes, scales, back, outer
    if fmt == "mxfp4":
        codes, scales = mxfp4.convert_to_mxfp4(x, axis=axis, is_2d_block=blocks_2d)
        return codes, scales, mxfp4.convert_from_mxfp4(codes, scales, x.dtype, axis=axis, is_2d_block=blocks_2d)
    codes, scales = mxfp8.convert_to_mxfp8(x, mxfp_format=fmt[-4:], axis=axis, is_2d_block=blocks_2d)
    back = mxfp8.convert_from_mxfp8(codes, scales, x.dtype, axis=axis, is_2d_block=blocks_2d)
    return codes.view(torch.uint8), scales, back


def _quantize_and_multiply(state):
    x, w = state["x"], state["w"]
    if state["case"]["recipe"] == "mxfp4":
        (a, a_s), (b, b_s) = mxfp4.convert_to_mxfp4(x), mxfp4.convert_to_mxfp4(w)
        return mxfp4.blockwise_mxfp4_gemm(a, a_s, b, b_s, trans_b=True, output_dtype=torch.bfloat16)
    (a, a_s), (b, b_s) = mxfp8.convert_to_mxfp8(x), mxfp8.convert_to_mxfp8(w)
    return mxfp8.blockwise_mxfp8_gemm(a, a_s, b, b_s, trans_b=True, output_dtype=torch.bfloat16)


def run(state):
    op = state["case"]["op"]
    if op == "linear":
        return _step(state, _call_linear)
    if op == "moe":
        return _step(state, _call_moe)
    return _quantize_round_trip(state) if op == "quantize" else _quantize_and_multiply(state)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how near two correct ones are
# ---------------------------------------------------------------------------------------------
_CODE_BITS = {"nvfp4": 4, "mxfp4": 4, "mxfp8_e4m3": 8, "mxfp8_e5m2": 8}


def work(case):
    op = case["op"]
    if op == "quantize":
        n, size = case["rows"] * case["cols"], 4 if case["dtype"] == "float32" else 2
        block = 16 if case["format"] == "nvfp4" else 32
        scales = n // (block * block if case["blocks_2d"] else block) * (4 if case["format"] == "nvfp4" else 1)
        return {"bytes": 2 * n * size + n * _CODE_BITS[case["format"]] // 8 + scales, "flops": 2 * n}
    k, n = case["k"], case["n"]
    if op == "gemm":
        m = case["m"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if op == "moe":
        m, weights, passes = case["tokens"] * case["top_k"], case["experts"] * k * n, 3
    else:
        m, weights, passes = case["m"], k * n, 3 if case["backward"] else 1
    # forward: x, w in, y out; backward: dy in, dx, dw out
    count = m * k + weights + m * n
    return {"bytes": 2 * count * (2 if passes == 3 else 1), "flops": passes * 2 * m * n * k}


def tolerance(case):
    # codes, scales and the values they stand for are the same in every correct implementation
    if case["op"] == "quantize":
        return "exact"
    # Exact codes, fp32 sums in any order, one rounding to bf16: what differs are the roundings that fall the
    # other way.  With the reduction axis permuted: rel 2.5e-5, max 2^-7.
    return {"rel": 1e-4, "max": 3e-2}


def _block_amax(t, size, blocks_2d):
    """max |t| over blocks of ``size`` along the last axis (or size x size tiles), spread over the block."""
    rows, cols = t.shape[-2:]
    a = torch.nn.functional.pad(t.abs(), (0, -cols % size, 0, -rows % size if blocks_2d else 0))
    a = a.unflatten(-1, (-1, size)).amax(-1)
    if blocks_2d:
        a = a.unflatten(-2, (-1, size)).amax(-2).repeat_interleave(size, -2)[..., :rows, :]
    return a.repeat_interleave(size, -1)[..., :cols].float()


def _random_words(seed, offset, rows, cols):
    """The word of every element of a [rows, cols] view: Philox-4x32-10 over a 64 x 64 tile that repeats;
    counter ``offset`` + pair index, output 0 for even and 1 for odd elements."""
    tile_rows, pairs = min(64, rows), min(64, cols) // 2
    low, m32 = 0xFFFF, 0xFFFFFFFF

    def multiply(a, b):
        p1, p0 = a * (b >> 16), a * (b & low)
        return (p1 + (p0 >> 16)) >> 16, (((p1 & low) << 16) + p0) & m32

    c0 = (torch.arange(tile_rows * pairs, device=DEVICE) + offset) & m32
    c1 = c2 = c3 = torch.zeros_like(c0)
    k0, k1 = seed & m32, seed >> 32
    for _ in range(10):
        (hi_b, lo_b), (hi_a, lo_a) = multiply(0xCD9E8D57, c2), multiply(0xD2511F53, c0)
        c0, c1, c2, c3 = hi_b ^ c1 ^ k0, lo_b, hi_a ^ c3 ^ k1, lo_a
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    tile = torch.stack([c0, c1], -1).reshape(tile_rows, 2 * pairs)
    return tile.repeat(-(-rows // tile_rows), -(-cols // (2 * pairs)))[:rows, :cols]


def _to_e2m1(v, words):
    """|v| on the E2M1 grid (spacing 0.5 below 2, 1 below 4, 2 up to 6): to nearest even, or stochastically."""
    a = v.abs().clamp(max=6.0)
    step = torch.where(a < 2.0, 0.5, torch.where(a < 4.0, 1.0, 2.0)).double()
    t = a / step
    if words is None:
        t = torch.round(t)
    else:
        below_one = torch.floor(t) + (words <= torch.floor((t - torch.floor(t)) * 2.0 ** 32))
        t = torch.where(a < 1.0, below_one, torch.floor(t + (words & 0x3FFFFF) / 2.0 ** 22))
    return torch.copysign(t * step, v)


def _outer_scale(t):
    # divided in 64 bits: a CUDA tensor divided by a Python number is multiplied by its rounded reciprocal
    return (t.abs().amax().double() / (448.0 * 6.0)).float().clamp(min=1e-30)


def _round_trip(t, fmt, blocks_2d=False, words=None):
    """The values that t's codes and scales stand for, blocks along the last axis."""
    if fmt == "mxfp4_two_level":
        bits = (6.0 / _block_amax(t, 128, blocks_2d).clamp(min=1e-12)).view(torch.int32) & 0x7F8000
        factor = (bits + (127 << 23)).view(torch.float32)
        return _round_trip((t.float() * factor).to(t.dtype), "mxfp4", blocks_2d, words) / factor.double()
    amax = _block_amax(t, 16 if fmt == "nvfp4" else 32, blocks_2d)
    if fmt == "nvfp4":
        outer = _outer_scale(t)
        inner = ((amax / outer).double() / 6.0).float().clamp(2.0 ** -6, 448.0).to(torch.float8_e4m3fn).float()
        scale = (inner * outer).double()
        # codes are defined on the quotient in fp32, where it can fall on a tie
        return _to_e2m1((t.double() / scale).float().double(), words) * scale
    mantissa_bits, target = {"mxfp4": (1, 2), "mxfp8_e4m3": (3, 8), "mxfp8_e5m2": (2, 15)}[fmt]
    mantissa, exponent = torch.frexp(amax)
    exponent = exponent - 1 + (2 * mantissa >= 2 - 2.0 ** -(mantissa_bits + 1)) - target
    scale = torch.exp2(exponent.clamp(min=-126).double())
    v = t.double() / scale
    if fmt == "mxfp4":
        return _to_e2m1(v, words) * scale
    dtype = getattr(torch, {"mxfp8_e4m3": "float8_e4m3fn", "mxfp8_e5m2": "float8_e5m2"}[fmt])
    top = torch.finfo(dtype).max
    return v.float().clamp(-top, top).to(dtype).double() * scale


def _rotated(t, matrix):
    """The block Hadamard transform of the token axis, in t's type."""
    if matrix is None:
        return t
    n = matrix.shape[0]
    return (matrix @ t.double().unflatten(0, (-1, n)) / n ** 0.5).flatten(0, 1).to(t.dtype)


def exact(case, seed):
    """The outputs in 64-bit arithmetic: operands rounded to their formats, then multiplied in float64.
    Codes and block scales are bytes and grid values, they have no such value."""
    inp = _inputs(case, seed)
    x = inp["x"]
    if case["op"] == "quantize":
        last = (lambda t: t) if case["axis"] == -1 else (lambda t: t.transpose(-1, -2))
        back = last(_round_trip(last(x), case["format"], case["blocks_2d"]))
        if case["format"] != "nvfp4":
            return None, None, back
        return None, None, back, (x.double().abs().amax() / (448.0 * 6.0)).reshape(1)
    w, fmt = inp["w"], {"mxfp8": "mxfp8_e4m3"}.get(case["recipe"], case["recipe"])
    if case["op"] == "gemm":
        return _round_trip(x, fmt) @ _round_trip(w, fmt).t()
    w_2d = case.get("weight_2d", True)
    x_k, w_k = _round_trip(x, fmt), _round_trip(w, fmt, w_2d)
    if case["op"] == "linear" and not case["backward"]:
        return x_k @ w_k.t()
    w_n = w_k if w_2d else _round_trip(w.t(), fmt).t()
    dy = inp["dy"]
    rows, n = dy.shape
    matrix, words = None, (None, None)
    if case["hadamard"]:
        # the drawn matrix is an input of the pass
        nvfp4.HadamardFactory.configure(block_size=case["hadamard"], randomized=True, dtype=torch.float32, seed=seed)
        matrix = nvfp4.HadamardFactory.create_transform(device=DEVICE).matrix().double().to(DEVICE)
    if case["sr"]:
        gen = torch.Generator().manual_seed(seed)
        keys = [torch.randint(0, 2 ** 31 - 1, (2,), generator=gen).tolist() for _ in range(2)]
        words = _random_words(*keys[0], rows, n), _random_words(*keys[1], n, rows)
    fmt_grad = "mxfp8_e5m2" if case["op"] == "moe" and case["recipe"] == "mxfp8" else fmt
    g_n = _round_trip(dy, fmt_grad, words=words[0])
    g_m = _round_trip(_rotated(dy, matrix).t(), fmt_grad, words=words[1])
    x_m = _round_trip(_rotated(x, matrix).t(), fmt)
    if case["op"] == "linear":
        return x_k @ w_k.t(), g_n @ w_n, g_m @ x_m.t()
    y, dx, dw = torch.zeros_like(g_n), torch.zeros_like(x_k), torch.zeros_like(w_k)
    start = 0
    for e, end in enumerate(inp["offs"].tolist()):
        run_ = slice(start, end)
        y[run_], dx[run_], dw[e] = x_k[run_] @ w_k[e].t(), g_n[run_] @ w_n[e], g_m[:, run_] @ x_m[:, run_].t()
        start = end
    return y, dx, dw
