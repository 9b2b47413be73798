"""Performance cases of the trellis linear layer: what a serving program has the library do.

A case is one of four operations, always through the public Python objects over the C ABI:

  decode  a decode step: one captured graph of single-layer plans over a stack of layers
          (1..8 activation rows), weights far larger than the L2 from step to step
  gemv    one layer, 1..8 rows: an immediate call ("call"), a frozen plan ("plan") or the
          tensor-parallel dense plan ("dense": float32 row views, scratch of the library)
  gemm    one layer, more than 8 rows (prefill): an immediate call or a frozen plan
  moe     a routed-expert block on one rank's expert bank, routes read on the device

Weights are seeded uniform random trellis words (every bit pattern is a valid code), scales
and activations have the distributions of `synthetic.py`, routes are softmax top-k of seeded
normal logits.
"""
import torch

from strix_trellis_b200 import native, synthetic
from strix_trellis_b200.runtime import Context, DensePlan, MoePlan

# The four layer shapes of the decode benchmark, (inputs, outputs).
STACK = ((4096, 4096), (5120, 5120), (1152, 4096), (4096, 14336))
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _one(name, op, rows, inputs, outputs, bits, dtype, how, codebook="mul1", bias=False):
    return dict(name=name, op=op, rows=rows, inputs=inputs, outputs=outputs, bits=bits, dtype=dtype, how=how,
                codebook=codebook, bias=bias)


def listed():
    return [
        # The smallest call a program makes: one token through one small layer, nothing kept
        # between calls but the weights.  Host path and launches count here.
        _one("gemv_call_r1_k4_small", "gemv", 1, 1152, 4096, 4, "f32", "call"),
        # Single-user decoding, the main use: one token through a stack of layers.
        dict(name="decode_step_r1_k4", op="decode", rows=1, copies=4, bits="4", dtype="f32", codebook="mul1"),
        # A small batch (or speculative tokens) through a stack quantised at mixed rates.
        dict(name="decode_step_r4_mixed", op="decode", rows=4, copies=4, bits="2,3,4,5,6", dtype="bf16",
             codebook="mul1"),
        # The vocabulary projection of one token: the widest layer of a model.
        _one("lm_head_r1_k5", "gemv", 1, 4096, 129280, 5, "f32", "dense"),
        # An attention output projection with a long input, eight rows.
        _one("o_proj_r8_k5_long", "gemv", 8, 16384, 4096, 5, "f32", "dense"),
        # Batched decoding just past the decode kernel's row limit.
        _one("gemm_r16_k4", "gemm", 16, 5120, 5120, 4, "f16", "plan"),
        # A short prompt, or a large decode batch, of an odd length.
        _one("gemm_r101_k4", "gemm", 101, 4096, 12288, 4, "f16", "plan", bias=True),
        # One prefill chunk.
        _one("gemm_r512_k5", "gemm", 512, 4096, 12288, 5, "bf16", "call"),
        # A prompt of ragged length, float32 tensors, another rate and shape.
        _one("gemm_r1777_k6", "gemm", 1777, 5120, 5120, 6, "f32", "call"),
        # The largest prefill of the benchmark.
        _one("gemm_r8192_k4", "gemm", 8192, 4096, 12288, 4, "f16", "call"),
        # One rank's bank of a 256-expert layer: a decode batch and a prefill chunk.
        dict(name="moe_t8_k2", op="moe", tokens=8, experts=32, top_k=8, model=4096, inter=2048, bits=2,
             codebook="mul1"),
        dict(name="moe_t64_k2", op="moe", tokens=64, experts=32, top_k=8, model=4096, inter=2048, bits=2,
             codebook="mul1"),
    ]


def _log(rng, low, high):
    return low * (high / low) ** rng.random()


def _dim(rng, low, high):
    """A layer dimension (a multiple of 128), spread over the logarithm."""
    return max(low, min(high, 128 * round(_log(rng, low, high) / 128)))


def _format(rng):
    """(bits, codebook): mostly the rates of the benchmark with the default codebook."""
    codebook = rng.choice(("mul1", "mul1", "mul1", "mul1", "mcg", "3inst"))
    bits = rng.choice((2, 3, 4, 4, 5, 6))
    if rng.random() < 0.15:
        bits = rng.choice((1, 7, 8, 1.5, 2.5, 3.5) if codebook == "mul1" else (1, 7, 8))
    return bits, codebook


def draw(rng):
    op = rng.choice(("decode", "gemv", "gemv", "gemm", "gemm", "gemm", "moe"))
    bits, codebook = _format(rng)
    if op == "decode":
        others = [bits] + [rng.choice((2, 3, 4, 5, 6)) for _ in range(rng.randint(0, 3))]
        return dict(op=op, rows=rng.randint(1, 8), copies=rng.randint(2, 5), bits=",".join(str(b) for b in others),
                    dtype=rng.choice(tuple(DTYPES)), codebook=codebook if bits in (2, 3, 4, 5, 6) else "mul1")
    if op == "moe":
        experts = rng.choice((8, 16, 32, 48))
        model, inter = _dim(rng, 1024, 5120), _dim(rng, 512, 2048)
        return dict(op=op, tokens=round(_log(rng, 1, 64)), experts=experts, top_k=rng.choice((2, 4, 6, 8)),
                    model=model, inter=inter, bits=rng.choice((2, 2, 3, 4)), codebook="mul1")
    how = rng.choice(("call", "plan"))
    dtype = rng.choice(tuple(DTYPES))
    bias = rng.random() < 0.25
    if op == "gemv":
        rows, inputs, outputs = rng.randint(1, 8), _dim(rng, 512, 16384), _dim(rng, 512, 32768)
        if rng.random() < 0.3:
            how, dtype = "dense", "f32"
        if inputs * outputs > 4096 * 65536:
            outputs = 8192
    else:
        rows, inputs, outputs = round(_log(rng, 9, 8192)), _dim(rng, 1024, 8192), _dim(rng, 1024, 14336)
        most = 8192 * 4096 * 12288
        if rows * inputs * outputs > most:
            rows = max(9, most // (inputs * outputs))
    case = _one("", op, rows, inputs, outputs, bits, dtype, how, codebook, bias)
    del case["name"]
    return case


_contexts = {}


def _context():
    device = torch.cuda.current_device()
    if device not in _contexts:
        _contexts[device] = Context(device)
    return _contexts[device]


class _State:
    """What a program keeps: weights, plans, buffers; given back when the state goes away."""

    def __init__(self):
        self.weights, self.plans, self.graph = [], [], None

    def __del__(self):
        self.graph = None
        for plan in self.plans:
            plan.close()
        for w in self.weights:
            w.close()


def _rows(generator, rows, width, dtype="f32"):
    """N(0,1) activation rows as binary16 values, widened or rounded to the tensor's type."""
    x = torch.randn((rows, width), generator=generator, device="cuda", dtype=torch.float32)
    return x.to(torch.float16).to(DTYPES[dtype])


def _rates(case):
    return [float(b) if "." in b else int(b) for b in case["bits"].split(",")]


def _stack(case):
    """(inputs, outputs, bits) of every layer of a decode stack."""
    rates = _rates(case)
    shapes = STACK * case["copies"]
    return [(i, n, rates[k % len(rates)]) for k, (i, n) in enumerate(shapes)]


def prepare(case, seed):
    ctx, s = _context(), _State()
    s.op, s.how = case["op"], case.get("how")
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def layer(index, inputs, outputs, bits, bias=False):
        w = ctx.prepare(synthetic.make_layer(inputs, outputs, bits, seed=1000 * seed + index, codebook=case["codebook"],
                                             bias=bias))
        s.weights.append(w)
        return w

    if s.op == "decode":
        s.x = {i: _rows(gen, case["rows"], i, case["dtype"]) for i, _ in STACK}
        s.y = []
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for k, (i, n, bits) in enumerate(_stack(case)):
                w = layer(k, i, n, bits)
                y = torch.empty((case["rows"], n), dtype=DTYPES[case["dtype"]], device="cuda")
                s.plans.append(w.plan(s.x[i], y, native.OP_GEMV))
                s.y.append(y)
            for plan in s.plans:
                plan.submit()
            stream.synchronize()
            s.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s.graph, stream=stream):
                for plan in s.plans:
                    plan.submit()
        torch.cuda.current_stream().wait_stream(stream)
    elif s.op == "moe":
        model, inter, bits = case["model"], case["inter"], case["bits"]
        bank = []
        for e in range(case["experts"]):
            bank.append((layer(3 * e, model, inter, bits), layer(3 * e + 1, model, inter, bits),
                         layer(3 * e + 2, inter, model, bits)))
        ids, scores = synthetic.make_routes(case["tokens"], case["experts"], case["top_k"], seed=seed)
        s.x = _rows(gen, case["tokens"], model)
        s.y = torch.empty_like(s.x)
        s.plans.append(MoePlan(ctx, bank, s.x, s.y, torch.from_numpy(ids.view("int32")).cuda(),
                               torch.from_numpy(scores).cuda(), device_routed=True))
    else:
        w = layer(0, case["inputs"], case["outputs"], case["bits"], case["bias"])
        s.x = _rows(gen, case["rows"], case["inputs"], case["dtype"])
        if s.how != "call":
            s.y = torch.empty((case["rows"], case["outputs"]), dtype=s.x.dtype, device="cuda")
            operation = native.OP_GEMV if s.op == "gemv" else native.OP_GEMM
            s.plans.append(DensePlan(w, s.x, s.y) if s.how == "dense" else w.plan(s.x, s.y, operation))
    return s


def run(state):
    if state.op == "decode":
        state.graph.replay()
        return state.y
    if state.how == "call":
        w, x = state.weights[0], state.x
        y = torch.empty((x.shape[0], w.outputs), dtype=x.dtype, device=x.device)
        return w.gemv(x, y) if state.op == "gemv" else w.gemm(x, y)
    state.plans[0].submit()
    return state.y


def _layer_work(rows, inputs, outputs, bits, element):
    moved = inputs * outputs * bits / 8 + 2 * (inputs + outputs) + rows * (inputs + outputs) * element
    return moved, 2 * rows * inputs * outputs


def work(case):
    if case["op"] == "decode":
        element = 4 if case["dtype"] == "f32" else 2
        each = [_layer_work(case["rows"], i, n, b, element) for i, n, b in _stack(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if case["op"] == "moe":
        tokens, model, inter, routes = case["tokens"], case["model"], case["inter"], case["tokens"] * case["top_k"]
        # experts that at least one token is expected to choose
        live = case["experts"] * (1 - (1 - case["top_k"] / case["experts"]) ** tokens)
        moved = live * 3 * (model * inter * case["bits"] / 8 + 2 * (model + inter)) + 8 * tokens * model + 8 * routes
        return {"bytes": moved, "flops": 6 * routes * model * inter}
    element = 4 if case["dtype"] == "f32" else 2
    moved, flops = _layer_work(case["rows"], case["inputs"], case["outputs"], case["bits"], element)
    return {"bytes": moved + (4 * case["outputs"] if case["bias"] else 0), "flops": flops}


def tolerance(case):
    if case["op"] == "moe":
        # the hidden rows are rounded to binary16 between two projections: sums that differ in their
        # last bits flip some of those roundings
        return {"rel": 2.5e-4, "max": 1e-2}
    # binary16 products summed in binary32, the result rounded to the tensor's type
    return {"f32": {"rel": 1e-5, "max": 4e-4}, "f16": {"rel": 3e-4, "max": 4e-3},
            "bf16": {"rel": 2e-3, "max": 2e-2}}[case["dtype"]]
