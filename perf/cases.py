"""Performance cases of the NVFP4 projection path.

Each case is one pass through the package's public entry points, the way a training or inference program calls
them, at a size taken from the model shapes this repository runs (GPT-2-small d_model 768 / MLP 3072, GPT-2-medium
1024 / 4096, the d_model 2048 / MLP 8192 shape, vocabulary 32000) or a generic one.  `draw` gives further cases of
the same kinds over the whole range: one token to full batches, ragged sizes, both element types, with and without
a bias.

Kinds:
  step        the C++ driver's whole training step: weights re-quantized, every linear and the LM head forward and
              backward (`HostStep.step`)
  forward     one projection, quantize X + GEMM + epilogue (`projection_forward`), weight already in NVFP4
  backward    one linear backward from dY (`LinearBackwardModule.backward_ms_eden`)
  mlp_f32     an MLP block forward through the f32 module methods with logical scale planes and NVFP4 biases
  weight      schedule-free weight materialisation from the two f32 masters (`OptimizerModule`)
  round_trip  quantize a tensor and decode it again
"""
import importlib
import math

import torch

nv = importlib.import_module("nanogpt-120a_b200")
host_step = importlib.import_module("nanogpt-120a_b200.host_step")
projection_set = importlib.import_module("nanogpt-120a_b200.projection_set")

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "bf16": 2}
NVFP4_BYTES = 0.5625  # half a byte of nibbles and a sixteenth of a scale byte per element


def listed():
    return [
        # one activation tensor with outliers stored as NVFP4 and read back (the quantizer's own configuration)
        dict(name="round_trip 8192x768", kind="round_trip", rows=8192, cols=768, dtype="bf16", rowwise=False),
        # a short prompt through one projection: latency and launches are all there is
        dict(name="forward 16 tokens", kind="forward", tokens=16, in_dim=768, out_dim=2304, dtype="bf16",
             out_dtype="bf16", epilogue="bias"),
        # c_attn forward of one micro-batch, 8 x 1024 tokens
        dict(name="forward c_attn 8192", kind="forward", tokens=8192, in_dim=768, out_dim=2304, dtype="bf16",
             out_dtype="bf16", epilogue="bias"),
        # logits of one evaluation sequence whose length is no multiple of anything, f32 out for the loss
        dict(name="forward lm_head 1000", kind="forward", tokens=1000, in_dim=768, out_dim=32000, dtype="bf16",
             out_dtype="f32", epilogue="none"),
        # a ragged batch's backward in the all-f32 form
        dict(name="backward fc 1000 f32", kind="backward", tokens=1000, in_dim=768, out_dim=3072, dtype="f32",
             grad_dtype="f32", bias=True),
        # c_attn backward of one micro-batch in bf16
        dict(name="backward c_attn 8192", kind="backward", tokens=8192, in_dim=768, out_dim=2304, dtype="bf16",
             grad_dtype="bf16", bias=True),
        # LM-head backward: the widest gradient there is
        dict(name="backward lm_head 8192", kind="backward", tokens=8192, in_dim=768, out_dim=32000, dtype="bf16",
             grad_dtype="bf16", bias=False),
        # the f32 module methods on one 4096-token sequence of the d_model 2048 model
        dict(name="mlp_f32 4096x2048", kind="mlp_f32", tokens=4096, d_model=2048, d_mlp=8192),
        # what an optimizer step does to one MLP weight
        dict(name="weight 3072x768", kind="weight", rows=3072, cols=768, packed=True),
        # one GPT-2-small layer forward and backward at 8192 tokens (the driver's head kept to 128 columns)
        dict(name="step one layer 8192", kind="step", layers=1, d_model=768, d_mlp=3072, vocab=128, tokens=8192),
        # one GPU's share of a GPT-2-medium step split eight ways
        dict(name="step medium 8192", kind="step", layers=24, d_model=1024, d_mlp=4096, vocab=32000, tokens=8192),
        # the full GPT-2-small training step on one GPU
        dict(name="step small 65536", kind="step", layers=12, d_model=768, d_mlp=3072, vocab=32000, tokens=65536),
    ]


def _spread(rng, lo, hi, multiple=1):
    """A size between lo and hi, spread over its logarithm, rounded to `multiple`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["forward", "forward", "backward", "backward", "step", "mlp_f32", "weight", "round_trip"])
    if kind == "forward":
        return dict(kind=kind, tokens=_spread(rng, 1, 32768), in_dim=_spread(rng, 256, 4096, 64),
                    out_dim=_spread(rng, 256, 8192, rng.choice([1, 8, 64, 256])), dtype=rng.choice(["bf16", "bf16", "f32"]),
                    out_dtype=rng.choice(["bf16", "bf16", "f32"]), epilogue=rng.choice(["bias", "bias", "relu2", "none"]))
    if kind == "backward":
        return dict(kind=kind, tokens=_spread(rng, 64, 32768, rng.choice([1, 32, 128, 128])),
                    in_dim=_spread(rng, 256, 4096, 64), out_dim=_spread(rng, 256, 8192, rng.choice([1, 64, 64, 128])),
                    dtype=rng.choice(["bf16", "bf16", "f32"]), grad_dtype=rng.choice(["bf16", "f32"]),
                    bias=rng.random() < 0.75)
    if kind == "mlp_f32":
        d = _spread(rng, 256, 2048, 64)
        return dict(kind=kind, tokens=_spread(rng, 16, 8192), d_model=d, d_mlp=4 * d)
    if kind == "weight":
        return dict(kind=kind, rows=_spread(rng, 256, 32000, rng.choice([1, 64])), cols=_spread(rng, 256, 4096, 64),
                    packed=rng.random() < 0.5)
    if kind == "round_trip":
        return dict(kind=kind, rows=_spread(rng, 16, 65536), cols=_spread(rng, 256, 4096, rng.choice([16, 64])),
                    dtype=rng.choice(["bf16", "bf16", "f32"]), rowwise=rng.random() < 0.5)
    d = _spread(rng, 256, 1024, 64)
    return dict(kind=kind, layers=rng.randint(1, 6), d_model=d, d_mlp=4 * d, vocab=_spread(rng, 256, 32000, 64),
                tokens=_spread(rng, 128, 16384, 128))


# ---- inputs ---------------------------------------------------------------------------------------------------

class _Source:
    """Seeded N(0, std) tensors on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)

    def normal(self, shape, std, dtype):
        return (torch.randn(shape, generator=self.gen, device=self.dev) * std).to(dtype)

    def seed(self):
        return int(torch.randint(0, 1 << 31, (1,), generator=self.gen, device=self.dev).item())


def prepare(case, seed):
    src = _Source(seed)
    quant = nv.Nvfp4QuantModule()
    kind = case["kind"]
    if kind == "step":
        shape = projection_set.ModelShape("case", case["layers"], case["d_model"], case["d_mlp"], case["vocab"])
        inputs = projection_set.ProjectionSet(shape, case["tokens"], src.dev, seed=seed, inputs_only=True)
        step = host_step.HostStep(inputs)
        outputs = {"bucket%d" % i: b.view(-1) for i, b in enumerate(step.buckets)}
        for w in sorted({case["d_model"], case["d_mlp"]}):
            outputs["dx%d" % w] = step.dx(w)
        for w in sorted({3 * case["d_model"], case["d_model"], case["vocab"]}):
            outputs["y%d" % w] = step.y(w)
        for t in outputs.values():  # views of memory the driver owns: they keep it alive
            t.owner = step
        return dict(kind=kind, step=step, outputs=outputs)
    if kind == "forward":
        w = src.normal((case["out_dim"], case["in_dim"]), 0.02, torch.bfloat16)
        return dict(kind=kind, x=src.normal((case["tokens"], case["in_dim"]), 1.0, DTYPES[case["dtype"]]),
                    weight=quant.quantize_four_six(w, rowwise=False, packed=True),
                    bias=None if case["epilogue"] == "none" else src.normal((case["out_dim"],), 0.02, torch.float32),
                    epilogue={"none": nv.EPI_NONE, "bias": nv.EPI_BIAS, "relu2": nv.EPI_RELU2}[case["epilogue"]],
                    out_dtype=DTYPES[case["out_dtype"]])
    if kind == "backward":
        t, i, o = case["tokens"], case["in_dim"], case["out_dim"]
        w = src.normal((o, i), 0.02, torch.bfloat16)
        x = src.normal((t, i), 1.0, torch.bfloat16)
        return dict(kind=kind, module=nv.LinearBackwardModule(), e=src.normal((t, o), 1e-3, DTYPES[case["dtype"]]),
                    weight=quant.quantize_four_six(w, rowwise=False, packed=True),
                    input=quant.quantize_four_six(x, rowwise=True, packed=True, decoded_amax=True),
                    scratch=nv.LinearBackwardScratch(t, i, o, src.dev), side=nv.SideStream(src.dev),
                    grad_dtype=DTYPES[case["grad_dtype"]], dweight=torch.empty((o, i), device=src.dev),
                    bias=case["bias"], sign_seed=src.seed(), scale_seed=src.seed())
    if kind == "mlp_f32":
        t, d, h = case["tokens"], case["d_model"], case["d_mlp"]

        def weight(rows, cols):
            return quant.quantize_four_six(src.normal((rows, cols), 0.02, torch.float32), rowwise=False, packed=False)

        return dict(kind=kind, quant=quant, mlp=nv.MlpModule(), x=src.normal((t, d), 1.0, torch.float32),
                    w_fc=weight(h, d), b_fc=weight(1, h), w_proj=weight(d, h), b_proj=weight(1, d),
                    residual=src.normal((t, d), 1.0, torch.float32))
    if kind == "weight":
        z = src.normal((case["rows"], case["cols"]), 0.02, torch.float32)
        return dict(kind=kind, optimizer=nv.OptimizerModule(), z=z,
                    x=z + src.normal((case["rows"], case["cols"]), 1e-3, torch.float32), packed=case["packed"])
    x = src.normal((case["rows"], case["cols"]), 1.0, torch.float32)
    outlier = torch.rand(x.shape, generator=src.gen, device=src.dev) < 1e-3
    x = torch.where(outlier, x * 50.0, x).to(DTYPES[case["dtype"]])
    return dict(kind=kind, quant=quant, decode=nv.Nvfp4DecodeModule(), x=x, rowwise=case["rowwise"])


# ---- one pass -------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "step":
        state["step"].step()
        return state["outputs"]
    if kind == "forward":
        y, xq = nv.projection_forward(state["x"], state["weight"], bias=state["bias"], epilogue=state["epilogue"],
                                      out_dtype=state["out_dtype"])
        return y, xq.bytes, xq.scales, xq.global_scales
    if kind == "backward":
        return state["module"].backward_ms_eden(
            e=state["e"], weight=state["weight"], input=state["input"], scratch=state["scratch"],
            sign_seed=state["sign_seed"], scale_seed=state["scale_seed"], want_dbias=state["bias"],
            grad_dtype=state["grad_dtype"], dweight=state["dweight"], side=state["side"])
    if kind == "mlp_f32":
        quant, mlp = state["quant"], state["mlp"]
        xq = quant.fp32_to_nvfp4_four_six_rowwise(state["x"], quant.row_amax(state["x"]))
        pre, act = mlp.up_relu2(xq, state["w_fc"], state["b_fc"])
        hq = quant.fp32_to_nvfp4_four_six_rowwise(act, quant.row_amax(act))
        return pre, mlp.down_residual(hq, state["w_proj"], state["b_proj"], state["residual"])
    if kind == "weight":
        t, amax = state["optimizer"].materialize_schedule_free(state["z"], state["x"], 0.9, packed=state["packed"])
        return t.bytes, t.scales, t.global_scales, amax
    t = state["quant"].quantize_four_six(state["x"], rowwise=state["rowwise"], packed=False)
    return t.bytes, t.scales, t.global_scales, state["decode"].decode(t)


# ---- what a pass cannot do without ----------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "step":
        t, d, h = case["tokens"], case["d_model"], case["d_mlp"]
        linears = [(d, 3 * d), (d, d), (d, h), (h, d)] * case["layers"] + [(d, case["vocab"])]
        # X, dX, Y and dY in bf16 per linear, the bf16 master weight and the f32 weight gradient
        return dict(bytes=sum(4.0 * t * (i + o) + 6.0 * i * o for i, o in linears),
                    flops=6.0 * t * sum(i * o for i, o in linears))
    if kind == "forward":
        t, i, o = case["tokens"], case["in_dim"], case["out_dim"]
        bias = 0 if case["epilogue"] == "none" else 4 * o
        return dict(bytes=t * i * (SIZE[case["dtype"]] + NVFP4_BYTES) + 4.0 * t + NVFP4_BYTES * i * o + bias +
                    float(SIZE[case["out_dtype"]]) * t * o, flops=2.0 * t * i * o)
    if kind == "backward":
        t, i, o = case["tokens"], case["in_dim"], case["out_dim"]
        return dict(bytes=float(SIZE[case["dtype"]]) * t * o + NVFP4_BYTES * (i * o + t * i) +
                    float(SIZE[case["grad_dtype"]]) * t * i + 4.0 * i * o + (4.0 * o if case["bias"] else 0.0),
                    flops=4.0 * t * i * o)
    if kind == "mlp_f32":
        t, d, h = case["tokens"], case["d_model"], case["d_mlp"]
        # X in, pre-activation and activation out, residual in and out, the two NVFP4 weights
        return dict(bytes=4.0 * t * d * 3 + 8.0 * t * h + 2 * NVFP4_BYTES * d * h, flops=4.0 * t * d * h)
    n = float(case["rows"]) * case["cols"]
    if kind == "weight":
        return dict(bytes=n * (8 + NVFP4_BYTES), flops=0.0)
    return dict(bytes=n * (SIZE[case["dtype"]] + NVFP4_BYTES + 4), flops=0.0)


def tolerance(case):
    kind = case["kind"]
    if kind in ("weight", "round_trip"):
        return "exact"  # quantized bytes are specified bit for bit
    if kind == "mlp_f32":
        # a different summation order of the first GEMM moves a few of its results across a rounding boundary of
        # the second one's 4-bit input
        return dict(rel=1e-3)
    if kind == "step" or "bf16" in (case.get("out_dtype"), case.get("grad_dtype")):
        return dict(rel=4e-3)  # one bf16 rounding (2^-8)
    return dict(rel=1e-5)  # f32 sums; the quantized operands are specified bit for bit
