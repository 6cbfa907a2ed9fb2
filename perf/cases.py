"""What this framework is timed on: the Metis NVFP4 linear layer as training and rollout call it, and the quantizers
and the GEMM that it is made of, each through its public entry point.

Sizes are those of the repository's own benchmark and of its model configurations (the 16384 x 4096 x 4096 rank-128
layer, the 2048^3 fp32 layer, the projections of the 1.5B and 7B Qwen2-style decoders, the RMSNorm -> NVFP4 sweep
over hidden 1536 / 3584 / 4096, the GEMM sweep) and, drawn, whatever lies between their ends.

Launch-bound work is issued the way this framework's users issue it: a training step and a decode forward are one
captured graph each (fp4_post_b200.graphs.GraphedStep over static inputs), prefill, the fp32 layer and the direct
quantizer calls are issued from Python.  A captured forward takes its tokens as one sequence of at least two: a
sequence of one token updates the rolling decode mean on the host, which a graph freezes."""
import math

import torch

from fp4_post_b200 import cabi, ops
from fp4_post_b200.decoder import QWEN2_1P5B, QWEN2_7B, Block
from fp4_post_b200.graphs import GraphedStep
from fp4_post_b200.grpo.grpo import MetisArgs, replace_linear_with_metis
from fp4_post_b200.Metis.Metis.bitlinear import BitLinear
from fp4_post_b200.Metis.Metis.quant import Cast2NVFp4e2m1Block

DEV = torch.device("cuda", 0)
CONFIGS = {"1.5b": QWEN2_1P5B, "7b": QWEN2_7B}


# ---- the cases ----------------------------------------------------------------------------------------------------

def listed():
    return [
        # The headline: forward + backward of one layer on 16384 tokens, rank 128, GRPO defaults (mean-centred
        # operands, round to nearest forward, stochastic rounding backward, weights quantized every step).
        dict(name="train_16k_4096", kind="train", tokens=16384, k=4096, n=4096, rank=128, dtype="bf16", sr=True, graph=True),
        # gate_proj / up_proj of the 1.5B decoder on 8 x 1024 tokens, rank 64.
        dict(name="train_8k_1536x8960", kind="train", tokens=8192, k=1536, n=8960, rank=64, dtype="bf16", sr=True, graph=True),
        # A micro-batch whose token count no tile divides, o_proj of the 7B decoder.
        dict(name="train_1k_ragged_3584", kind="train", tokens=1120, k=3584, n=3584, rank=128, dtype="bf16", sr=True, graph=True),
        # The fp32 layer of the CPU baseline (2048 tokens x 2048, rank 64, round to nearest throughout), issued from Python.
        dict(name="train_2k_2048_fp32", kind="train", tokens=2048, k=2048, n=2048, rank=64, dtype="fp32", sr=False, graph=False),
        # Prefill of 16 prompts of 256 tokens through up_proj of the 7B decoder: no autograd, packed weights cached.
        dict(name="prefill_4k_3584x18944", kind="forward", tokens=4096, k=3584, n=18944, rank=128, graph=False),
        # Decode of 16 sequences through one layer.
        dict(name="decode_16_14336x4096", kind="forward", tokens=16, k=14336, n=4096, rank=128, graph=True),
        # Decode of 64 sequences through one decoder block of the 7B configuration: seven projections, norms, attention.
        dict(name="decode_block_7b_64", kind="block", tokens=64, config="7b", rank=128),
        # An output gradient quantized for both backward products: centred, stochastic, both orientations.
        dict(name="quant_dual_16k_4096", kind="quant", tokens=16384, hidden=4096, form="dual", dtype="bf16", centred=True, sr=True),
        # The plain row-major quantizer on a long batch.
        dict(name="quant_rows_64k_4096", kind="quant", tokens=65536, hidden=4096, form="rows", dtype="bf16", centred=False, sr=False),
        # Fused RMSNorm -> NVFP4: the long end and the short end of the sweep.
        dict(name="rmsnorm_64k_3584", kind="rmsnorm", tokens=65536, hidden=3584),
        dict(name="rmsnorm_1k_1536", kind="rmsnorm", tokens=1024, hidden=1536),
        # One product of the GEMM sweep with the widest side product.
        dict(name="gemm_4k_14336x4096_r256", kind="gemm", tokens=4096, k=4096, n=14336, rank=256),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


MOST_FLOPS = 6 * 16384 * 4096 * 4096      # of one drawn case


def draw(rng):
    kind = rng.choice(["train", "train", "forward", "forward", "block", "quant", "quant", "rmsnorm", "gemm"])
    if kind == "train":
        sr = rng.random() < 0.75
        dtype = "bf16" if rng.random() < 0.8 else "fp32"
        c = dict(kind=kind, tokens=_log(rng, 256, 16384, 32), k=_log(rng, 1024, 8960, 32), n=_log(rng, 512, 8960, 32),
                 rank=rng.choice([32, 64, 128]), dtype=dtype, sr=sr, graph=dtype == "bf16")
        while 6 * c["tokens"] * c["k"] * c["n"] * (4 if dtype == "fp32" else 1) > MOST_FLOPS:
            c["tokens"] = c["tokens"] // 64 * 32
        return c
    if kind == "forward":
        decode = rng.random() < 0.5
        c = dict(kind=kind, tokens=_log(rng, 2, 512) if decode else _log(rng, 512, 16384), k=_log(rng, 1024, 18944, 32),
                 n=_log(rng, 512, 18944, 16), rank=rng.choice([32, 64, 128]), graph=decode)
        while 2 * c["tokens"] * c["k"] * c["n"] > MOST_FLOPS:
            c["tokens"] //= 2
        return c
    if kind == "block":
        return dict(kind=kind, tokens=_log(rng, 2, 256), config=rng.choice(["1.5b", "7b"]), rank=rng.choice([64, 128]))
    if kind == "quant":
        form = rng.choice(["rows", "transposed", "dual"])
        sr = rng.random() < 0.5
        return dict(kind=kind, tokens=_log(rng, 16, 32768, 1 if form == "rows" else 16), hidden=_log(rng, 1024, 8192, 16), form=form,
                    dtype=rng.choice(["bf16", "bf16", "fp32"]), centred=rng.random() < 0.6, sr=sr)
    if kind == "rmsnorm":
        return dict(kind=kind, tokens=_log(rng, 1, 65536), hidden=_log(rng, 1024, 4096, 16))
    c = dict(kind=kind, tokens=_log(rng, 16, 16384), k=_log(rng, 1024, 14336, 32), n=_log(rng, 1024, 14336, 16), rank=rng.choice([0, 32, 128, 256]))
    while 2 * c["tokens"] * c["k"] * c["n"] > MOST_FLOPS:
        c["tokens"] //= 2
    return c


# ---- inputs (plain torch, from the seed alone) ----------------------------------------------------------------------

def _dtype(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _layer_inputs(case, seed):
    """Activation with 1 % outlier channels, factors U diag(s) V with the spread of a singular value decomposition
    and a residual, output gradient."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    m, k, n, r = case["tokens"], case["k"], case["n"], case["rank"]

    def randn(*shape):
        return torch.randn(*shape, device=DEV, generator=g)

    dt = _dtype(case)
    x = randn(1, m, k)
    x[..., torch.randperm(k, device=DEV, generator=g)[: max(1, k // 100)]] *= 20
    p = dict(x=x.to(dt), u=(randn(n, r) / n ** 0.5).to(dt), v=(randn(r, k) / k ** 0.5).to(dt),
             s=torch.linspace(1.9, 1.1, r, device=DEV).to(dt), w=(randn(n, k) / k ** 0.5).to(dt))
    if case["kind"] == "train":
        p["g"] = (randn(1, m, n) + 0.1 * randn(1, 1, n)).to(dt)
    return p


def _layer(case, p):
    r, dt = case["rank"], _dtype(case)
    args = MetisArgs(forward_svd_rank=r, activation_lowrank_svd=r, backward_lowrank_svd=r, cache_quantized_weight=case["kind"] == "forward")
    args.device = DEV
    if case["kind"] == "train" and not case["sr"]:
        args.q_backward_input = args.q_backward_weight = args.q_backward_outputgrad = "nvfp4e2m1bnosr"
    # a small layer is split (the singular value decomposition of the full one takes seconds) and given its factors,
    # as loading a checkpoint of a split layer does
    layer = BitLinear(max(r, 16), max(r, 16), args=args, bias=False, dtype=dt, compute_dtype=dt)
    with torch.no_grad():
        layer.warmup_linear.weight.copy_(torch.eye(max(r, 16), device=DEV))
        layer.split()
        for mod, w in ((layer.vlinear, p["v"]), (layer.warmup_linear, p["w"]), (layer.ulinear, p["u"])):
            mod.weight = torch.nn.Parameter(w.clone())
            mod.out_features, mod.in_features = w.shape
        layer.s = torch.nn.Parameter(p["s"].clone())
    layer.layer_name = "perf"
    return layer


def _reset_random():
    """The stochastic quantizer's call counters at a fixed value, so that two runs draw the same bits."""
    for lane in (0, 1):
        for c in [t for (d, ln), t in Cast2NVFp4e2m1Block._counters.items() if ln == lane]:
            c.fill_(1)


def _norm_input(case, seed):
    """Student-t activations with a per-channel bias, RMSNorm weight around one."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    m, h = case["tokens"], case["hidden"]
    x = torch.randn(m, h, device=DEV, generator=g)
    chi = sum(torch.randn(m, h, device=DEV, generator=g).square_() for _ in range(3))
    x /= (chi / 3).sqrt_()
    x += 2 * torch.randn(1, h, device=DEV, generator=g)
    return x.to(torch.bfloat16), (1 + 0.1 * torch.randn(h, device=DEV, generator=g)).to(torch.bfloat16)


def _quant_input(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    m, h = case["tokens"], case["hidden"]
    x = torch.randn(m, h, device=DEV, generator=g)
    x[:, torch.randperm(h, device=DEV, generator=g)[: max(1, h // 100)]] *= 20
    x = x.add_(0.2 * torch.randn(1, h, device=DEV, generator=g)).to(_dtype(case))
    return x, x.double().mean(0).float() if case["centred"] else None


def _gemm_input(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    m, k, n, r = case["tokens"], case["k"], case["n"], case["rank"]
    a = torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)
    b = (torch.randn(n, k, device=DEV, generator=g) / k ** 0.5).to(torch.bfloat16)
    t = 30 * torch.randn(m, r, device=DEV, generator=g).to(torch.bfloat16) if r else None
    u = torch.randn(n, r, device=DEV, generator=g).to(torch.bfloat16) if r else None
    return a, b, t, u


# ---- prepare and run ------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        p = _layer_inputs(case, seed)
        layer = _layer(case, p)
        state = dict(case=case, layer=layer, x=p["x"])
        if kind == "train":
            x, grad = p["x"].requires_grad_(True), p["g"]
            leaves = [x, layer.ulinear.weight, layer.s, layer.vlinear.weight, layer.warmup_linear.weight]

            def step():
                for t in leaves:
                    t.grad = None
                y = layer(x)
                y.backward(grad)
                return [y.detach()] + [t.grad for t in leaves]
        else:
            def step():
                with torch.no_grad():
                    return layer(p["x"])
        if case["graph"]:
            state["step"] = GraphedStep(step)
        else:
            with torch.no_grad():
                layer.vlinear._get_quantized_weight(layer.vlinear.weight)          # a serving process has its weights packed
                layer.warmup_linear._get_quantized_weight(layer.warmup_linear.weight)
            state["step"] = step
        _reset_random()
        return state
    if kind == "block":
        cfg = CONFIGS[case["config"]]
        g = torch.Generator(device=DEV).manual_seed(seed)
        r = case["rank"]
        args = MetisArgs(forward_svd_rank=r, activation_lowrank_svd=r, backward_lowrank_svd=r, cache_quantized_weight=True)
        args.device = DEV
        with torch.device("meta"):
            blk = Block(cfg, fuse_norms=True)
        sizes = {name: (mod.out_features, mod.in_features, mod.bias is not None) for name, mod in blk.named_modules() if isinstance(mod, torch.nn.Linear)}
        small = Block(type(cfg)(hidden=r, layers=1, heads=1, kv_heads=1, head_dim=r, ffn=r, vocab=r), fuse_norms=True).to(DEV, torch.bfloat16)
        replace_linear_with_metis(small, dtype=torch.bfloat16, metis_args=args, compute_dtype=torch.bfloat16)
        small.self_attn.cfg = cfg

        def randn(*shape):
            return torch.randn(*shape, device=DEV, generator=g)

        with torch.no_grad():
            for norm in (small.input_layernorm, small.post_attention_layernorm):
                norm.weight = torch.nn.Parameter((1 + 0.1 * randn(cfg.hidden)).to(torch.bfloat16))
            for name, (n, k, has_bias) in sizes.items():
                layer = small.get_submodule(name)
                for mod, w in ((layer.vlinear, randn(r, k) / k ** 0.5), (layer.warmup_linear, randn(n, k) / k ** 0.5),
                               (layer.ulinear, randn(n, r) / n ** 0.5)):
                    mod.weight = torch.nn.Parameter(w.to(torch.bfloat16))
                    mod.out_features, mod.in_features = n if mod is not layer.vlinear else r, k if mod is not layer.ulinear else r
                layer.s = torch.nn.Parameter(torch.linspace(1.9, 1.1, r, device=DEV).to(torch.bfloat16))
                if has_bias:
                    layer.warmup_linear.bias = torch.nn.Parameter((0.1 * randn(n)).to(torch.bfloat16))
        x = randn(1, case["tokens"], cfg.hidden).to(torch.bfloat16)
        ang = torch.outer(torch.arange(case["tokens"], device=DEV).float(),
                          cfg.rope_theta ** (-torch.arange(0, cfg.head_dim, 2, device=DEV).float() / cfg.head_dim))
        ang = torch.cat((ang, ang), dim=-1)[None, None]
        cos, sin = ang.cos().to(torch.bfloat16), ang.sin().to(torch.bfloat16)

        def step():
            with torch.no_grad():
                return small(x, cos, sin)
        return dict(case=case, keep=(small, x, cos, sin), step=GraphedStep(step))
    if kind == "quant":
        x, mean = _quant_input(case, seed)
        return dict(case=case, x=x, mean=mean, seed=seed)
    if kind == "rmsnorm":
        x, gamma = _norm_input(case, seed)
        return dict(case=case, x=x, gamma=gamma)
    a, b, t, u = _gemm_input(case, seed)
    return dict(case=case, a=ops.nvfp4_quantize(a), b=ops.nvfp4_quantize(b), lowrank=(t, u) if t is not None else None)


def _parts(q):
    return [q.codes, q.scales, q.unit]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("train", "forward", "block"):
        return state["step"]()
    if kind == "quant":
        kw = dict(stochastic=case["sr"], seed=state["seed"], offset=1, mean=state["mean"])
        if case["form"] == "dual":
            q, qt = ops.nvfp4_quantize_dual(state["x"], token_sums=case["centred"], **kw)
            return _parts(q) + _parts(qt) + ([qt.token_sums] if qt.token_sums is not None else [])
        return _parts(ops.nvfp4_quantize(state["x"], transpose=case["form"] == "transposed", **kw))
    if kind == "rmsnorm":
        return _parts(ops.rmsnorm_nvfp4_quantize(state["x"], state["gamma"], 1e-6))
    return ops.nvfp4_gemm(state["a"], state["b"], lowrank=state["lowrank"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

PACKED = 0.5 + 1 / 16


def _projection(m, k, n, r, e=2):
    """Bytes and flops of one no-grad forward on packed weights."""
    return m * (k + n) * e + (n * k + r * k) * PACKED + n * r * e, 2 * m * n * k + 2 * m * r * (k + n)


def work(case):
    kind = case["kind"]
    if kind in ("quant", "rmsnorm"):
        m, h = case["tokens"], case["hidden"]
        e = 4 if case.get("dtype") == "fp32" else 2
        return {"bytes": m * h * (e + PACKED * (2 if case.get("form") == "dual" else 1)), "flops": 2 * m * h}
    if kind == "block":
        c, m, r = CONFIGS[case["config"]], case["tokens"], case["rank"]
        shapes = [(c.hidden, c.heads * c.head_dim)] + 2 * [(c.hidden, c.kv_heads * c.head_dim)] + [(c.heads * c.head_dim, c.hidden)] \
            + 2 * [(c.hidden, c.ffn)] + [(c.ffn, c.hidden)]
        weights = sum((n * k + r * k) * PACKED + n * r * 2 for k, n in shapes)
        return {"bytes": weights + 2 * m * c.hidden * 2, "flops": sum(_projection(m, k, n, r)[1] for k, n in shapes)}
    m, k, n, r = case["tokens"], case["k"], case["n"], case["rank"]
    if kind == "gemm":
        return {"bytes": (m * k + n * k) * PACKED + m * n * 2 + (m + n) * r * 2, "flops": 2 * m * n * (k + r)}
    if kind == "forward":
        b, f = _projection(m, k, n, r)
        return {"bytes": b, "flops": f}
    e = 4 if case["dtype"] == "fp32" else 2
    weights = n * k + r * k + n * r + r
    return {"bytes": (2 * m * (k + n) + 2 * weights) * e, "flops": 6 * m * n * k + 6 * m * r * (k + n)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quant", "rmsnorm"):
        return "exact" if kind == "rmsnorm" or not case["centred"] else {"rel": 1e-5, "max": 1e-3, "differ": 0.0}
    if kind == "gemm":
        return {"rel": 1e-2, "max": 2e-2}
    # fp32: the sums agree to 1e-6, a code that flips at a tie moves an input gradient by 1e-4 of its norm
    return {"rel": 5e-4 if case.get("dtype") == "fp32" else 1e-2, "max": 0.5}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
# Which FP4 code and which E4M3 scale an element gets is part of the algorithm and is decided in fp32, as the
# reference decides it; everything that is summed or multiplied is float64.

def _codes(x32):
    """(values in units of their block's scale, scales / unit in E4M3, unit) of fp32 x along its last dimension."""
    blocks = x32.reshape(x32.shape[0], -1, 16)
    six, two, top = (torch.tensor(v, device=x32.device) for v in (6.0, 2.0, 448.0))
    s = blocks.abs().amax(dim=2, keepdim=True) / six + 1e-9
    unit = s.amax() / top
    q = blocks.abs() / (s / two)
    q = torch.round(q - (torch.relu(q - 4) / 2 + torch.relu(q - 8) / 4))
    q = (q + (torch.relu(q - 4) + torch.relu(q - 6) * 2)) * blocks.sign() / two
    return q, (s / unit).to(torch.float8_e4m3fn).double(), unit


def _qdq(x32):
    q, d, unit = _codes(x32)
    return (q.double() * d * unit.double()).reshape(x32.shape)


def _centred(x, both=True):
    """x (float64 view of the data) as mean + quantized remainder, along the rows and along the columns."""
    mean = x.mean(0)
    rest = x.float() - mean.float()
    return mean, _qdq(rest), _qdq(rest.T.contiguous()).T if both else None


def _exact_layer(case, seed):
    p = _layer_inputs(case, seed)
    x, u, v, s, w = p["x"][0].double(), p["u"].double(), p["v"].double(), p["s"].double(), p["w"].double()
    train = case["kind"] == "train"
    mu, xr, xt = _centred(x, train)
    del x
    xr += mu
    vr, wr = _qdq(v.float()), _qdq(w.float())
    yv = xr @ vr.T
    y = (yv * s) @ u.T + xr @ wr.T
    del xr, wr
    if not train:
        return y[None]
    g = p["g"][0].double()
    dts = g @ u
    du, ds = g.T @ (yv * s), (dts * yv).sum(0)
    if case["sr"]:
        return [y[None], None, du, ds, None, None]
    dyv = dts * s
    xt += mu
    dx = 0
    grads = []
    for d, q in ((dyv, v), (g, w)):
        md, dr, dt = _centred(d)
        qn = _qdq(q.float().T.contiguous()).T
        dx = dx + (dr + md) @ qn
        grads.append((dt + md).T @ xt)
    bf16 = case["dtype"] == "bf16"       # d_yv is rounded to bf16 before it is quantized there: another input
    return [y[None], None if bf16 else dx[None], du, ds, None if bf16 else grads[0], grads[1]]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        return _exact_layer(case, seed)
    if kind == "block":
        return None
    if kind == "gemm":
        a, b, t, u = _gemm_input(case, seed)
        (qa, da, ua), (qb, db, ub) = _codes(a.float()), _codes(b.float())
        a, b = (qa.double() * da).reshape(a.shape), (qb.double() * db).reshape(b.shape)
        acc = a @ b.T
        if t is not None:
            acc += t.double() @ u.double().T
        return acc * (ua.double() * ub.double())
    if kind == "rmsnorm":
        return None                       # bytes, and a unit that follows the fp32 roundings of the norm
    x, mean = _quant_input(case, seed)
    x = x.float() if mean is None else x.float() - mean

    def unit(t):
        return (t.reshape(-1, 16).abs().amax().double() / 6 + 1e-9) / 448

    def sums():                           # of the quantized values of each column
        return _qdq(x.T.contiguous()).sum(1) if not case["sr"] else None
    if case["form"] == "dual":
        out = [None, None, unit(x).reshape(1), None, None, unit(x.T.contiguous()).reshape(1)]
        return out + ([sums()] if case["centred"] and case["tokens"] % 64 == 0 else [])
    return [None, None, unit(x.T.contiguous() if case["form"] == "transposed" else x).reshape(1)]
