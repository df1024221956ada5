"""The work that a program using this package has it do, as cases that can be timed and checked.

Operators of the device (row softmax, fused RMS norm and gate, matrix products), the Llama model on its fused engine
(prompts and decode steps), the two layer-list models (a prompt and the tokens after it) and the Llama graph that the
lazy host layer schedules and runs.  Model sizes are those of the benchmark configurations.  A case is a dict of plain
values; `kind` says which path it takes:

  softmax, rms_silu   rows, cols                       f32 row operators
  matmul              dtype, b, m, n, k, layout        [b, m, k] x one [k, n] (layout "kn") or [n, k] transposed ("nk")
  llama               batch, prompt, steps             steps = 0: the prompt is timed; else steps on top of a cached prompt
  kabidra, zidevik    batch, prompt, steps             one request: reset, prompt, `steps` further tokens
  graph               prompt, steps                    one sequence in f32, the graph built and scheduled for every token
"""
import math

import numpy as np
import torch

from ug_b200 import kabidra_config, llama_config, zidevik_config

EPS = 1e-5
GRAPH_LAYERS = 6          # of the 22: the host's work and the kernels are the same in every layer


def listed():
    return [
        # one row operator between two other calls of a caller's own step: a launch counts for as much as its bytes
        dict(name="softmax_1024x4096", kind="softmax", rows=1024, cols=4096),
        # the fused norm and gate of a block of activations, far larger than the L2 cache
        dict(name="rms_silu_8192x4096", kind="rms_silu", rows=8192, cols=4096),
        # batched dense contraction of 16-bit activations with one matrix
        dict(name="matmul_bf16_16x512", kind="matmul", dtype="bf16", b=16, m=512, n=4096, k=4096, layout="kn"),
        # a linear layer of the f32 graph on a prompt of odd length
        dict(name="matmul_f32_257", kind="matmul", dtype="f32", b=1, m=257, n=5632, k=2048, layout="nk"),
        # a batch of prompts of one length
        dict(name="llama_prompt_8x512", kind="llama", batch=8, prompt=512, steps=0),
        # one user's prompt, of a length that fills no tile
        dict(name="llama_prompt_1x777", kind="llama", batch=1, prompt=777, steps=0),
        # a serving batch deep in its sequences, tokens chosen by the host
        dict(name="llama_decode_64x2048", kind="llama", batch=64, prompt=2048, steps=8),
        # one user's chat
        dict(name="llama_decode_1x300", kind="llama", batch=1, prompt=300, steps=16),
        # requests to the recurrent / latent attention model: a prompt and its answer
        dict(name="kabidra_8x512_32", kind="kabidra", batch=8, prompt=512, steps=32),
        # the same for the model with attention and scan side by side
        dict(name="zidevik_8x512_32", kind="zidevik", batch=8, prompt=512, steps=32),
        # a long document read once
        dict(name="zidevik_prompt_1x2048", kind="zidevik", batch=1, prompt=2048, steps=0),
        # a program that drives the lazy graph itself, token by token
        dict(name="graph_decode_100", kind="graph", prompt=100, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["softmax", "rms_silu", "matmul", "matmul", "llama", "llama", "llama", "kabidra", "zidevik", "graph"])
    if kind in ("softmax", "rms_silu"):
        cols = _log(rng, 32, 8192)
        if rng.random() < 0.6:
            cols = max(32, cols // 8 * 8)
        return dict(kind=kind, rows=_log(rng, 16, min(32768, (1 << 25) // cols)), cols=cols)
    if kind == "matmul":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        odd = rng.random() < (0.3 if dtype == "f32" else 0.1)
        n, k = (_log(rng, 128, 8192) for _ in range(2))
        if not odd:
            n, k = n // 8 * 8, k // 8 * 8
        b = rng.choice([1, 1, 2, 5, 16])
        most = (1.2e11 if dtype != "f32" and not odd else 6e9) / (2.0 * b * n * k)
        return dict(kind=kind, dtype=dtype, b=b, m=_log(rng, 1, max(2.0, min(2048.0, most))), n=n, k=k, layout=rng.choice(["nk", "nk", "kn"]))
    if kind == "llama" and rng.random() < 0.5:
        batch = _log(rng, 1, 128)
        return dict(kind=kind, batch=batch, prompt=_log(rng, 16, min(3000, 131072 // batch)), steps=rng.randint(4, 16))
    if kind == "graph":
        return dict(kind=kind, prompt=_log(rng, 4, 300), steps=rng.randint(3, 6))
    batch = _log(rng, 1, 16)
    return dict(kind=kind, batch=batch, prompt=_log(rng, 16, min(2048, 4096 // batch)), steps=0 if kind == "llama" else rng.randint(4, 32))


# ------------------------------------------------------------------ inputs ---
def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _normal(seed, shape, dtype=torch.float32, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=_gen(seed))


def _tokens(seed, shape, vocab):
    return np.random.default_rng(seed).integers(0, vocab, shape, dtype=np.int32)


def _kabidra_tensor(name, x):
    """Matrices of variance 1 / columns; gains, biases, taps and averages spread enough to count."""
    tail = name.split(".", 1)[-1]
    if tail == "dwa":
        x *= 0.3
        x[-1] += 0.8
    elif tail in ("mix.dq.norm", "mix.dkv.norm"):
        x = 1.0 + 0.2 * x
    elif tail in ("canon1", "canon2"):
        x *= 0.35
    elif tail == "mix.z.b":
        x -= 1.5
    elif x.ndim == 1 and not tail.endswith(".b"):
        x *= 0.2
    elif x.ndim == 2 and name != "embed":
        x *= x.shape[1] ** -0.5
    return x


def _zidevik_tensor(name, x):
    tail = name.split(".", 1)[-1]
    if tail in ("norm1", "norm", "side.norm", "mix.right.D"):
        x = 1.0 + 0.2 * x
    elif tail == "mix.right.conv":
        x *= 0.5
    elif tail in ("mix.right.conv.b", "step"):
        x *= 0.3
    elif tail == "mix.right.dt.b":
        x = 0.5 * x - 1.5
    elif tail == "mix.right.A_log":
        x = 1.5 * x - 2.0
    elif name == "loop.in":
        x *= 0.6 * x.shape[1] ** -0.5
        x[:, :x.shape[0]] += 0.8 * torch.eye(x.shape[0], device=x.device)
    elif x.ndim == 2 and tail != "embed":
        x *= x.shape[1] ** -0.5
    return x


def _config(case):
    if case["kind"] == "kabidra":
        return kabidra_config.Config.like_llama_1b()
    if case["kind"] == "zidevik":
        return zidevik_config.Config.like_llama()
    cfg = llama_config.Config.llama_1b()
    if case["kind"] == "graph":
        cfg.num_hidden_layers = GRAPH_LAYERS
    return cfg


def _weights(case, seed):
    """(name, tensor) of a model with random weights, one at a time."""
    kind, cfg = case["kind"], _config(case)
    if kind in ("llama", "graph"):
        dtype = torch.bfloat16 if kind == "llama" else torch.float32
        for i, name in enumerate(llama_config.weight_names(cfg)):
            shape = llama_config.weight_shape(cfg, name)
            yield name, (torch.ones(shape, device="cuda") if len(shape) == 1 else _normal(seed * 7919 + i, shape, dtype, 0.02))
        return
    if kind == "kabidra":
        for i, (name, shape) in enumerate(kabidra_config.weight_shapes(cfg).items()):
            yield name, _kabidra_tensor(name, _normal(seed * 7919 + i, shape)).to(torch.bfloat16)
        return
    # A trained router is sure of most of its choices, one of random rows is sure of few.  Each token's embedding holds two of
    # as many directions as there are experts, and every layer's router reads them in an order of its own.
    count = max(l.mlp.count for l in cfg.layers if isinstance(l.mlp, zidevik_config.Experts))
    ways = _normal(seed * 7919 - 1, (count, cfg.width), std=cfg.width ** -0.5)
    for i, (name, shape) in enumerate(zidevik_config.weight_shapes(cfg).items()):
        x = _zidevik_tensor(name, _normal(seed * 7919 + i, shape))
        if name == "embed":
            two = torch.rand(shape[0], count, device="cuda", generator=_gen(seed + 3000)).topk(2, 1).indices
            x += 120.0 * ways[two].sum(1)
        elif name.endswith("mlp.router"):
            x = 0.02 * cfg.width ** -0.5 * x + 0.25 * ways[torch.randperm(count, device="cuda", generator=_gen(seed + 4000 + i))]
        yield name, x.to(torch.bfloat16)


def _model_tokens(case, seed):
    cfg = _config(case)
    vocab = cfg.vocab if hasattr(cfg, "vocab") else cfg.vocab_size
    return _tokens(seed + 17, (case.get("batch", 1), case["prompt"] + case["steps"]), vocab)


_TORCH = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _matmul_inputs(case, seed):
    b, m, n, k = (case[x] for x in "bmnk")
    std, dtype = (0.5 if case["dtype"] == "f32" else 0.02), _TORCH[case["dtype"]]
    return _normal(seed, (b, m, k), dtype, std), _normal(seed + 1000, (n, k) if case["layout"] == "nk" else (k, n), dtype, std)


def _row_inputs(case, seed):
    shape = (case["rows"], case["cols"])
    if case["kind"] == "softmax":
        return (_normal(seed, shape, std=2.0),)
    w = torch.empty(case["cols"], device="cuda").uniform_(0.5, 1.5, generator=_gen(seed + 2000))
    return _normal(seed, shape), w, _normal(seed + 1000, shape)


# ----------------------------------------------------------------- the path ---
_PROCESS = {}


def _device():
    """The one device handle, host device and compilation cache that a program has."""
    if "dev" not in _PROCESS:
        from ug_b200.device import Device
        _PROCESS["dev"] = Device(0)
    return _PROCESS["dev"]


def _graph_device():
    if "graph" not in _PROCESS:
        from ug_b200.lazy import CompilationCache, HostDevice
        _PROCESS["graph"] = HostDevice(_device()), CompilationCache()
    return _PROCESS["graph"]


class _Memory:
    def __init__(self, s, typestr):
        self.slice = s
        self.__cuda_array_interface__ = {"shape": (len(s),), "typestr": typestr, "data": (s.device_ptr, False), "version": 3, "strides": None}


def _new_slice(shape, dtype):
    """A slice of the device and the torch tensor over its memory."""
    from ug_b200.device import DType
    code, typestr = {torch.bfloat16: (DType.BF16, "<i2"), torch.float16: (DType.F16, "<f2"), torch.float32: (DType.F32, "<f4")}[dtype]
    s = _device().allocate_uninit(code, math.prod(shape))
    _device().synchronize()
    view = torch.as_tensor(_Memory(s, typestr), device="cuda")
    return s, (view.view(torch.bfloat16) if dtype == torch.bfloat16 else view).view(shape)


def _to_slice(x):
    s, view = _new_slice(x.shape, x.dtype)
    view.copy_(x)
    torch.cuda.synchronize()
    return s


def prepare(case, seed):
    kind, dev = case["kind"], _device()
    state = dict(case, dev=dev)
    if kind in ("softmax", "rms_silu"):
        state["in"] = [_to_slice(x) for x in _row_inputs(case, seed)]
        state["dst"], state["out"] = _new_slice((case["rows"], case["cols"]), torch.float32)
    elif kind == "matmul":
        b, m, n, k = (case[x] for x in "bmnk")
        lhs, rhs = _matmul_inputs(case, seed)
        state["in"] = [_to_slice(lhs), _to_slice(rhs)]
        state["dst"], state["out"] = _new_slice((b, m, n), lhs.dtype)
        state["layouts"] = ([b, m, k], [m * k, k, 1], 0), ([b, k, n], [0, 1, k] if case["layout"] == "nk" else [0, n, 1], 0)
    elif kind == "graph":
        from ug_b200 import llama_graph
        host, cache = _graph_device()
        state["model"] = llama_graph.Model(_config(case), {k: w.cpu().numpy() for k, w in _weights(case, seed)}, host)
        state["host"], state["cache"] = host, cache
        tokens = _model_tokens(case, seed)
        state["kv"] = state["model"].new_cache()
        _graph_forward(state, tokens[:, :case["prompt"]], 0, state["kv"])
        state["next"] = [np.ascontiguousarray(tokens[:, case["prompt"] + i:case["prompt"] + i + 1]) for i in range(case["steps"])]
    else:
        from ug_b200 import kabidra, llama, zidevik
        tokens = _model_tokens(case, seed)
        t_max = case["prompt"] + max(case["steps"], 1)
        m = {"llama": llama, "kabidra": kabidra, "zidevik": zidevik}[kind].Model(_config(case), dev, case["batch"], t_max)
        for name, w in _weights(case, seed):
            m.load_slice(name, _to_slice(w))
        state["model"] = m
        state["prompt"] = np.ascontiguousarray(tokens[:, :case["prompt"]])
        state["depth"] = case["prompt"]
        state["next"] = [np.ascontiguousarray(tokens[:, case["prompt"] + i]) for i in range(case["steps"])]
        if kind == "llama" and case["steps"]:
            m.prefill(state["prompt"])
    dev.synchronize()
    torch.cuda.synchronize()
    return state


def _graph_forward(state, ids, pos, kv):
    """The loop body of a program on the lazy graph: build, schedule, compile, run, read the logits."""
    from ug_b200.lazy import LB, Schedule
    host = state["host"]
    out = state["model"].fwd(LB.copy(ids, ids.shape, host), LB.copy(np.array([[pos]], np.int32), (1, 1), host), kv)
    Schedule.create_one(out).compile(state["cache"]).run()
    return out.data_vec()


def run(state):
    kind, dev = state["kind"], state["dev"]
    if kind == "softmax":
        dev.custom_softmax(state["in"][0], state["dst"], state["rows"], state["cols"])
        return state["out"]
    if kind == "rms_silu":
        x, w, gate = state["in"]
        dev.rms_norm_silu_gate(x, w, gate, state["dst"], state["rows"], state["cols"], EPS)
        return state["out"]
    if kind == "matmul":
        dev.matmul(state["dst"], *state["in"], tuple(state[x] for x in "bmnk"), *state["layouts"])
        return state["out"]
    if kind == "graph":
        kv, pos, logits = [list(l) for l in state["kv"]], state["prompt"], []
        for i, ids in enumerate(state["next"]):
            logits.append(_graph_forward(state, ids, pos + i, kv))
        return logits
    m = state["model"]
    if kind == "llama" and state["steps"]:
        m.reset(state["depth"])
    else:
        m.reset()
        m.prefill(state["prompt"])
        m.next_tokens()
    for ids in state["next"]:            # the caller chooses what is fed next, and looks at every choice
        m.fwd(ids)
        m.next_tokens()
    return m.logits()


# ------------------------------------------------------------ what it costs ---
def _linear_params(case):
    """(matrix elements that one token is multiplied with, matrix elements that are read when every row has its own)."""
    cfg = _config(case)
    if case["kind"] in ("llama", "graph"):
        h, f, kv = cfg.hidden_size, cfg.intermediate_size, cfg.head_dim() * cfg.num_key_value_heads
        n = cfg.num_hidden_layers * (2 * h * h + 2 * h * kv + 3 * h * f)
        return n, cfg.vocab_size * h
    if case["kind"] == "kabidra":
        n = sum(math.prod(s) for k, s in kabidra_config.weight_shapes(cfg).items() if len(s) == 2 and k not in ("embed", "head") and "canon" not in k)
        return n, cfg.vocab * cfg.width
    shapes = zidevik_config.weight_shapes(cfg)
    times = [cfg.loop.times if cfg.loop and cfg.loop.start <= i < cfg.loop.stop else 1 for i in range(len(cfg.layers))]
    n = cfg.loop.times * 2 * cfg.width ** 2 if cfg.loop else 0
    for name, s in shapes.items():
        if not name.startswith("l") or name.startswith("loop") or len(s) != 2 or name.endswith((".conv", ".A_log")):
            continue
        i = int(name[1:name.index(".")])
        part = cfg.layers[i].mlp.top / cfg.layers[i].mlp.count if ".mlp.e" in name else 1.0
        n += times[i] * part * math.prod(s)
    return n, cfg.vocab * cfg.width


def _all_params(case):
    cfg = _config(case)
    if case["kind"] in ("llama", "graph"):
        return sum(_linear_params(case))
    shapes = (kabidra_config if case["kind"] == "kabidra" else zidevik_config).weight_shapes(cfg)
    return sum(math.prod(s) for k, s in shapes.items() if k not in ("embed", "side.embed"))


def _step_params(case):
    """Matrix elements that a step of `batch` tokens reads: of the experts no more than its tokens can choose."""
    cfg, n = _config(case), _all_params(case)
    if case["kind"] != "zidevik":
        return n
    for l in cfg.layers:
        if isinstance(l.mlp, zidevik_config.Experts):
            share = (1 - l.mlp.top / l.mlp.count) ** case["batch"]
            n -= share * l.mlp.count * 3 * cfg.width * l.mlp.ff
    return n


def _cache_bytes(case):
    """Bytes of keys, values or latents per cached position of a sequence."""
    cfg = _config(case)
    if case["kind"] in ("llama", "graph"):
        return cfg.num_hidden_layers * 2 * cfg.num_key_value_heads * cfg.head_dim() * (2 if case["kind"] == "llama" else 4)
    if case["kind"] == "kabidra":
        return 2 * sum(l.mixer["kv_rank"] for l in cfg.layers if l.type == kabidra_config.LATENT)
    runs = len(cfg.layers) + (cfg.loop.times - 1) * (cfg.loop.stop - cfg.loop.start)
    return 2 * runs * cfg.layers[0].left.kv_heads * (cfg.layers[0].left.dim + cfg.layers[0].left.vdim)


def _pair_flops(case):
    """Operations of attention per pair of a query and a key that it sees."""
    cfg = _config(case)
    if case["kind"] in ("llama", "graph"):
        return 4 * cfg.num_hidden_layers * cfg.hidden_size
    if case["kind"] == "kabidra":
        return sum(2 * l.mixer["heads"] * (l.mixer["dim"] + l.mixer["vdim"]) for l in cfg.layers if l.type == kabidra_config.LATENT)
    runs = len(cfg.layers) + (cfg.loop.times - 1) * (cfg.loop.stop - cfg.loop.start)
    a = cfg.layers[0].left
    return 2 * runs * a.heads * (a.dim + a.vdim)


def work(case):
    kind = case["kind"]
    if kind == "softmax":
        return {"bytes": 8 * case["rows"] * case["cols"], "flops": 5 * case["rows"] * case["cols"]}
    if kind == "rms_silu":
        return {"bytes": 12 * case["rows"] * case["cols"] + 4 * case["cols"], "flops": 10 * case["rows"] * case["cols"]}
    if kind == "matmul":
        b, m, n, k = (case[x] for x in "bmnk")
        return {"bytes": (4 if case["dtype"] == "f32" else 2) * (b * m * k + k * n + b * m * n), "flops": 2 * b * m * n * k}
    batch, t, steps = case.get("batch", 1), case["prompt"], case["steps"]
    layers, head = _linear_params(case)
    vocab = _config(case).vocab if kind in ("kabidra", "zidevik") else _config(case).vocab_size
    size = 4 if kind == "graph" else 2
    nbytes = flops = 0.0
    if not (steps and kind in ("llama", "graph")):          # the prompt is part of the pass
        nbytes += size * _all_params(case) + batch * t * _cache_bytes(case)
        flops += 2 * batch * (t * layers + head) + batch * t * (t + 1) / 2 * _pair_flops(case)
    for i in range(steps):
        nbytes += size * _step_params(case) + batch * (t + i + 1) * _cache_bytes(case)
        flops += 2 * batch * (layers + head) + batch * (t + i + 1) * _pair_flops(case)
    return {"bytes": nbytes + 4 * batch * vocab * (steps if kind == "graph" else 1), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("softmax", "rms_silu"):
        return {"rel": 1e-6, "max": 2e-5}
    if kind == "matmul":
        # 16-bit results: one rounding of a 32-bit sum, which another order of summation moves by one unit here and there
        return {"bf16": {"rel": 2e-3, "max": 1e-2}, "f16": {"rel": 3e-4, "max": 2e-3}, "f32": {"rel": 4e-6, "max": 1e-4}}[case["dtype"]]
    if kind == "graph":
        return {"rel": 2e-5, "max": 2e-4}
    # bf16 activations through 22 layers and more: other splits and chunks of the same products move the logits by 0.006
    # (kabidra), 0.013 (llama) and 0.015 (zidevik), one row by 0.08 of the value; each is about as far from 64 bits
    return {"rel": 0.025 if kind == "kabidra" else 0.03, "max": 0.3}


# -------------------------------------------------- the same in 64 bits, torch ---
def _rms(x, eps=EPS):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale):
    """Causal attention, q [t, heads, d], k / v [t, groups, ...]: one group of heads at a time."""
    t, heads, _ = q.shape
    share = heads // k.shape[1]
    hide = torch.ones(t, t, dtype=torch.bool, device=q.device).triu(1)
    out = []
    for g in range(k.shape[1]):
        s = torch.einsum("ihd,jd->hij", q[:, g * share:(g + 1) * share], k[:, g]).mul_(scale).masked_fill_(hide, -math.inf)
        out.append(torch.einsum("hij,jd->ihd", s.softmax(-1), v[:, g]))
    return torch.cat(out, 1).reshape(t, -1)


def _angles(t, dims, base):
    i = torch.arange(0, dims, 2, dtype=torch.float64, device="cuda")
    a = torch.arange(t, dtype=torch.float64, device="cuda")[:, None] * base ** (-i / dims)
    return a.cos()[:, None], a.sin()[:, None]


def _conv(h, w):
    """sum_j w[:, j] h[t - (taps - 1) + j], rows before the first are zero."""
    taps = w.shape[1]
    full = torch.cat([h.new_zeros(taps - 1, h.shape[1]), h])
    return sum(w[:, j] * full[j:j + h.shape[0]] for j in range(taps))


def _llama_exact(cfg, w, tokens, last):
    """Logits of the last `last` positions of one sequence."""
    d, t = cfg.head_dim(), len(tokens)
    cos, sin = _angles(t, d, cfg.rope_theta)

    def rope(x):
        a, b = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = w["model.embed_tokens.weight"][tokens]
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        h = _rms(x, cfg.rms_norm_eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].T).view(t, -1, d) for n in "qkv")
        x = x + _attend(rope(q), rope(k), v, d ** -0.5) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, cfg.rms_norm_eps) * w[p + "post_attention_layernorm.weight"]
        x = x + (_silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return (_rms(x[-last:], cfg.rms_norm_eps) * w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T


def _kabidra_exact(cfg, w, tokens, last):
    t = len(tokens)
    norm = lambda x, name: _rms(x, cfg.eps) * (1 + w[name])
    x = norm(w["embed"][tokens], "embed.norm")
    depth = [x]
    for i, l in enumerate(cfg.layers):
        p, m = f"l{i}.", l.mixer
        h = norm(x, p + "norm1")
        h = h + _conv(h, w[p + "canon1"])
        if l.type == kabidra_config.MINGRU:
            z = torch.sigmoid(h @ w[p + "mix.z"].T + w[p + "mix.z.b"])
            u = h @ w[p + "mix.x"].T + w[p + "mix.x.b"]
            u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            s, rows = torch.zeros_like(z[0]), []
            for j in range(t):
                s = torch.lerp(s, u[j], z[j])
                rows.append(s)
            y = (torch.stack(rows) * _silu(h @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
        else:
            q = (_rms(h @ w[p + "mix.dq"].T, cfg.eps) * w[p + "mix.dq.norm"]) @ w[p + "mix.uq"].T
            c = _rms(h @ w[p + "mix.dkv"].T, cfg.eps) * w[p + "mix.dkv.norm"]
            q, k, v = (a.view(t, m["heads"], -1) for a in (q, c @ w[p + "mix.uk"].T, c @ w[p + "mix.uv"].T))
            o = _attend(q, k, v, m["scale"]).view(t, m["heads"], -1) * torch.sigmoid(h @ w[p + "mix.g"].T)[:, :, None]
            y = o.reshape(t, -1) @ w[p + "mix.o"].T
        x = x + norm(y, p + "norm1b")
        if l.ff is not None:
            h = norm(x, p + "norm2")
            h = h + _conv(h, w[p + "canon2"])
            x = x + norm((h @ w[p + "mlp.up"].T).clamp(min=0).square() @ w[p + "mlp.down"].T, p + "norm2b")
        depth.append(x)
        x = sum(a * b for a, b in zip(w[p + "dwa"], depth))
    return norm(x[-last:], "final.norm") @ w["head"].T


def _zidevik_exact(cfg, w, tokens, last):
    t, n = len(tokens), len(cfg.layers)
    runs = [(i, None) for i in range(n)]
    if cfg.loop:
        lo, hi = cfg.loop.start, cfg.loop.stop
        runs = [(i, None) for i in range(lo)] + [(i, k if i == lo else None) for k in range(cfg.loop.times) for i in range(lo, hi)] + \
               [(i, None) for i in range(hi, n)]
    gated = lambda h, q: (_silu(h @ w[q + "gate"].T) * (h @ w[q + "up"].T)) @ w[q + "down"].T
    x = x0 = w["embed"][tokens]
    for i, enter in runs:
        l, p = cfg.layers[i], f"l{i}."
        a, s = l.left, l.right
        if enter is not None:
            x = torch.cat([x, x0], 1) @ w["loop.in"].T + w["loop.step"][enter]
        h = _rms(x, cfg.eps) * w[p + "norm1"]
        cos, sin = _angles(t, a.rot_dims, a.rot_base)

        def head(name):
            y = (h @ w[p + name].T).view(t, -1, a.dim).clone()
            u, v = y[..., 0:a.rot_dims:2].clone(), y[..., 1:a.rot_dims:2].clone()
            y[..., 0:a.rot_dims:2], y[..., 1:a.rot_dims:2] = u * cos - v * sin, v * cos + u * sin
            return _rms(y, cfg.eps)

        v = (h @ w[p + "mix.left.v"].T).view(t, -1, a.vdim)
        y = l.left_scale * _attend(head("mix.left.q"), head("mix.left.k"), v, a.scale) @ w[p + "mix.left.o"].T
        u, z = (h @ w[p + "mix.right.in"].T).split(s.inner, 1)
        u = _silu(_conv(u, w[p + "mix.right.conv"]) + w[p + "mix.right.conv.b"])
        low, b, c = (u @ w[p + "mix.right.x"].T).split([s.dt_rank, s.state, s.state], 1)
        dt = torch.nn.functional.softplus(low @ w[p + "mix.right.dt"].T + w[p + "mix.right.dt.b"], threshold=1e9)
        neg, S, rows = -w[p + "mix.right.A_log"].exp(), w["embed"].new_zeros(s.inner, s.state), []
        du = dt * u
        for j in range(t):
            S = torch.addcmul(du[j][:, None] * b[j], S, (dt[j][:, None] * neg).exp_())
            rows.append(S @ c[j])
        o = (torch.stack(rows) + w[p + "mix.right.D"] * u) * _silu(z)
        y = y + l.right_scale * o @ w[p + "mix.right.o"].T
        q = p + "mlp."
        if isinstance(l.mlp, zidevik_config.Experts):
            score, chosen = torch.sigmoid(h @ w[q + "router"].T).topk(l.mlp.top, 1)
            for e in range(l.mlp.count):
                row, col = (chosen == e).nonzero(as_tuple=True)
                y.index_add_(0, row, gated(score[row, col][:, None] * h[row], f"{q}e{e}."))
            if l.mlp.shared:
                y = y + gated(h, q + "shared.")
        elif l.mlp is not None:
            y = y + gated(h, q)
        x = x + y
        if cfg.side_dim:
            g = torch.nn.functional.gelu(x @ w[p + "side.gate"].T, approximate="tanh")
            g = g * w["side.embed"][tokens][:, i * cfg.side_dim:(i + 1) * cfg.side_dim]
            x = x + _rms(g @ w[p + "side.proj"].T, cfg.eps) * w[p + "side.norm"]
    y = (_rms(x[-last:], cfg.eps) * w["final.norm"]) @ w["head"].T
    return cfg.logit_softcap * torch.tanh(y / cfg.logit_softcap) if cfg.logit_softcap else y


def exact(case, seed):
    kind = case["kind"]
    if kind == "softmax":
        return _row_inputs(case, seed)[0].double().softmax(-1)
    if kind == "rms_silu":
        x, w, gate = (a.double() for a in _row_inputs(case, seed))
        return _rms(x) * w * _silu(gate)
    if kind == "matmul":
        a, b = (x.double() for x in _matmul_inputs(case, seed))
        return a @ (b.T if case["layout"] == "nk" else b)
    cfg, tokens = _config(case), torch.from_numpy(_model_tokens(case, seed)).long().cuda()
    w = {k: v.double() for k, v in _weights(case, seed)}
    forward = {"llama": _llama_exact, "graph": _llama_exact, "kabidra": _kabidra_exact, "zidevik": _zidevik_exact}[kind]
    # the recurrences are serial here: what would take long has no 64-bit value
    if kind in ("kabidra", "zidevik") and tokens.numel() > 4608 or kind == "llama" and tokens.numel() > 140000:
        return None
    if kind == "graph":
        return list(forward(cfg, w, tokens[0], case["steps"]).cpu())
    return torch.cat([forward(cfg, w, row, 1) for row in tokens])
