"""What is timed: requests served by the engine's step function, from admission to release.

A case is one model (its architecture, sizes and dtype) and one batch of requests.  ``prepare`` has what a
program has in hand before it serves: the model with its weights on the device, a ``ModelRunner`` and the
requests' token ids on the host.  ``run`` serves the batch once: every request is admitted, its prompt goes
through ``ModelRunner.step`` (whole, or in portions beside the tokens of requests that already decode), then
token after token, and it is released.  The tokens are given, so that every pass does the same work; the
output is the float32 logits of all steps, one after the other.

The sizes are those of the repository's benchmarks: Qwen1.5-MoE-A2.7B's layers with a share of its 24 layers
and the same share of its vocabulary, and the other architectures' mixers at the design benchmark's "medium"
and "small" sizes.  Each of those models is two layers of mixers without feed-forwards, so that an output is two
mixers away from its input; their feed-forwards are the products and routed experts that the Qwen2-MoE cases run.
"""
import math
import random
import zlib

import torch

import cajeta_llm_b200  # noqa: F401
from cajeta_llm_b200.config import parse_config_dict
from cajeta_llm_b200.engine.model import build_model
from cajeta_llm_b200.engine.step import ModelRunner, StepEntry
from cajeta_llm_b200.parts.base import Runtime

F64 = torch.float64
EPS = 1e-6
CTX = 4096            # tokens a request may hold, as the engine's default
PAGE = 16

# layer sizes: Qwen1.5-MoE-A2.7B's, and a model of half its width with grouped key heads
SIZES = {
    "a2.7b": dict(width=2048, heads=16, kv=16, experts=60, top=4, eff=1408, shared=5632, rank=512, state=128),
    "small": dict(width=1024, heads=8, kv=2, experts=16, top=2, eff=512, shared=1024, rank=256, state=64),
}


def _case(name, arch, dtype, requests, prompt, most, steps, chunk=0, want=16, size="a2.7b", layers=2, vocab=1000):
    """``prompt`` to ``most``: the requests' prompt lengths (drawn once from the case's own numbers, log-uniform);
    ``steps``: tokens decoded by each request; ``chunk``: longest portion of a prompt (0 = whole prompts, all in one step);
    ``want``: rows at a portion's end whose logits are wanted (0 = all rows)."""
    c = dict(arch=arch, dtype=dtype, size=size, layers=layers, vocab=vocab, requests=requests, prompt=prompt, most=most, steps=steps,
             chunk=chunk, want=want)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user talking to the model: a step is a chain of small launches
        _case("decode, batch 1", "qwen2_moe", "bfloat16", 1, 512, 512, 48, layers=4, vocab=25322),
        # the headline: a small batch of chats
        _case("decode, batch 8", "qwen2_moe", "bfloat16", 8, 512, 512, 32, layers=4, vocab=25322),
        # a busy server's decode steps
        _case("decode, batch 64", "qwen2_moe", "bfloat16", 64, 128, 128, 24, layers=4, vocab=25322),
        # one long prompt read in one step
        _case("prompt of 2048", "qwen2_moe", "bfloat16", 1, 2048, 2048, 0, layers=4, vocab=25322),
        # a batch of prompts of odd lengths read in one step (scoring, or a queue that has filled up)
        _case("ragged prompts", "qwen2_moe", "bfloat16", 8, 61, 1021, 0, layers=4, vocab=25322),
        # the true 32-bit path, as it checks the 16-bit one: portions of 256 beside decoding requests
        _case("float32, mixed steps", "qwen2_moe", "float32", 8, 64, 1024, 8, chunk=256, vocab=3001),
        # the same path on a whole prompt
        _case("float32, prompt", "qwen2_moe", "float32", 1, 1777, 1777, 0, vocab=3001),
        # state-space and delta-rule mixers reading a long prompt
        _case("Balalorn recurrences, prompt", "Balalorn", "bfloat16", 1, 2048, 2048, 0, want=0),
        # the same recurrences decoding: a state per request read and written each step
        _case("Balalorn recurrences, decode", "Balalorn", "bfloat16", 8, 57, 64, 48),
        # matrix memory, and mixed-heads attention beside gated linear attention, on prompts of odd lengths
        _case("Govuvik mixers, prompts", "Govuvik", "bfloat16", 2, 700, 1100, 0, want=0),
        # differential and latent attention on a long prompt
        _case("Dimuvik attention, prompt", "Dimuvik", "bfloat16", 1, 2048, 2048, 0, want=0),
        # windowed latent attention and linear attention: ragged prompts, then tokens
        _case("Zoporax mixers, serving", "Zoporax", "bfloat16", 4, 300, 900, 24, want=0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    arch = rng.choice(["qwen2_moe", "qwen2_moe", "qwen2_moe", "Balalorn", "Govuvik", "Dimuvik", "Zoporax"])
    size = rng.choice(["a2.7b", "small"])
    f32 = arch == "qwen2_moe" and rng.random() < 0.34
    requests = log_int(1, 8 if f32 or arch != "qwen2_moe" else 64)
    rows = log_int(16, 1500 if f32 else 4000)               # prompt tokens of the whole batch
    lo = max(1, rows // requests // 2)
    most = max(lo, min(2 * rows // requests, 2000))
    steps = rng.choice([0, log_int(1, 24)])
    chunk = rng.choice([0, 0, 256]) if most <= 1024 else 0
    return _case("", arch, "float32" if f32 else "bfloat16", requests, lo, most, min(steps, 8) if f32 else steps, chunk=chunk, size=size,
                 layers=rng.choice([1, 2, 4]) if arch == "qwen2_moe" and not f32 else 2, vocab=rng.choice([1000, 3001, 8192]),
                 want=0 if arch != "qwen2_moe" else 16)


# -- the models ---------------------------------------------------------------------------------
def _config(c):
    s = SIZES[c["size"]]
    h, H = s["width"], s["heads"]
    if c["arch"] == "qwen2_moe":
        return {"architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe", "hidden_size": h, "intermediate_size": s["shared"],
                "num_hidden_layers": c["layers"], "num_attention_heads": H, "num_key_value_heads": s["kv"], "head_dim": 128,
                "vocab_size": c["vocab"], "max_position_embeddings": CTX, "rms_norm_eps": EPS, "rope_theta": 1000000.0,
                "num_experts": s["experts"], "num_experts_per_tok": s["top"], "moe_intermediate_size": s["eff"],
                "shared_expert_intermediate_size": s["shared"], "norm_topk_prob": False, "decoder_sparse_step": 1, "mlp_only_layers": [],
                "tie_word_embeddings": False, "use_sliding_window": False}
    out = {"architecture": c["arch"], "width": h, "vocab": c["vocab"], "norm": {"eps": EPS}}
    latent = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": s["rank"], "q_rank": 3 * s["rank"], "scale": 192 ** -0.5}
    if c["arch"] == "Balalorn":
        out["layers"] = [
            {"type": "mamba2", "mixer": {"heads": 2 * h // 64, "vdim": 64, "state": s["state"], "groups": 8, "norm_groups": 8, "conv": 4}},
            {"type": "delta", "mixer": {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4}}]
    elif c["arch"] == "Govuvik":
        left = {"conv": 4, "dim": 128, "heads": H, "kv_heads": H // 4, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                "rot": {"base": 500000.0, "dims": 64}}
        right = {"heads": H // 4, "dim": 128, "vdim": 256, "tau": 8.0, "decay_rank": 16}
        out.update(canon={"taps": 3}, logit_softcap=50.0)
        out["layers"] = [{"type": "mlstm", "mixer": {"heads": H // 2, "dim": 128, "vdim": 256, "gate_cap": 10.0}},
                         {"type": "parallel", "mixer": {"left": left, "right": right}}]
    elif c["arch"] == "Dimuvik":
        out["layers"] = [
            {"type": "attention", "mixer": {"heads": H, "kv_heads": H // 2, "dim": 64, "vdim": 128, "conv": 4, "diff": 0.5,
                                            "scale": 64 ** -0.5, "q_temp": {"coef": 0.1, "every": 1024}}},
            {"type": "latent_attention", "mixer": dict(latent, rot={"base": 10000.0, "dims": 64})}]
    else:
        out["layers"] = [
            {"type": "lightning", "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": _decays(H)}},
            {"type": "latent_attention", "mixer": dict(latent, mask={"size": 1024}, rot={"base": 50000.0, "dims": 64})}]
    return out


def _decays(heads):
    return [1.0 - 2.0 ** (-2.0 - 6.0 * i / heads) for i in range(heads)]


# standard deviations of the tensors that are no matrices (matrices: 0.02); norms' weights are near one
STD = {"conv": 0.3, "canon1": 0.2, "a2": 0.2, "talk": 0.25, "sink": 1.0, "i.b": 1.0, "a2.b": 1.0, "lq1": 0.1, "lk1": 0.1, "lq2": 0.1,
       "lk2": 0.1}
NEAR_ONE = ("norm", "norm1", "norm2", "norm1b", "temp", "D", "out", "input_layernorm.weight", "post_attention_layernorm.weight",
            "model.norm.weight")


def _tensor(c, seed, name, shape):
    """A weight by its name: trained models' magnitudes, in the dtype a file of this model holds."""
    g = torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) * 1000003 + seed * 7919) & 0x7FFFFFFF)
    shape = tuple(shape)

    def last(k):
        return name == k or name.endswith("." + k)

    if last("A_log"):         # decay rates between 1 and 16
        t = torch.empty(shape, device="cuda").uniform_(1.0, 16.0, generator=g).log_()
    elif last("dt_bias"):     # steps between 0.001 and 0.1 (the inverse of softplus)
        dt = torch.empty(shape, device="cuda").uniform_(math.log(1e-3), math.log(1e-1), generator=g).exp_()
        t = torch.log(torch.expm1(dt))
    elif last("f.b"):         # forget gates that remember
        t = torch.empty(shape, device="cuda").uniform_(3.0, 6.0, generator=g)
    elif last("alpha"):
        t = torch.full(shape, 0.75, device="cuda")
    elif any(last(k) for k in NEAR_ONE):
        t = torch.randn(shape, device="cuda", generator=g).mul_(0.1).add_(1.0)
    elif name == "embed":
        t = torch.randn(shape, device="cuda", generator=g)
    else:
        std = next((v for k, v in STD.items() if last(k)), 0.02)
        t = torch.randn(shape, device="cuda", generator=g, dtype=torch.bfloat16 if c["dtype"] == "bfloat16" and len(shape) > 1 else None)
        t = t.mul_(std)
    return t.to(torch.bfloat16) if c["dtype"] == "bfloat16" else t


class _Weights:
    """Where the model's parts fetch their tensors, as they do from a folder."""

    def __init__(self, c, seed):
        self.c, self.seed = c, seed

    def check(self, schema):
        return None

    def get(self, name, spec):
        return _tensor(self.c, self.seed, name, spec.shape)


# -- the batch of requests ------------------------------------------------------------------------
def _lengths(c):
    r = random.Random(c["requests"] * 1000003 + c["prompt"] * 8191 + c["most"])
    return [int(round(math.exp(r.uniform(math.log(c["prompt"]), math.log(c["most"]))))) for _ in range(c["requests"])]


def _tokens(c, seed):
    """Token ids by request: its prompt, then the tokens it decodes."""
    r = random.Random(seed)
    return [[r.randrange(c["vocab"]) for _ in range(n + c["steps"])] for n in _lengths(c)]


def _plan(c):
    """The steps: lists of (request, first token, one past the last, wanted places among them)."""
    lengths, R = _lengths(c), c["requests"]

    def portion(i, a, b):
        n = b - a
        k = n if c["want"] == 0 else min(n, c["want"])
        return (i, a, b, list(range(n - k, n)))

    steps, at = [], [0] * R
    if not c["chunk"]:
        steps.append([portion(i, 0, n) for i, n in enumerate(lengths)])
        at = list(lengths)
    while any(at[i] < lengths[i] + c["steps"] for i in range(R)):
        now, reading = [], False
        for i in range(R):
            if at[i] < lengths[i]:
                if not reading:
                    b = min(lengths[i], at[i] + c["chunk"])
                    now.append(portion(i, at[i], b))
                    at[i], reading = b, True
            elif at[i] < lengths[i] + c["steps"]:
                now.append((i, at[i], at[i] + 1, [0]))
                at[i] += 1
        steps.append(now)
    return steps


def prepare(case, seed):
    runtime = Runtime(case["dtype"], device="cuda:0")
    model = build_model(parse_config_dict(_config(case)), runtime)
    model.load(_Weights(case, seed))
    rows = max(sum(b - a for _, a, b, _ in step) for step in _plan(case))
    runner = ModelRunner(model, page_tokens=PAGE, max_seqs=case["requests"], max_tokens_per_seq=CTX,
                         num_pages=sum(-(-(n + case["steps"]) // PAGE) + 1 for n in _lengths(case)), max_step_tokens=rows)
    toks = _tokens(case, seed)
    return {"runner": runner, "steps": [[(i, toks[i][a:b], want) for i, a, b, want in step] for step in _plan(case)],
            "requests": case["requests"]}


def run(state):
    runner = state["runner"]
    slots = [runner.admit() for _ in range(state["requests"])]
    out = [runner.step([StepEntry(slots[i], toks, want) for i, toks, want in step]) for step in state["steps"]]
    for s in slots:
        runner.release(s)
    return torch.cat(out)


# -- what a pass cannot do without ----------------------------------------------------------------
def work(case):
    """Weights once a step (a step needs the one before it, and they are larger than any cache; of the experts those
    that the step's rows are expected to pick), cached keys and values or states once a step and request, logits once."""
    s, c = SIZES[case["size"]], case
    h, H, E, R = s["width"], s["heads"], s["experts"], s["rank"]
    el = 4 if c["dtype"] == "float32" else 2
    lengths = _lengths(c)
    total_b = total_f = 0.0
    # per layer: (weights of dense products, bytes cached a token, flops a (query, visible key) pair, window, state floats, flops a row of state)
    if c["arch"] == "qwen2_moe":
        dense = h * (H + 2 * s["kv"]) * 128 + H * 128 * h + E * h + 3 * h * s["shared"]
        kinds = [(dense, 2 * s["kv"] * 128 * el, 4 * H * 128, 0, 0, 0)] * c["layers"]
    elif c["arch"] == "Balalorn":
        mh, N = 2 * h // 64, s["state"]
        kinds = [(h * (2 * mh * 64 + 16 * N + mh) + mh * 64 * h, 0, 0, 0, mh * N * 64, mh * N * 64 * 5),
                 (h * (H * 128 * 4 + 2 * H), 0, 0, 0, H * 128 * 128, H * 128 * 128 * 7)]
    elif c["arch"] == "Govuvik":
        M, G = H // 2, H // 4
        kinds = [(h * M * (2 * 128 + 3 * 256), 0, 0, 0, M * 128 * 257, M * 128 * 256 * 5),
                 (h * 128 * (2 * H + 2 * G) + h * G * (2 * 128 + 3 * 256), 2 * G * 128 * el, H * (4 * 128 + 2 * H), 1024, G * 128 * 256,
                  G * 128 * 256 * 5)]
    else:
        low = (h * (4 * R + 64) + 3 * R * H * 192 + 2 * R * H * 128 + H * 128 * h, (R + 64) * el, 2 * H * 320, 0, 0, 0)
        if c["arch"] == "Dimuvik":
            kinds = [(h * 128 * (2 * H + H), H * 128 * el, 2 * H * (128 + 256), 0, 0, 0), low]
        else:
            kinds = [(5 * h * H * 128, 0, 0, 0, H * 128 * 128, H * 128 * 128 * 5), (low[0] + h * H * 128,) + low[1:3] + (1024, 0, 0)]
    for step in _plan(c):
        rows = sum(b - a for _, a, b, _ in step)
        wanted = sum(len(w) for *_, w in step)
        total_b += wanted * c["vocab"] * 4 + (h * c["vocab"] * el if wanted else 0) + rows * h * el
        total_f += 2.0 * wanted * h * c["vocab"]
        for dense, kv, pair, window, state, per_row in kinds:
            total_b += dense * el + 2 * 4 * state * len(step)
            total_f += 2.0 * dense * rows + float(per_row) * rows
            for _, a, b, _ in step:
                total_b += kv * (min(b, window) if window else b)
                total_f += pair * float(sum(min(p + 1, window) if window else p + 1 for p in range(a, b)))
            if c["arch"] == "qwen2_moe":
                one = 3 * h * s["eff"]
                total_b += one * el * E * (1.0 - (1.0 - s["top"] / E) ** rows)
                total_f += 2.0 * one * s["top"] * rows
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    """About four times the measured distance from the same in 64 bits: 2.9e-6 on the float32 path (sums of some thousand
    products); in bfloat16 what rounding the activations between kernels to 8 bits gives, 1.2e-3 (Zoporax), 1.8e-3 (Dimuvik),
    3.2e-3 (Balalorn), 4.4e-3 (Govuvik), and 0.8e-2 to 1.2e-2 through Qwen2-MoE's layers, where a rounding also moves
    the choice between two nearly tied experts for some rows."""
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5}
    return {"rel": {"qwen2_moe": 3e-2, "Balalorn": 1.3e-2, "Govuvik": 1.8e-2, "Dimuvik": 7e-3, "Zoporax": 5e-3}[case["arch"]]}


# -- the same in 64 bits ----------------------------------------------------------------------------
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(u, w):
    """Causal, per channel: y_t = sum_j w[:, j] u_(t - taps + 1 + j)."""
    taps = w.shape[1]
    p = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=u.dtype, device=u.device), u])
    return sum(w[:, j] * p[j:j + u.shape[0]] for j in range(taps))


def _turn(x, base, dims, pairs):
    """Rotation of the first ``dims`` entries of x [T, heads, D] by the row's position: neighbours, or i with i + dims/2."""
    T, half = x.shape[0], dims // 2
    # the angle is a float32 product, as the architecture defines it
    f = (base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)).float()
    a = (torch.arange(T, device=x.device).float()[:, None] * f).to(F64)
    co, si = torch.cos(a)[:, None], torch.sin(a)[:, None]
    head, rest = x[..., :dims], x[..., dims:]
    u, v = (head[..., 0::2], head[..., 1::2]) if pairs else (head[..., :half], head[..., half:])
    p, q = u * co - v * si, v * co + u * si
    return torch.cat([torch.stack([p, q], -1).flatten(-2) if pairs else torch.cat([p, q], -1), rest], -1)


def _softmax(s, window=0, sink=None):
    """Causal softmax of the last axis of s [..., T, T]."""
    T = s.shape[-1]
    i = torch.arange(T, device=s.device)
    keep = i[None, :] <= i[:, None]
    if window:
        keep &= i[None, :] > i[:, None] - window
    s = s.masked_fill(~keep, float("-inf"))
    if sink is None:
        return torch.softmax(s, -1)
    m = torch.maximum(s.amax(-1, keepdim=True), sink)
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + torch.exp(sink - m))


def _attend(q, k, v, scale, window=0, sink=None):
    """q [T, H, D], k and v [T, G, .]: one head after the other (their scores are T x T in 64 bits)."""
    H, n = q.shape[1], q.shape[1] // k.shape[1]
    return torch.stack([_softmax(q[:, i] @ k[:, i // n].T * scale, window, None if sink is None else sink[i]) @ v[:, i // n]
                        for i in range(H)], 1)


def _mamba2(h, W, s):
    D, N = h.shape[1], s["state"]
    H, I, G = 2 * D // 64, 2 * D, 8
    z, x, dt = (h @ W("in", (2 * I + 2 * G * N + H, D)).T).split([I, I + 2 * G * N, H], 1)
    x = _silu(_conv(x, W("conv", (I + 2 * G * N, 4))) + W("conv.b", (I + 2 * G * N,)))
    x, B, C = x.split([I, G * N, G * N], 1)
    T = h.shape[0]
    x = x.view(T, H, 64)
    B, C = (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = torch.nn.functional.softplus(dt + W("dt_bias", (H,)))
    a = torch.exp(-torch.exp(W("A_log", (H,))) * dt)
    S, ys = torch.zeros((H, N, 64), dtype=F64, device=h.device), []
    for t in range(T):
        S = a[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * x[t][:, None, :]
        ys.append((C[t][:, None, :] @ S)[:, 0])
    y = (torch.stack(ys) + W("D", (H,))[:, None] * x).reshape(T, I) * _silu(z)
    return (_rms(y.view(T, 8, I // 8)).reshape(T, I) * W("norm", (I,))) @ W("o", (D, I)).T


def _delta(h, W, s):
    D, T, H = h.shape[1], h.shape[0], s["heads"]
    KH = H // 2

    def proj(n, heads):
        return _silu(_conv(h @ W(n, (heads * 128, D)).T, W(n + ".conv", (heads * 128, 4)))).view(T, heads, 128)

    q, k, v = proj("q", KH), proj("k", KH), proj("v", H)
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (q * 128 ** -0.5).repeat_interleave(2, 1), k.repeat_interleave(2, 1)
    beta = torch.sigmoid(h @ W("b", (H, D)).T)
    a = torch.exp(-torch.exp(W("A_log", (H,))) * torch.nn.functional.softplus(h @ W("a", (H, D)).T + W("dt_bias", (H,))))
    S, ys = torch.zeros((H, 128, 128), dtype=F64, device=h.device), []
    for t in range(T):
        S = a[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        ys.append((q[t][:, None] @ S)[:, 0])
    o = (_rms(torch.stack(ys)) * W("norm", (128,))).reshape(T, H * 128) * _silu(h @ W("g", (H * 128, D)).T)
    return o @ W("o", (D, H * 128)).T


def _mlstm(h, W, s):
    D, T, H, V = h.shape[1], h.shape[0], s["heads"] // 2, 256
    q, k, v = ((h @ W(n, (H * d, D)).T).view(T, H, d) for n, d in (("q", 128), ("k", 128), ("v", V)))
    q = q * 128 ** -0.5
    gi = 10.0 * torch.tanh((h @ W("i", (H, D)).T + W("i.b", (H,))) / 10.0)
    gf = torch.nn.functional.logsigmoid(10.0 * torch.tanh((h @ W("f", (H, D)).T + W("f.b", (H,))) / 10.0))
    S, n, m = (torch.zeros(x, dtype=F64, device=h.device) for x in ((H, 128, V), (H, 128), (H,)))
    ys = []
    for t in range(T):
        new = torch.maximum(gf[t] + m, gi[t])
        a, b = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new)
        S = a[:, None, None] * S + (b[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        n = a[:, None] * n + b[:, None] * k[t]
        m = new
        ys.append((q[t][:, None] @ S)[:, 0] / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None])
    o = _rms(torch.stack(ys)).reshape(T, H * V) * W("norm", (H * V,))
    return (o * torch.sigmoid(h @ W("g", (H * V, D)).T)) @ W("o", (D, H * V)).T


def _parallel(h, W, s):
    D, T, H, G = h.shape[1], h.shape[0], s["heads"], s["heads"] // 4

    def proj(n, heads):
        return _conv(h @ W("left." + n, (heads * 128, D)).T, W(f"left.{n}.conv", (heads * 128, 4)))

    q = (_rms(proj("q", H)) * W("left.q.norm", (H * 128,))).view(T, H, 128)
    k = (_rms(proj("k", G)) * W("left.k.norm", (G * 128,))).view(T, G, 128)
    v = proj("v", G).view(T, G, 128)
    q, k = _turn(q, 500000.0, 64, False), _turn(k, 500000.0, 64, False)
    sc = torch.einsum("thd,shd->hts", q, k.repeat_interleave(4, 1)) * 128 ** -0.5 * W("left.temp", (H,))[:, None, None]
    sc = torch.einsum("gh,hts->gts", W("left.talk", (H, H)), sc)
    p = _softmax(sc, 1024, W("left.sink", (H,))[:, None, None])
    left = torch.einsum("hts,shd->thd", p, v.repeat_interleave(4, 1)).reshape(T, H * 128) @ W("left.o", (D, H * 128)).T
    q, k, v = ((h @ W("right." + n, (G * d, D)).T).view(T, G, d) for n, d in (("q", 128), ("k", 128), ("v", 256)))
    q = q * 128 ** -0.5
    z = (h @ W("right.a1", (16, D)).T) @ W("right.a2", (G * 128, 16)).T + W("right.a2.b", (G * 128,))
    a = (torch.sigmoid(z) ** 0.125).view(T, G, 128)
    S, ys = torch.zeros((G, 128, 256), dtype=F64, device=h.device), []
    for t in range(T):
        S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        ys.append((q[t][:, None] @ S)[:, 0])
    o = (_rms(torch.stack(ys)) * W("right.norm", (256,))).reshape(T, G * 256) * _silu(h @ W("right.g", (G * 256, D)).T)
    right = o @ W("right.o", (D, G * 256)).T
    return 0.5 * (_rms(left, W("left.out", (D,))) + _rms(right, W("right.out", (D,))))


def _differential(h, W, s):
    D, T, H, G = h.shape[1], h.shape[0], s["heads"], s["heads"] // 2

    def proj(n, heads):
        return _conv(h @ W(n, (heads * 128, D)).T + W(n + ".b", (heads * 128,)), W(n + ".conv", (heads * 128, 4))).view(T, heads, 128)

    q, k, v = proj("q", H), proj("k", G), proj("v", G)
    pos = torch.arange(T, device=h.device)
    q = q * (1.0 + 0.1 * torch.log((pos + 1).div(1024, rounding_mode="floor").to(F64) + 1.0))[:, None, None]
    lam = (torch.exp((W("lq1", (64,)) * W("lk1", (64,))).sum()) - torch.exp((W("lq2", (64,)) * W("lk2", (64,))).sum()) + 0.5)
    o = _attend(q[..., :64], k[..., :64], v, 0.125) - lam * _attend(q[..., 64:], k[..., 64:], v, 0.125)
    return (_rms(o) * 0.5).reshape(T, H * 128) @ W("o", (D, H * 128)).T


def _latent(h, W, s, base, pairs, window, sink, gate):
    D, T, H, R = h.shape[1], h.shape[0], s["heads"], s["rank"]
    q = (_rms(h @ W("dq", (3 * R, D)).T, W("dq.norm", (3 * R,))) @ W("uq", (H * 192, 3 * R)).T).view(T, H, 192)
    d = h @ W("dkv", (R + 64, D)).T
    c = _rms(d[:, :R], W("dkv.norm", (R,)))
    r = _turn(d[:, None, R:], base, 64, pairs).expand(T, H, 64)
    q = torch.cat([q[..., :128], _turn(q[..., 128:], base, 64, pairs)], -1)
    k = torch.cat([(c @ W("uk", (H * 128, R)).T).view(T, H, 128), r], -1)
    o = _attend(q, k, (c @ W("uv", (H * 128, R)).T).view(T, H, 128), 192 ** -0.5, window, W("sink", (H,)) if sink else None)
    o = o.reshape(T, H * 128)
    if gate:
        o = o * torch.sigmoid(h @ W("g", (H * 128, D)).T)
    return o @ W("o", (D, H * 128)).T


def _lightning(h, W, s):
    D, T, H = h.shape[1], h.shape[0], s["heads"]
    q, k, v = (_silu(h @ W(n, (H * 128, D)).T).view(T, H, 128) for n in ("q", "k", "v"))
    a = torch.tensor(_decays(H), dtype=F64, device=h.device)[:, None, None]
    S, ys = torch.zeros((H, 128, 128), dtype=F64, device=h.device), []
    for t in range(T):
        S = a * S + k[t][:, :, None] * v[t][:, None, :]
        ys.append((q[t][:, None] @ S)[:, 0])
    o = _rms(torch.stack(ys).reshape(T, H * 128), W("norm", (H * 128,)))
    return (o * torch.sigmoid(h @ W("g", (H * 128, D)).T)) @ W("o", (D, H * 128)).T


def _by_request(x, lengths, mixer):
    return torch.cat([mixer(t) for t in x.split(lengths)])


def _qwen_layer(x, W, s, lengths):
    H, G, D = s["heads"], s["kv"], x.shape[1]
    a = _rms(x, W("input_layernorm.weight", (D,)))

    def proj(n, heads):
        return (a @ W(f"self_attn.{n}_proj.weight", (heads * 128, D)).T + W(f"self_attn.{n}_proj.bias", (heads * 128,))).view(-1, heads, 128)

    parts = [t.split(lengths) for t in (proj("q", H), proj("k", G), proj("v", G))]
    o = torch.cat([_attend(_turn(q, 1e6, 128, False), _turn(k, 1e6, 128, False), v, 128 ** -0.5) for q, k, v in zip(*parts)])
    x = x + o.reshape(-1, H * 128) @ W("self_attn.o_proj.weight", (D, H * 128)).T
    a = _rms(x, W("post_attention_layernorm.weight", (D,)))

    def swiglu(t, n, ff):
        return (_silu(t @ W(n + "gate_proj.weight", (ff, D)).T) * (t @ W(n + "up_proj.weight", (ff, D)).T)) @ W(n + "down_proj.weight", (D, ff)).T

    p, sel = torch.softmax(a @ W("mlp.gate.weight", (s["experts"], D)).T, -1).topk(s["top"], -1)
    y = torch.sigmoid(a @ W("mlp.shared_expert_gate.weight", (1, D)).T) * swiglu(a, "mlp.shared_expert.", s["shared"])
    for e in range(s["experts"]):
        r, j = torch.nonzero(sel == e, as_tuple=True)
        if r.numel():
            y.index_add_(0, r, p[r, j][:, None] * swiglu(a[r], f"mlp.experts.{e}.", s["eff"]))
    return x + y


def exact(case, seed):
    c, s = case, SIZES[case["size"]]
    D, V, lengths = s["width"], c["vocab"], [n + c["steps"] for n in _lengths(c)]

    def W(name, shape):
        return _tensor(c, seed, name, shape).to(F64)

    def under(prefix):
        return lambda name, shape: W(prefix + name, shape)

    ids = torch.tensor([t for toks in _tokens(c, seed) for t in toks], device="cuda")
    qwen = c["arch"] == "qwen2_moe"
    x = _tensor(c, seed, "model.embed_tokens.weight" if qwen else "embed", (V, D))[ids].to(F64)

    def dyt(t, n):
        return torch.tanh(W(n + ".alpha", ()) * t) * W(n, (D,)) + W(n + ".b", (D,))

    if qwen:
        for i in range(c["layers"]):
            x = _qwen_layer(x, under(f"model.layers.{i}."), s, lengths)
        x, head = _rms(x, W("model.norm.weight", (D,))), W("lm_head.weight", (V, D))
    elif c["arch"] == "Balalorn":
        for i, mixer in enumerate((_mamba2, _delta)):
            x = x + _rms(_by_request(x, lengths, lambda t: mixer(t, under(f"l{i}.mix."), s)), W(f"l{i}.norm1", (D,)))
        x, head = _rms(x, W("final.norm", (D,))), W("head", (V, D))
    elif c["arch"] == "Govuvik":
        x = _rms(x, W("embed.norm", (D,)))
        for i, mixer in enumerate((_mlstm, _parallel)):
            h = _rms(x, W(f"l{i}.norm1", (D,)))
            y = _by_request(h, lengths, lambda t: mixer(t + _conv(t, W(f"l{i}.canon1", (D, 3))), under(f"l{i}.mix."), s))
            x = x + _rms(y, W(f"l{i}.norm1b", (D,)))
        x, head = _rms(x, W("final.norm", (D,))), W("head", (V, D))
    elif c["arch"] == "Dimuvik":
        for i, mixer in enumerate((_differential, lambda t, w, z: _latent(t, w, z, 10000.0, True, 0, True, False))):
            x = x + dyt(_by_request(dyt(x, f"l{i}.norm1"), lengths, lambda t: mixer(t, under(f"l{i}.mix."), s)), f"l{i}.norm1b")
        x, head = dyt(x, "final.norm"), W("head", (V, D))
    else:
        for i, mixer in enumerate((_lightning, lambda t, w, z: _latent(t, w, z, 50000.0, False, 1024, False, True))):
            x = x + _by_request(_rms(x, W(f"l{i}.norm1", (D,))), lengths, lambda t: mixer(t, under(f"l{i}.mix."), s))
        x, head = _rms(x, W("final.norm", (D,))), W("embed", (V, D))
    start = [sum(lengths[:i]) for i in range(len(lengths))]
    out = []
    for step in _plan(c):
        rows = [start[i] + a + w for i, a, _, want in step for w in want]
        z = x[torch.tensor(rows, device=x.device)] @ head.T
        out.append(50.0 * torch.tanh(z / 50.0) if c["arch"] == "Govuvik" else z)
    return torch.cat(out)
