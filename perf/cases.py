"""The work that the engine's speed is measured on: steps of the engine's step function.

A case is one step through `ModelRunner`, the call under `Engine` and `bin/trace_run`: prompt steps (`ModelRunner.step`
with the tokens of one or several requests, whole prompts from an empty cache) and decode steps
(`ModelRunner.decode_tokens`, one token for each of several requests that hold a context).  The models have the layer sizes
of `bench.py` and random weights: Falcon-H1 at the 0.5B and 7B sizes, and one period of the layers of Boketar, Nikodra and
Sorovik, which between them hold every kind of mixer state (pages behind windows, in chunks, of latents; state-space,
delta-rule, retention and time-mixing states) and both kinds of feed-forward (dense, routed).  Two cases are whole models of
36 layers, the others a few layers, so that a change of rounding does not travel far.

A step returns its logits and the state that it leaves: the requests' fixed-size states and, after prompt steps, the pages.
`exact` has the same in float64 from plain formulas.
"""
import math

import numpy as np
import torch

import poor_mans_mamba_b200.architectures  # noqa: F401  (registers the architectures)
from poor_mans_mamba_b200.cache import CacheManager
from poor_mans_mamba_b200.config.registry import resolve_architecture
from poor_mans_mamba_b200.engine import Model, ModelRunner, StepEntry

DEVICE = "cuda:0"
PAGE = 64
LAP = 128      # a decode case starts over from its first context after so many steps, so that its cost does not drift


# ----------------------------------------------------------------------------- the models
def falcon_config(layers, sizes):
    cfg = {"model_type": "falcon_h1", "num_hidden_layers": layers, "hidden_size": 1024, "vocab_size": 32784,
           "intermediate_size": 2048, "num_attention_heads": 8, "num_key_value_heads": 2, "head_dim": 64, "rope_theta": 1e11,
           "attention_bias": False, "mlp_bias": False, "mamba_d_ssm": 1536, "mamba_n_heads": 24, "mamba_d_head": 64,
           "mamba_d_state": 128, "mamba_n_groups": 1, "mamba_d_conv": 4, "mamba_chunk_size": 128, "mamba_conv_bias": True,
           "mamba_proj_bias": False, "mamba_rms_norm": False, "mamba_norm_before_gate": False, "rms_norm_eps": 1e-5,
           "hidden_act": "silu", "tie_word_embeddings": False, "embedding_multiplier": 1.0, "lm_head_multiplier": 1.0,
           "attention_in_multiplier": 1.0, "attention_out_multiplier": 1.0, "key_multiplier": 1.0, "ssm_in_multiplier": 1.0,
           "ssm_out_multiplier": 1.0, "ssm_multipliers": [1.0] * 5, "mlp_multipliers": [1.0, 1.0],
           "bos_token_id": 1, "eos_token_id": 11, "pad_token_id": 0}
    if sizes == "7b":
        cfg.update(hidden_size=3072, num_attention_heads=12, num_key_value_heads=2, head_dim=128, intermediate_size=12288,
                   vocab_size=130049, mamba_d_ssm=6144, mamba_n_heads=48, mamba_d_head=128, mamba_d_state=256,
                   mamba_chunk_size=256)
    return cfg


def decays(heads):
    return [1.0 - 2.0 ** -(4 + 6 * h / (heads - 1)) for h in range(heads)]


def boketar_config(layers):
    delta = {"heads": 8, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
    left = {"heads": 8, "kv_heads": 2, "dim": 64, "vdim": 64, "conv": 3, "mask": {"size": 1024}, "scale": 0.125,
            "rot": {"dims": 64, "base": 1e6}}
    right = {"heads": 8, "dim": 64, "vdim": 128, "decay": decays(8)}
    kinds = [("channel_delta", delta), ("parallel", {"left": left, "right": right})]
    return {"architecture": "Boketar", "vocab": 32784, "width": 1024, "streams": 2, "embedding": {"scale": 1.0},
            "norm": {"eps": 1e-6},
            "layers": [dict(zip(("type", "mixer"), kinds[i % 2]), mlp={"kind": "dense", "ff": 2048}) for i in range(layers)]}


def nikodra_config(layers):
    att = {"heads": 8, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.125, "v_mix": True,
           "rot": {"dims": 64, "base": 5e5, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    left = {"heads": 8, "kv_heads": 2, "dim": 64, "vdim": 64, "mask": {"size": 1024}, "scale": 0.125}
    right = {"heads": 8, "dim": 64, "vdim": 128, "decay": decays(8), "rot": {"dims": 64, "base": 1e6}}
    kinds = [("attention", att), ("parallel", {"left": left, "right": right}),
             ("wkv", {"heads": 16, "dim": 64, "decay_rank": 64}), ("attention", att)]
    return {"architecture": "Nikodra", "vocab": 32784, "width": 1024, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "embedding": {"bigram": {"buckets": 50021, "mul_prev": 8191, "mul_cur": 131}},
            "layers": [dict(zip(("type", "mixer"), kinds[i % 4]), mlp={"kind": "dense", "ff": 3072}) for i in range(layers)]}


def sorovik_config(layers):
    lat = {"heads": 8, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 96, "scale": 96 ** -0.5, "rot": {"dims": 32, "base": 1e6},
           "mask": {"size": 1024}}
    att = {"heads": 8, "kv_heads": 2, "dim": 64, "vdim": 64, "conv": 3, "scale": 0.125, "rot": {"dims": 32, "base": 5e4},
           "mask": {"size": 1024, "keep_first": 4}}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 4, "groups": {"count": 4, "keep": 2}}, "expert": {"ff": 256}}
    out = []
    for i in range(layers):
        ffn = {"kind": "dense", "ff": 2048} if i == 0 else moe
        if i % 4 == 1:
            out.append({"type": "attention", "mixer": att, "mlp": ffn})
        else:
            out.append({"type": "latent_attention", "mixer": dict(lat, kv_from=i - 1) if i % 4 == 3 else lat, "mlp": ffn})
    return {"architecture": "Sorovik", "vocab": 32784, "width": 1024, "norm": {"eps": 1e-6}, "layers": out}


def config_of(case):
    if case["model"] == "falcon":
        return falcon_config(case["layers"], case["sizes"])
    return {"boketar": boketar_config, "nikodra": nikodra_config, "sorovik": sorovik_config}[case["model"]](case["layers"])


# ----------------------------------------------------------------------------- the cases
def prompt(name, model, layers, tokens, seqs=1, rows=1, sizes="0.5b"):
    """`tokens` in `seqs` requests of unequal lengths; the logits of the last `rows` tokens of each are wanted."""
    return {"name": name, "kind": "prompt", "model": model, "sizes": sizes, "layers": layers, "tokens": tokens, "seqs": seqs,
            "rows": rows}


def decode(name, model, layers, batch, context, sizes="0.5b"):
    return {"name": name, "kind": "decode", "model": model, "sizes": sizes, "layers": layers, "batch": batch, "context": context}


def listed():
    return [
        # one user's reply, token by token: the smallest step there is, bound by its chain of launches
        decode("falcon-decode-1x700", "falcon", 8, 1, 700),
        # the benchmark's decode step, the whole model
        decode("falcon-decode-8x2048-whole", "falcon", 36, 8, 2048),
        # a busy server's decode step, as many requests as the engine takes by default
        decode("falcon-decode-64x1000", "falcon", 8, 64, 1000),
        # a short question
        prompt("falcon-prompt-37", "falcon", 8, 37),
        # the benchmark's prompt step, the whole model
        prompt("falcon-prompt-2048-whole", "falcon", 36, 2048),
        # several prompts of unequal lengths admitted in one step
        prompt("falcon-prompts-5-of-1403", "falcon", 8, 1403, seqs=5),
        # a prompt through the 7B layer sizes, where the products are large
        prompt("falcon-7b-prompt-1024", "falcon", 2, 1024, sizes="7b"),
        # a full step of the scheduler's token budget through delta rule, window attention and retention
        prompt("boketar-prompt-2048", "boketar", 4, 2048, rows=16),
        # a batch of replies through the same
        decode("boketar-decode-8x1500", "boketar", 4, 8, 1500),
        # a prompt of a length that is a multiple of nothing through chunked attention, retention and time mixing
        prompt("nikodra-prompt-1501", "nikodra", 4, 1501, rows=16),
        # a full step through latent attention and routed experts, and a batch of replies through the same
        prompt("sorovik-prompt-2048", "sorovik", 4, 2048, rows=16),
        decode("sorovik-decode-8x1000", "sorovik", 4, 8, 1000),
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["falcon", "falcon", "boketar", "nikodra", "sorovik"])
    layers = 8 if model == "falcon" else 4
    if rng.random() < 0.6:
        tokens = log_uniform(rng, 17, 2048)
        seqs = rng.randint(2, 8) if tokens > 200 and rng.random() < 0.35 else 1
        case = prompt("", model, layers, tokens, seqs, rows=rng.choice([1, 1, 7, 16]) if seqs == 1 else 1)
    else:
        case = decode("", model, layers, log_uniform(rng, 1, 64), log_uniform(rng, 50, 2000))
    del case["name"]
    return case


def lengths(case):
    """Tokens of each request of a prompt step: unequal, none empty."""
    n, t = case["seqs"], case["tokens"]
    weights = [2 + (5 * i) % 7 for i in range(n)]
    out = [max(1, t * w // sum(weights)) for w in weights]
    out[0] += t - sum(out)
    return out


def wanted(case):
    """Per request the number of last tokens whose logits come back."""
    return [min(case["rows"], n) for n in lengths(case)]


# ----------------------------------------------------------------------------- inputs
def weights_of(case, model, seed):
    """Random tensors by the rules that the parts declare for themselves; the convolution taps of Falcon-H1 are drawn as
    wide as the other models' (0.5), so that its state-space branch carries a share of the stream."""
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 17)
    out = {}
    for name, spec in model.param_specs().items():
        rule = ("normal", 0.5) if name.endswith("conv1d.weight") else spec.init
        shape = tuple(spec.shape)
        if rule[0] in ("ones", "zeros"):
            t = torch.full(shape, 1.0 if rule[0] == "ones" else 0.0, device=DEVICE)
        elif rule[0] == "normal":
            t = torch.randn(shape, generator=g, device=DEVICE) * float(rule[1])
        else:
            u = torch.rand(shape, generator=g, device=DEVICE)
            lo, hi = float(rule[1]), float(rule[2])
            if rule[0] == "uniform":
                t = lo + (hi - lo) * u
            elif rule[0] == "log_uniform":
                t = torch.log(lo + (hi - lo) * u)
            else:  # the inverse softplus of a log-uniform step
                step = torch.exp(math.log(lo) + (math.log(hi) - math.log(lo)) * u)
                t = step + torch.log(-torch.expm1(-step))
        t = t.to(torch.bfloat16)
        out[name] = t.contiguous() if spec.kind == "matrix" else t.float().contiguous()
    return out


def token_ids(case, seed, vocab):
    """Prompt steps: the tokens of each request.  Decode steps: [batch, context] and one more for each request."""
    rng = np.random.RandomState((seed * 104729 + 5) % (1 << 31))
    if case["kind"] == "prompt":
        return [rng.randint(0, vocab, n).astype(np.int32) for n in lengths(case)]
    return rng.randint(0, vocab, (case["batch"], case["context"] + 1)).astype(np.int32)


def build_model(case, seed):
    cfg = config_of(case)
    arch = resolve_architecture(cfg)
    model = Model(arch.model_spec(arch.parse(cfg)))
    model.bind(weights_of(case, model, seed), torch.bfloat16, torch.device(DEVICE))
    return model


class State:
    pass


def prepare(case, seed):
    """A server that is up: model, cache, runner with graphs; the shape of the step has come before, so it is recorded.
    For a decode step the requests' contexts have been fed."""
    s = State()
    s.case = case
    model = build_model(case, seed)
    ids = token_ids(case, seed, model.vocab_size)
    if case["kind"] == "prompt":
        longest, slots, held = 2048, 8, case["tokens"] + PAGE * case["seqs"]
    else:
        longest, slots = 4096, max(8, 1 << (case["batch"] - 1).bit_length())
        held = case["batch"] * (case["context"] + LAP + PAGE)
    s.cache = CacheManager(model.state_specs(), page_size=PAGE, num_pages=held // PAGE + 2, num_slots=slots,
                           dtype=torch.bfloat16, device=DEVICE)
    s.runner = ModelRunner(model, s.cache)
    s.runner.enable_graphs(longest)
    if case["kind"] == "prompt":
        s.entries = [StepEntry(("p", i), t, list(range(len(t) - r, len(t)))) for i, (t, r) in enumerate(zip(ids, wanted(case)))]
        n_live = case["seqs"]
        for _ in range(3):
            run_prompt(s)
    else:
        s.reqs = [("d", i) for i in range(case["batch"])]
        s.tokens = [int(t) for t in ids[:, -1]]
        n_live = case["batch"]
        for r, row in zip(s.reqs, ids):
            for a in range(0, case["context"], 2048):
                s.runner.step([StepEntry(r, row[a:min(a + 2048, case["context"])], [])])
        for at in (case["context"] + 1, case["context"] + LAP):
            s.runner.graphs.bucket_for(case["batch"], at)
    tables = {k: torch.zeros((1, 1), dtype=torch.int32, device=DEVICE) for k in s.cache.groups}
    views = s.cache.layer_caches(tables)
    s.states = {}
    for layer, specs in sorted(model.state_specs().items()):
        for name, spec in specs:
            if spec.kind == "fixed" and name not in s.states:  # the layers' states of one name are slices of one tensor
                t = views[layer].fixed(name)
                s.states[name] = (t if t._base is None else t._base)[:, :n_live]
    s.pages = {}
    if case["kind"] == "prompt":
        s.pages = {"pages%d" % i: g.storage[:, :g.num_pages] for i, g in enumerate(s.cache.groups.values())}
    torch.cuda.synchronize()
    return s


def run_prompt(s):
    logits = s.runner.step(s.entries)
    for e in reversed(s.entries):  # the next step's requests find the slots in the same order
        s.runner.finish(e.req)
    return logits


def start_over(s):
    """The requests end and others of the same context take their places (nothing is computed for them)."""
    for r in reversed(s.reqs):
        s.runner.finish(r)
    for r in s.reqs:
        s.runner.start(r)
        s.cache.grow(r, s.case["context"])
        s.cache.advance(r, s.case["context"])


def run(s):
    if s.case["kind"] == "prompt":
        return {"logits": run_prompt(s), **s.states, **s.pages}
    if s.runner.length(s.reqs[0]) >= s.case["context"] + LAP:
        start_over(s)
    s.runner.decode_tokens(s.reqs, s.tokens)
    return {"logits": s.runner.graphs.last_logits(len(s.reqs)), **s.states}


# ----------------------------------------------------------------------------- what a step cannot do without
def mixers(cfg):
    """("attend", heads, key + value entries a head, cache row entries, window) and ("state", entries of the state)."""
    out = []
    if cfg.get("model_type") == "falcon_h1":
        d, kv = cfg["head_dim"], cfg["num_key_value_heads"]
        for _ in range(cfg["num_hidden_layers"]):
            out.append(("attend", cfg["num_attention_heads"], 2 * d, 2 * kv * d, 0))
            out.append(("state", cfg["mamba_n_heads"] * cfg["mamba_d_head"] * cfg["mamba_d_state"]))
        return out
    for layer in cfg["layers"]:
        parts = [layer["mixer"]] if "left" not in layer["mixer"] else [layer["mixer"]["left"], layer["mixer"]["right"]]
        for m in parts:
            window = (m.get("mask") or {}).get("size", 0)
            if "kv_rank" in m:  # a latent row serves all heads as key and as value
                out.append(("attend", m["heads"], 2 * m["kv_rank"] + m["rot_dim"], m["kv_rank"] + m["rot_dim"], window))
            elif "scale" in m:
                out.append(("attend", m["heads"], m["dim"] + m["vdim"], m["kv_heads"] * (m["dim"] + m["vdim"]), window))
            else:
                out.append(("state", m["heads"] * m["dim"] * m.get("vdim", m["dim"])))
    return out


def work(case):
    cfg = config_of(case)
    arch = resolve_architecture(cfg)
    specs = Model(arch.model_spec(arch.parse(cfg))).param_specs()
    D, V = cfg.get("hidden_size", cfg.get("width")), cfg.get("vocab_size", cfg.get("vocab"))
    if case["kind"] == "prompt":
        seqs, new, past = case["seqs"], lengths(case), [0] * case["seqs"]
        rows = sum(wanted(case))
    else:
        seqs, new, past = case["batch"], [1] * case["batch"], [case["context"]] * case["batch"]
        rows = seqs
    T = sum(new)
    expert = dense = 0
    for name, spec in specs.items():
        if name in ("embed", "bigram", "model.embed_tokens.weight", "head", "lm_head.weight") or len(spec.shape) < 2:
            continue
        n = int(np.prod(spec.shape))
        if ".mlp.e" in name:
            expert += n
        else:
            dense += n
    top, experts = 4, 16  # of the routed feed-forwards
    flops = 2.0 * T * (dense + expert * top / experts) + 2.0 * rows * D * V
    size = 2.0 * (dense + expert * min(1.0, T * top / experts) + D * V + T * D) + 4.0 * rows * V
    for m in mixers(cfg):
        if m[0] == "state":
            flops += 5.0 * T * m[1]
            size += (4.0 if case["kind"] == "prompt" else 8.0) * seqs * m[1]
            continue
        _, heads, entries, row, window = m
        for n, p in zip(new, past):
            seen = [min(p + i + 1, window or (1 << 30)) for i in range(n)]
            flops += 2.0 * heads * entries * sum(seen)
            size += 2.0 * row * (n + (min(p, window or p)))
    return {"bytes": size, "flops": flops}


def tolerance(case):
    # Relative to the result's norm, of two implementations that round alike.  Measured: against float64 the logits are off by
    # 0.015 after 8 layers of Falcon-H1 in bfloat16, 0.03 after 36, 0.007 after 4 of Boketar, 0.01 to 0.035 (a single row)
    # after 4 of Nikodra, 0.03 to 0.06 after 4 of Sorovik, whose routed feed-forward's choice between nearly equal experts
    # falls one way or the other with the rounding before it and moves whole rows; two runs of the same Falcon-H1 code,
    # whose output products add in no fixed order, differ by 0.005 after 8 layers and 0.007 after 36.
    if case["model"] == "sorovik":
        return {"rel": 0.03, "max": 0.9}
    if case["model"] == "boketar":
        return {"rel": 0.02, "max": 0.4}
    return {"rel": 0.03 if case["model"] == "nikodra" or case["layers"] > 8 else 0.025, "max": 0.6}


# ----------------------------------------------------------------------------- the same in float64
def silu(x):
    return x * torch.sigmoid(x)


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def causal_conv(u, w):
    """u [B, T, C], w [C, taps], zeros before the start."""
    T, taps = u.shape[1], w.shape[1]
    padded = torch.nn.functional.pad(u, (0, 0, taps - 1, 0))
    return sum(padded[:, j:j + T] * w[:, j] for j in range(taps))


def last_rows(u, n):
    """The last n rows of u [B, T, C], zeros before the start."""
    return torch.nn.functional.pad(u, (0, 0, n, 0))[:, -n:]


def rotate(x, freq, halves, amplitude=1.0):
    """x [B, T, heads, d], the first 2 len(freq) entries: pairs (i, i + n) with `halves`, else (2i, 2i + 1)."""
    n = freq.shape[0]
    ang = torch.arange(x.shape[1], device=x.device).to(freq.dtype)[:, None] * freq
    c, s = (torch.cos(ang.double()) * amplitude)[:, None], (torch.sin(ang.double()) * amplitude)[:, None]
    out = x.clone()
    i, j = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
    out[..., i] = x[..., i] * c - x[..., j] * s
    out[..., j] = x[..., j] * c + x[..., i] * s
    return out


def plain_freq(dims, base):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=DEVICE)


def attend(q, k, v, scale, visible, extra=None):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv]; visible [T, T]; `extra` [H]: a score without a value."""
    B, T, H, _ = q.shape
    rep = H // k.shape[2]
    out = []
    for b in range(B):
        s = torch.einsum("thd,shd->hts", q[b], k[b].repeat_interleave(rep, 1)) * scale
        s = s.masked_fill(~visible, -math.inf)
        if extra is not None:
            s = torch.cat([s, extra[:, None, None].expand(H, T, 1)], -1)
        p = torch.softmax(s, -1)[..., :T]
        out.append(torch.einsum("hts,shd->thd", p, v[b].repeat_interleave(rep, 1)))
    return torch.stack(out)


def visible_pairs(T, window=0, keep_first=0, chunk=0):
    i = torch.arange(T, device=DEVICE)
    m = i[None, :] <= i[:, None]
    if chunk:
        m &= i[:, None] // chunk == i[None, :] // chunk
    if window:
        m &= (i[:, None] - i[None, :] < window) | (i[None, :] < keep_first)
    return m


def recurrence(q, k, v, g, beta=None, bonus=None):
    """Per head S <- g S + k u^T, o = S^T q.  q, k, g [B, T, H, d], v [B, T, H, dv].  u = v, or with `beta` [B, T, H] the delta
    rule's beta (v - S^T k) on the decayed state.  With `bonus` [H, d] o reads the state before the step plus
    diag(bonus) k v^T, and the decay follows.  Returns o and the last S."""
    B, T, H, d = q.shape
    S = torch.zeros(B, H, d, v.shape[3], dtype=q.dtype, device=q.device)
    o = torch.empty(B, T, H, v.shape[3], dtype=q.dtype, device=q.device)
    for t in range(T):
        kt, u = k[:, t, :, :, None], v[:, t]
        if bonus is not None:
            kv = kt * u[:, :, None]
            o[:, t] = ((S + bonus[..., None] * kv) * q[:, t, :, :, None]).sum(2)
            S = S * g[:, t, :, :, None] + kv
            continue
        S = S * g[:, t, :, :, None]
        if beta is not None:
            u = beta[:, t, :, None] * (u - (S * kt).sum(2))
        S = S + kt * u[:, :, None]
        o[:, t] = (S * q[:, t, :, :, None]).sum(2)
    return o, S


class Oracle:
    """Whole sequences [B, T] from an empty cache through one model, in float64; `left` collects the states."""

    def __init__(self, case, seed):
        cfg = config_of(case)
        arch = resolve_architecture(cfg)
        self.cfg = cfg
        self.W = {k: v.double() for k, v in weights_of(case, Model(arch.model_spec(arch.parse(cfg))), seed).items()}
        self.left = {}

    def leave(self, name, value):
        self.left.setdefault(name, []).append(value)

    def lin(self, x, name):
        return x @ self.W[name].t() + (self.W[name + ".b"] if name + ".b" in self.W else 0.0)

    def forward(self, ids, rows):
        """Logits [B, rows, V] of the last `rows` tokens."""
        return getattr(self, "falcon" if "model_type" in self.cfg else self.cfg["architecture"].lower())(ids, rows)

    # ---- Falcon-H1
    def falcon(self, ids, rows):
        c, W, eps = self.cfg, self.W, self.cfg["rms_norm_eps"]
        B, T = ids.shape
        H, G, d = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        I, N, Hs, P = c["mamba_d_ssm"], c["mamba_d_state"], c["mamba_n_heads"], c["mamba_d_head"]
        i = torch.arange(d // 2, dtype=torch.float32, device=DEVICE)
        freq = 1.0 / torch.pow(torch.tensor(c["rope_theta"], dtype=torch.float32, device=DEVICE), 2.0 * i / d)
        see = visible_pairs(T)
        x = W["model.embed_tokens.weight"][ids]
        for l in range(c["num_hidden_layers"]):
            p = "model.layers.%d." % l
            n = rms(x, eps) * W[p + "input_layernorm.weight"]
            z, u, dt = self.lin(n, p + "mamba.in_proj.weight").split([I, I + 2 * N, Hs], -1)
            a = silu(causal_conv(u, W[p + "mamba.conv1d.weight"]) + W[p + "mamba.conv1d.bias"])
            self.leave("mamba.conv", last_rows(u, c["mamba_d_conv"] - 1))
            xs, b, cc = a.split([I, N, N], -1)
            xs = xs.reshape(B, T, Hs, P)
            delta = torch.nn.functional.softplus(dt + W[p + "mamba.dt_bias"])
            da = torch.exp(-delta * torch.exp(W[p + "mamba.A_log"]))
            S = torch.zeros(B, Hs, P, N, dtype=torch.float64, device=DEVICE)
            y = torch.empty_like(xs)
            for t in range(T):
                S = S * da[:, t, :, None, None] + (delta[:, t, :, None] * xs[:, t])[..., None] * b[:, t, None, None]
                y[:, t] = torch.einsum("bhpn,bn->bhp", S, cc[:, t])
            self.leave("mamba.ssm", S)
            y = (y + W[p + "mamba.D"][:, None] * xs).reshape(B, T, I) * silu(z)
            q = rotate(self.lin(n, p + "self_attn.q_proj.weight").reshape(B, T, H, d), freq, True)
            k = rotate(self.lin(n, p + "self_attn.k_proj.weight").reshape(B, T, G, d), freq, True)
            v = self.lin(n, p + "self_attn.v_proj.weight").reshape(B, T, G, d)
            o = attend(q, k, v, d ** -0.5, see).reshape(B, T, H * d)
            x = x + self.lin(y, p + "mamba.out_proj.weight") + self.lin(o, p + "self_attn.o_proj.weight")
            f = p + "feed_forward."
            n = rms(x, eps) * W[p + "pre_ff_layernorm.weight"]
            x = x + self.lin(silu(self.lin(n, f + "gate_proj.weight")) * self.lin(n, f + "up_proj.weight"), f + "down_proj.weight")
        return self.lin(rms(x[:, -rows:], eps) * W["model.final_layernorm.weight"], "lm_head.weight")

    # ---- Boketar
    def boketar(self, ids, rows):
        c, W, eps = self.cfg, self.W, self.cfg["norm"]["eps"]
        xs = [W["embed"][ids]] * 2

        def sub(xs, p, q, fn):
            w_in, w_out, w_mix = W["%shc%d.in" % (p, q)], W["%shc%d.out" % (p, q)], W["%shc%d.mix" % (p, q)]
            y = fn(rms(w_in[0] * xs[0] + w_in[1] * xs[1], eps) * (1.0 + W["%snorm%d" % (p, q)]))
            return [w_mix[0, t] * xs[0] + w_mix[1, t] * xs[1] + w_out[t] * y for t in range(2)]

        for l, layer in enumerate(c["layers"]):
            p, m = "l%d." % l, layer["mixer"]
            mix = self.channel_delta if layer["type"] == "channel_delta" else self.boketar_parallel
            xs = sub(xs, p, 1, lambda h: mix(h, p + "mix.", m, eps))
            p += "mlp."
            xs = sub(xs, p[:-4], 2, lambda h: self.lin(silu(self.lin(h, p + "gate")) * self.lin(h, p + "up"), p + "down"))
        return self.lin(rms((xs[0] + xs[1])[:, -rows:], eps) * (1.0 + W["final.norm"]), "head")

    def channel_delta(self, h, p, m, eps):
        W, (B, T), H, d = self.W, h.shape[:2], m["heads"], m["dim"]
        u = torch.cat([self.lin(h, p + s) for s in "qkv"], -1)
        self.leave("mix.conv", last_rows(u, m["conv"] - 1))
        q, k, v = silu(causal_conv(u, torch.cat([W[p + s + ".conv"] for s in "qkv"]))).reshape(B, T, 3 * H, d).split(H, 2)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        a = self.lin(self.lin(h, p + "a1"), p + "a2") + W[p + "dt_bias"]
        g = torch.exp(-torch.exp(W[p + "A_log"])[:, None] * torch.nn.functional.softplus(a).reshape(B, T, H, d))
        o, S = recurrence(q, k, v, g, beta=torch.sigmoid(self.lin(h, p + "b")))
        self.leave("mix.S", S)
        gate = torch.sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2")).reshape(B, T, H, d)
        return self.lin((rms(o, eps) * W[p + "norm"] * gate).reshape(B, T, H * d), p + "o")

    def boketar_parallel(self, h, p, m, eps):
        W, (B, T), L, R = self.W, h.shape[:2], m["left"], m["right"]
        H, G, d, lp, rp = L["heads"], L["kv_heads"], L["dim"], p + "left.", p + "right."
        u = torch.cat([self.lin(h, lp + s) for s in "qkv"], -1)
        self.leave("mix.left.conv", last_rows(u, L["conv"] - 1))
        q, k, v = causal_conv(u, torch.cat([W[lp + s + ".conv"] for s in "qkv"])).reshape(B, T, H + 2 * G, d).split([H, G, G], 2)
        freq = plain_freq(L["rot"]["dims"], L["rot"]["base"])
        a = attend(rotate(q, freq, False), rotate(k, freq, False), v, L["scale"], visible_pairs(T, L["mask"]["size"]), W[lp + "sink"])
        left = self.lin(a.reshape(B, T, H * d), lp + "o")
        H, d, dv = R["heads"], R["dim"], R["vdim"]
        q, k, v = (silu(self.lin(h, rp + s)).reshape(B, T, H, n) for s, n in zip("qkv", (d, d, dv)))
        g = torch.tensor(R["decay"], dtype=torch.float64, device=DEVICE)[:, None].expand(B, T, H, 1)
        o, S = recurrence(q, k, v, g)
        self.leave("mix.right.S", S)
        o = rms(o.reshape(B, T, H * dv), eps) * W[rp + "norm"] * torch.sigmoid(self.lin(h, rp + "g"))
        return 0.5 * (rms(left, eps) * W[lp + "out"] + rms(self.lin(o, rp + "o"), eps) * W[rp + "out"])

    # ---- Nikodra
    def nikodra(self, ids, rows):
        c, W, eps = self.cfg, self.W, self.cfg["norm"]["eps"]
        g = c["embedding"]["bigram"]
        pair = torch.full_like(ids, g["buckets"])
        pair[:, 1:] = (ids[:, :-1] * g["mul_prev"] + ids[:, 1:] * g["mul_cur"]) % g["buckets"]
        x = W["embed"][ids] + W["bigram"][pair]
        self.first_values = None
        mix = {"attention": self.mixed_attention, "parallel": self.nikodra_parallel, "wkv": self.wkv}
        for l, layer in enumerate(c["layers"]):
            p = "l%d." % l
            y = mix[layer["type"]](rms(x, eps) * (1.0 + W[p + "norm1"]), p + "mix.", layer["mixer"], eps)
            x = x + c["residual_mult"] * rms(y, eps) * (1.0 + W[p + "norm1b"])
            h = rms(x, eps) * (1.0 + W[p + "norm2"])
            y = self.lin(torch.nn.functional.gelu(self.lin(h, p + "mlp.up")), p + "mlp.down")
            x = x + c["residual_mult"] * rms(y, eps) * (1.0 + W[p + "norm2b"])
        return self.lin(rms(x[:, -rows:], eps) * (1.0 + W["final.norm"]), "head")

    def mixed_attention(self, h, p, m, eps):
        W, (B, T), H, G, d = self.W, h.shape[:2], m["heads"], m["kv_heads"], m["dim"]
        s, n = m["rot"]["scaling"], m["rot"]["dims"]
        freq = plain_freq(n, m["rot"]["base"])
        lo, hi = (n * math.log(s["original"] / (2.0 * math.pi * s[w])) / (2.0 * math.log(m["rot"]["base"])) for w in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), n - 1)
        r = ((torch.arange(n // 2, device=DEVICE, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        freq, amp = freq / s["factor"] * r + freq * (1.0 - r), 0.1 * math.log(s["factor"]) + 1.0
        q = rms(self.lin(h, p + "q").reshape(B, T, H, d), eps) * W[p + "q.norm"]
        k = rms(self.lin(h, p + "k").reshape(B, T, G, d), eps) * W[p + "k.norm"]
        v = self.lin(h, p + "v").reshape(B, T, G, d)
        if self.first_values is None:
            self.first_values = v
        else:
            v = (1.0 - W[p + "vmix"]) * v + W[p + "vmix"] * self.first_values
        one = torch.zeros(H, dtype=torch.float64, device=DEVICE)
        o = attend(rotate(q, freq, False, amp), rotate(k, freq, False, amp), v, m["scale"], visible_pairs(T), one)
        return self.lin(o.reshape(B, T, H * d), p + "o")

    def nikodra_parallel(self, h, p, m, eps):
        W, (B, T), L, R = self.W, h.shape[:2], m["left"], m["right"]
        H, G, d = L["heads"], L["kv_heads"], L["dim"]
        q, k, v = (self.lin(h, p + "left." + s).reshape(B, T, n, d) for s, n in zip("qkv", (H, G, G)))
        one = torch.zeros(H, dtype=torch.float64, device=DEVICE)
        a = attend(rms(q, eps), rms(k, eps), v, L["scale"], visible_pairs(T, chunk=L["mask"]["size"]), one)
        left = self.lin(a.reshape(B, T, H * d), p + "left.o")
        H, d, dv = R["heads"], R["dim"], R["vdim"]
        freq = plain_freq(R["rot"]["dims"], R["rot"]["base"])
        q, k, v = (self.lin(h, p + "right." + s).reshape(B, T, H, n) for s, n in zip("qkv", (d, d, dv)))
        g = torch.tensor(R["decay"], dtype=torch.float64, device=DEVICE)[:, None].expand(B, T, H, 1)
        o, S = recurrence(rotate(q, freq, True), rotate(k, freq, True) * d ** -0.5, v, g)
        self.leave("mix.right.S", S)
        o = rms(o, eps).reshape(B, T, H * dv) * silu(self.lin(h, p + "right.g"))
        return 0.5 * (rms(left, eps) * W[p + "left.out"] + rms(self.lin(o, p + "right.o"), eps) * W[p + "right.out"])

    def wkv(self, h, p, m, eps):
        W, (B, T), H, d = self.W, h.shape[:2], m["heads"], m["dim"]
        self.leave("mix.h", h[:, -1])
        before = torch.nn.functional.pad(h, (0, 0, 1, 0))[:, :-1]
        mix = {s: h + (before - h) * W[p + "mu." + s] for s in "rkvgw"}
        r, k, v = (self.lin(mix[s], p + s).reshape(B, T, H, d) for s in "rkv")
        w = torch.exp(-torch.exp(self.lin(torch.tanh(self.lin(mix["w"], p + "w1")), p + "w2") + W[p + "w0"])).reshape(B, T, H, d)
        o, S = recurrence(r, k, v, w, bonus=W[p + "u"])
        self.leave("mix.S", S)
        return self.lin(rms(o, eps).reshape(B, T, H * d) * W[p + "norm"] * silu(self.lin(mix["g"], p + "g")), p + "o")

    # ---- Sorovik
    def sorovik(self, ids, rows):
        c, W, eps = self.cfg, self.W, self.cfg["norm"]["eps"]
        x = rms(W["embed"][ids], eps) * W["embed.norm"]
        latents = {}
        for l, layer in enumerate(c["layers"]):
            p, m = "l%d." % l, layer["mixer"]
            h = rms(x, eps) * W[p + "norm1"]
            if layer["type"] == "attention":
                y = self.conv_attention(h, p + "mix.", m, eps)
            else:
                freq = plain_freq(m["rot"]["dims"], m["rot"]["base"])
                if m.get("kv_from") is None:
                    low = self.lin(h, p + "mix.dkv")
                    R = m["kv_rank"]
                    latents[l] = (rms(low[..., :R], eps) * W[p + "mix.dkv.norm"], rotate(low[..., None, R:], freq, True))
                y = self.latent_attention(h, p + "mix.", m, freq, *latents[m.get("kv_from", l)])
            x = x + rms(y, eps) * W[p + "norm1b"]
            h, p = rms(x, eps) * W[p + "norm2"], p + "mlp."
            if layer["mlp"]["kind"] == "dense":
                y = torch.nn.functional.gelu(self.lin(h, p + "gate"), approximate="tanh") * self.lin(h, p + "up")
                y = self.lin(y, p + "down")
            else:
                y = self.routed(h, p, layer["mlp"]["router"])
            x = x + rms(y, eps) * W[p[:-4] + "norm2b"]
        return self.lin(rms(x[:, -rows:], eps) * W["final.norm"], "head")

    def latent_attention(self, h, p, m, freq, c, r):
        (B, T), H, d, dv = h.shape[:2], m["heads"], m["dim"], m["vdim"]
        q = self.lin(h, p + "q").reshape(B, T, H, d + m["rot_dim"])
        q = torch.cat([q[..., :d], rotate(q[..., d:], freq, True)], -1)
        k = torch.cat([self.lin(c, p + "uk").reshape(B, T, H, d), r.expand(B, T, H, m["rot_dim"])], -1)
        o = attend(q, k, self.lin(c, p + "uv").reshape(B, T, H, dv), m["scale"], visible_pairs(T, m["mask"]["size"]), self.W[p + "sink"])
        return self.lin(o.reshape(B, T, H * dv), p + "o")

    def conv_attention(self, h, p, m, eps):
        W, (B, T), H, G, d = self.W, h.shape[:2], m["heads"], m["kv_heads"], m["dim"]
        u = torch.cat([self.lin(h, p + "q"), self.lin(h, p + "k")], -1)
        self.leave("mix.conv", last_rows(u, m["conv"] - 1))
        q, k = causal_conv(u, torch.cat([W[p + "q.conv"], W[p + "k.conv"]])).split([H * d, G * d], -1)
        freq = plain_freq(m["rot"]["dims"], m["rot"]["base"])
        v = k.reshape(B, T, G, d)
        q = rotate((rms(q, eps) * W[p + "q.norm"]).reshape(B, T, H, d), freq, True)
        k = rotate((rms(k, eps) * W[p + "k.norm"]).reshape(B, T, G, d), freq, True)
        one = torch.zeros(H, dtype=torch.float64, device=DEVICE)
        o = attend(q, k, v, m["scale"], visible_pairs(T, m["mask"]["size"], m["mask"]["keep_first"]), one)
        o = o * torch.sigmoid(self.lin(h, p + "g"))[..., None]
        return self.lin(o.reshape(B, T, H * d), p + "o")

    def routed(self, h, p, r):
        s = torch.softmax(self.lin(h, p + "router"), -1)
        groups = s.reshape(*s.shape[:-1], r["groups"]["count"], -1)
        kept = torch.zeros_like(groups[..., 0]).scatter(-1, groups.max(-1).values.topk(r["groups"]["keep"], -1).indices, 1.0)
        best = (groups * kept[..., None]).reshape(s.shape).topk(r["top"], -1)
        weight = torch.zeros_like(s).scatter(-1, best.indices, best.values)
        out = torch.zeros_like(h)
        for e in range(r["experts"]):
            f = "%se%d." % (p, e)
            out += weight[..., e:e + 1] * self.lin(silu(self.lin(h, f + "gate")) * self.lin(h, f + "up"), f + "down")
        return out


def exact(case, seed):
    tokens_cost = case["tokens"] if case["kind"] == "prompt" else case["batch"] * case["context"]
    if tokens_cost * case["layers"] > 1_000_000:
        return None  # over 20 seconds
    oracle = Oracle(case, seed)
    vocab = config_of(case).get("vocab_size", 32784)
    ids = token_ids(case, seed, vocab)
    if case["kind"] == "prompt":
        logits, left = [], {}
        for row, rows in zip(ids, wanted(case)):
            oracle.left = {}
            logits.append(oracle.forward(torch.from_numpy(row).long().to(DEVICE)[None], rows)[0])
            for name, per_layer in oracle.left.items():
                left.setdefault(name, []).append(torch.stack(per_layer))
        out = {"logits": torch.cat(logits), **{name: torch.cat(v, 1) for name, v in left.items()}}
    else:
        logits = oracle.forward(torch.from_numpy(ids).long().to(DEVICE), 1)[:, 0]
        out = {"logits": logits, **{name: torch.stack(v) for name, v in oracle.left.items()}}
    return out
