"""Performance cases: forward passes of the model families that the framework serves, on one GPU, through ``Engine`` and ``Transformer``.

A case names a model, the kind of pass and its sizes:

* ``prefill``  ``Engine.prefill`` of new prompts given as host tensors, as ``Engine.generate`` does; the caches are emptied first.
* ``decode``   one token for every sequence over a filled cache: ``Transformer.forward`` captured once and replayed, the way a decode loop runs.
* ``step``     one step of continuous batching: a decode token for each running sequence and a chunk of one more prompt, assembled on the host
               by ``ForwardBatch.build`` and run eagerly, as ``LLM.step`` does.

The models are the shapes of ``models.config.PRESETS`` that the benchmark names (and the hybrid of ``bench.py --design``), cut to some of their layers where
the full model would only repeat them; the vocabulary and every width are the full ones.  Weights are random with the benchmark's deviation of 0.02:
16-bit values; values that e4m3 holds for MXFP8, as a checkpoint in that format has them (with larger embeddings); Q4_K blocks as they come out of a
GGUF file.  Caches in front of a decode step hold random rows of the size that normalised keys and projected values have.
"""
import random
import zlib

import torch

from gemm_b200.models.config import ModelConfig, get_config
from gemm_b200.models.transformer import ForwardBatch
from gemm_b200.models.weights import QBlocks, build_weights
from gemm_b200.ops import attention
from gemm_b200.serve.engine import Engine

PAGE = 128
Q4_K = 12                         # ggml's number of the type

# model -> (configuration, weight format)
MODELS = {
    "qwen3-0.6b": (get_config("qwen3-0.6b"), "bf16"),                                   # all 28 layers
    "qwen3-8b": (get_config("qwen3-8b").with_(n_layers=9), "bf16"),                     # 9 of 36
    "qwen3-30b-a3b": (get_config("qwen3-30b-a3b").with_(n_layers=8), "mxfp8"),          # 8 of 48
    "qwen3-32b": (get_config("qwen3-32b").with_(n_layers=8), "q4_k"),                   # 8 of 64
    # three Delta-Net layers to one of gated attention
    "qwen35-hybrid": (ModelConfig(arch="qwen35", n_layers=8, hidden=4096, n_heads=32, n_kv_heads=8, head_dim=128, ffn=12288, vocab=151936, rope_dim=64,
                                  full_attention_interval=4, ssm_d_conv=4, ssm_n_heads_k=32, ssm_n_heads_v=32, ssm_head_dim=128, attn_output_gate=True), "bf16"),
}

# Ranges of the drawn cases: (model, kind) -> sequences, longest length, most tokens (prefill: in all prompts; decode and step: in all caches).
RANGES = {
    ("qwen3-0.6b", "prefill"): ((1, 4), (8, 2048), 4096),
    ("qwen3-0.6b", "decode"): ((1, 16), (16, 4096), 16384),
    ("qwen3-8b", "prefill"): ((1, 16), (32, 8192), 8192),
    ("qwen3-8b", "decode"): ((1, 64), (32, 16384), 65536),
    ("qwen3-8b", "step"): ((2, 48), (64, 4096), 32768),
    ("qwen3-30b-a3b", "prefill"): ((1, 32), (32, 8192), 16384),
    ("qwen3-30b-a3b", "decode"): ((1, 96), (32, 8192), 131072),
    ("qwen3-32b", "prefill"): ((1, 4), (8, 2048), 2048),
    ("qwen3-32b", "decode"): ((1, 12), (16, 4096), 8192),
    ("qwen35-hybrid", "prefill"): ((1, 8), (32, 4096), 4096),
    ("qwen35-hybrid", "decode"): ((1, 48), (32, 8192), 32768),
}


def _case(model, kind, batch, length, ragged=False, chunk=0, **kw):
    """``batch`` sequences of ``length`` tokens (prompts, or tokens in the cache); ``ragged``: of a quarter of that to all of it; ``chunk``: tokens of the
    prompt beside a step's decoding sequences."""
    return dict(kw, model=model, kind=kind, batch=batch, length=length, ragged=ragged, chunk=chunk)


def listed():
    return [
        # interactive use of a small model: one token at a time, and the first token of a short question
        _case("qwen3-0.6b", "decode", 1, 160, name="small-decode-1"),
        _case("qwen3-0.6b", "prefill", 1, 61, name="small-prefill-1"),
        # the dense benchmark's batch, a few long conversations of different lengths, a batch of prompts, and a server's mixed step
        _case("qwen3-8b", "decode", 32, 1024, name="dense-decode-32"),
        _case("qwen3-8b", "decode", 5, 12001, ragged=True, name="dense-decode-long"),
        _case("qwen3-8b", "prefill", 6, 1999, ragged=True, name="dense-prefill"),
        _case("qwen3-8b", "step", 30, 1000, ragged=True, chunk=709, name="dense-step"),
        # the headline benchmark: 64 sequences behind prompts of 2048 tokens, and one chunk of those prompts
        _case("qwen3-30b-a3b", "decode", 64, 2048, name="moe-decode-64"),
        _case("qwen3-30b-a3b", "prefill", 8, 2048, name="moe-prefill"),
        # quantised weights: one stream (the latency benchmark) and its prompt
        _case("qwen3-32b", "decode", 1, 512, name="q4-decode-1"),
        _case("qwen3-32b", "prefill", 1, 512, name="q4-prefill"),
        # recurrent layers: a batch that decodes, and one longer prompt
        _case("qwen35-hybrid", "decode", 16, 2048, ragged=True, name="hybrid-decode-16"),
        _case("qwen35-hybrid", "prefill", 1, 3001, name="hybrid-prefill"),
    ]


def draw(rng):
    model, kind = rng.choice(sorted(RANGES))
    (b0, b1), (l0, l1), most = RANGES[model, kind]
    log = lambda a, b: round(a * (b / a) ** rng.random())
    batch = log(b0, b1)
    length = min(log(l0, l1), most // batch)
    return _case(model, kind, batch, length, rng.random() < 0.7, log(16, 1500) if kind == "step" else 0)


def _spans(case):
    """(new tokens, cached tokens) of every sequence."""
    r = random.Random("%(batch)d-%(length)d" % case)
    lens = [case["length"]] + [r.randint((case["length"] + 3) // 4, case["length"]) if case["ragged"] else case["length"] for _ in range(case["batch"] - 1)]
    if case["kind"] == "prefill":
        return [(n, 0) for n in lens]
    return [(1, n) for n in lens] + ([(case["chunk"], 0)] if case["chunk"] else [])


# ------------------------------------------------------------------------------------------------ inputs
class _Source:
    """The checkpoint: a tensor by its GGUF name, from the seed and that name alone."""

    def __init__(self, fmt, seed):
        self.fmt, self.seed, self.gen = fmt, seed, torch.Generator(device="cuda")

    def _normal(self, name, shape):
        self.gen.manual_seed(zlib.crc32(("%d/%s" % (self.seed, name)).encode()))
        return torch.randn(tuple(shape), generator=self.gen, device="cuda")

    def has(self, name):
        return True

    def get(self, name, shape):
        x = self._normal(name, shape)
        if name.endswith("norm.weight"):
            return (1 + 0.1 * x).to(torch.bfloat16)
        if name.endswith("ssm_a"):                            # decays from almost none to a few tokens
            return -torch.exp(x - 3)
        if name.endswith("ssm_dt.bias"):
            return x
        if name.endswith("ssm_conv1d.weight"):
            return x * 0.4
        if self.fmt == "mxfp8" and name == "token_embd.weight":
            # with experts the stream is large beside one layer's update, as in a trained model: were it not, rounding would decide near ties of
            # random routers, and two correct passes would pick other experts
            return x.to(torch.bfloat16)
        x *= 0.02
        if self.fmt == "mxfp8" and ("attn_" in name or "_exps" in name):
            return ((x * 4096).clamp_(-448, 448).to(torch.float8_e4m3fn).float() / 4096).to(torch.bfloat16)
        return x.to(torch.bfloat16)

    def get_expert(self, name, e, shape):
        return self.get("%s#%d" % (name, e), shape)

    def get_mat(self, name, shape):
        if self.fmt != "q4_k" or len(shape) == 1 or name == "token_embd.weight":
            return self.get(name, shape)
        return QBlocks(self._q4_blocks(name, shape), Q4_K, shape[1])

    def _q4_blocks(self, name, shape):
        """Q4_K super-blocks ``{f16 d, f16 dmin, 12 bytes of 6-bit scales and minima, 128 bytes of nibbles}``: values of deviation 0.02 around zero."""
        n, k = shape[0], shape[1] // 256
        x = self._normal(name, (n, k, 256))
        q = (x * 2.7 + 8).round_().clamp_(0, 15).to(torch.uint8).view(n, k, 4, 2, 32)
        sc = (x[..., :8] * 8 + 44).clamp_(1, 63).to(torch.uint8)
        d = ((x[..., 8] * 0.1 + 1).clamp_(0.5, 1.5) * (0.02 / 44 / 2.7)).to(torch.float16)
        out = torch.empty(n, k, 144, dtype=torch.uint8, device="cuda")
        out[..., 0:2] = d.view(torch.uint8).view(n, k, 2)
        out[..., 2:4] = (d * 8).view(torch.uint8).view(n, k, 2)       # the minimum of a sub-block is 8 steps: dmin m = 8 d sc
        out[..., 4:8] = out[..., 8:12] = (sc[..., :4] & 63) | (sc[..., 4:] >> 4 << 6)
        out[..., 12:16] = (sc[..., 4:] & 15) * 17
        out[..., 16:] = (q[..., 0, :] | q[..., 1, :] << 4).reshape(n, k, 128)
        return out.view(n, k * 144)

    # what the tensors hold, in 64 bits
    def exact(self, name, shape):
        t = self.get_mat(name, shape)
        if not isinstance(t, QBlocks):
            return t.double()
        b = t.raw.view(shape[0], shape[1] // 256, 144)
        d, dmin = (b[..., i: i + 2].contiguous().view(torch.float16).double() for i in (0, 2))
        lo, hi, mix = b[..., 4:8], b[..., 8:12], b[..., 12:16]
        sc = torch.cat([lo & 63, mix & 15 | lo >> 6 << 4], -1).double() * d
        mn = torch.cat([hi & 63, mix >> 4 | hi >> 6 << 4], -1).double() * dmin
        q = b[..., 16:].view(*b.shape[:2], 4, 32)
        q = torch.stack([q & 15, q >> 4], -2).view(*b.shape[:2], 8, 32).double()
        return (q * sc[..., None] - mn[..., None]).view(shape)


def _history(cfg, seed, li, like):
    """Random content of run ``li``'s cache tensors."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed((seed * 1009 + li) & 0x7FFFFFFF)
    rows = lambda name, shape: torch.randn(shape, generator=gen, device="cuda") * (0.1 if name == "rec" else 1.0)
    return {name: rows(name, shape).to(torch.bfloat16 if name in "kv" else torch.float32) for name, shape in like.items()}


def _cache_shapes(cfg, li, pages, slots):
    if cfg.is_ssm_layer(li):
        return {"conv": (slots, cfg.ssm_d_conv - 1, cfg.ssm_qkv_dim), "rec": (slots, cfg.ssm_n_heads_v, cfg.ssm_head_dim, cfg.ssm_head_dim)}
    return {n: (pages * PAGE, cfg.n_kv_heads, cfg.head_dim) for n in "kv"}


def _layout(spans):
    """First page of every sequence, and the number of pages."""
    first = [0]
    for q, c in spans:
        first.append(first[-1] + -(-(q + c) // PAGE))
    return first[:-1], first[-1]


def _ids(cfg, seed, n):
    gen = torch.Generator().manual_seed(seed)
    return torch.randint(0, cfg.vocab, (n,), generator=gen, dtype=torch.int32)


def prepare(case, seed):
    cfg, fmt = MODELS[case["model"]]
    spans = _spans(case)
    first, pages = _layout(spans)
    weights = build_weights(cfg, _Source(fmt, seed), fmt, "cuda")
    eng = Engine(weights, max_batch=len(spans), max_seq_len=max(q + c for q, c in spans), page_size=PAGE, num_pages=pages)
    q_lens, ctx = [q for q, _ in spans], [c for _, c in spans]
    ids = _ids(cfg, seed, sum(q_lens))
    state = {"engine": eng, "kind": case["kind"]}
    if case["kind"] == "prefill":
        state["prompts"] = list(ids.split(q_lens))
        return state
    table = torch.zeros(len(spans), eng.max_pages_per_seq, dtype=torch.int32)
    for s, (q, c) in enumerate(spans):
        n = -(-(q + c) // PAGE)
        table[s, :n] = torch.arange(first[s], first[s] + n, dtype=torch.int32)
    state["step"] = (q_lens, ctx, ids.tolist(), table, PAGE, eng.hq_local, eng.hkv_local, eng.device)
    with torch.no_grad():
        if case["kind"] == "decode":
            splits = attention.pick_splits(len(spans), eng.hkv_local, max(ctx) + 1)
            fb = ForwardBatch.build(*state["step"], num_splits=splits)
            side = torch.cuda.Stream()                            # first launches outside the capture
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                eng.model.forward(fb)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            state["graph"], state["batch"] = torch.cuda.CUDAGraph(), fb
            with torch.cuda.graph(state["graph"]):
                state["logits"] = eng.model.forward(fb)
        for li in range(cfg.n_layers):
            for name, t in _history(cfg, seed, li, _cache_shapes(cfg, li, pages, len(spans) + 1)).items():
                getattr(eng.kv, name)[li].copy_(t)
    return state


@torch.no_grad()
def run(state):
    eng, kv = state["engine"], state["engine"].kv
    if state["kind"] == "prefill":
        eng.reset()
        out = {"logits": eng.prefill(state["prompts"])}
        out.update(k=[t for t in kv.k if t.numel()], v=[t for t in kv.v if t.numel()])
    elif state["kind"] == "decode":
        state["graph"].replay()
        out = {"logits": state["logits"]}
    else:
        out = {"logits": eng.model.forward(ForwardBatch.build(*state["step"]))}
    if kv.rec is not None:
        out.update(conv=[t for t in kv.conv if t is not None], rec=[t for t in kv.rec if t is not None])
    return out


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    cfg, fmt = MODELS[case["model"]]
    spans = _spans(case)
    tok, h, d = sum(q for q, _ in spans), cfg.hidden, cfg.head_dim
    per = {"bf16": 2.0, "mxfp8": 33 / 32, "q4_k": 144 / 256}[fmt]
    n_ssm = sum(cfg.is_ssm_layer(i) for i in range(cfg.n_layers))
    n_att = cfg.n_layers - n_ssm
    att_w = h * (cfg.q_dim * (2 if cfg.attn_output_gate else 1) + 2 * cfg.kv_dim) + cfg.q_dim * h
    ssm_w = h * (cfg.ssm_qkv_dim + cfg.ssm_d_inner) + cfg.ssm_d_inner * h if n_ssm else 0
    if cfg.is_moe:
        one = 3 * h * cfg.expert_ffn
        hit = cfg.n_experts * (1 - (1 - cfg.n_experts_used / cfg.n_experts) ** tok)
        ffn_read, ffn_used = hit * one, cfg.n_experts_used * one
    else:
        ffn_read = ffn_used = 3 * h * cfg.ffn
    head = cfg.vocab * h
    rows = len(spans)
    kv_rows = sum(c + q for q, c in spans)
    state = (cfg.ssm_n_heads_v * cfg.ssm_head_dim ** 2 + (cfg.ssm_d_conv - 1) * cfg.ssm_qkv_dim) * 4 if n_ssm else 0
    b = (n_att * att_w + n_ssm * ssm_w + cfg.n_layers * ffn_read) * per + head * (per if fmt == "q4_k" else 2.0)
    b += n_att * kv_rows * 2 * cfg.kv_dim * 2 + n_ssm * rows * 2 * state + tok * h * 2 + rows * cfg.vocab * 4
    f = 2.0 * tok * (n_att * att_w + n_ssm * ssm_w + cfg.n_layers * ffn_used) + 2.0 * rows * head
    f += n_att * 4.0 * cfg.q_dim * sum(q * c + q * (q + 1) / 2 for q, c in spans) + n_ssm * tok * 6.0 * cfg.ssm_n_heads_v * cfg.ssm_head_dim ** 2
    return {"bytes": b, "flops": f}


def tolerance(case):
    # Every product rounds its operands and its result to 16 bits, MXFP8 and Q4_K their activations to 8: over these depths the passes measure 0.01 to
    # 0.03 from the same in 64 bits (16-bit weights; 0.03 to 0.06 the others), and two of them can be that far from each other.  A single value: six
    # deviations of that; where a router's near tie falls the other way, a row moves by an expert's share.
    return {"rel": 0.03, "max": 0.9 if MODELS[case["model"]][0].is_moe else 0.3}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, theta, rd):
    half = rd // 2
    ang = pos[:, None] * theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device="cuda") / rd)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:rd]
    return torch.cat([a * cos - b * sin, a * sin + b * cos, x[..., rd:]], -1)


class _Exact:
    def __init__(self, case, seed):
        self.cfg, fmt = MODELS[case["model"]]
        self.src, self.spans, self.seed = _Source(fmt, seed), _spans(case), seed
        self.first, self.pages = _layout(self.spans)
        self.fresh = case["kind"] == "prefill"
        self.caches = {n: [] for n in ("k", "v", "conv", "rec")}

    def w(self, name, *shape):
        return self.src.exact(name, shape)

    def cache(self, li):
        shapes = _cache_shapes(self.cfg, li, self.pages, len(self.spans) + 1)
        got = {n: torch.zeros(s, device="cuda", dtype=torch.float64) for n, s in shapes.items()} if self.fresh else \
            {n: t.double() for n, t in _history(self.cfg, self.seed, li, shapes).items()}
        for n, t in got.items():
            self.caches[n].append(t)
        return got

    def attention(self, li, pre, x):
        cfg, h, d, hq, hkv = self.cfg, self.cfg.hidden, self.cfg.head_dim, self.cfg.n_heads, self.cfg.n_kv_heads
        q = x @ self.w(pre + "attn_q.weight", cfg.q_dim * (2 if cfg.attn_output_gate else 1), h).t()
        gate = None
        if cfg.attn_output_gate:
            q, gate = q.view(-1, hq, 2, d).unbind(2)
        k, v = ((x @ self.w(pre + n, cfg.kv_dim, h).t()).view(-1, hkv, d) for n in ("attn_k.weight", "attn_v.weight"))
        pos = torch.cat([torch.arange(c, c + n, device="cuda", dtype=torch.float64) for n, c in self.spans])
        rd = cfg.rope_dim or d
        q = _rotate(_rms(q.reshape(-1, hq, d), self.w(pre + "attn_q_norm.weight", d), cfg.rms_eps), pos, cfg.rope_theta, rd)
        k = _rotate(_rms(k, self.w(pre + "attn_k_norm.weight", d), cfg.rms_eps), pos, cfg.rope_theta, rd)
        cache, out, t = self.cache(li), torch.empty_like(q), 0
        for page, (n, c) in zip(self.first, self.spans):
            at = page * PAGE
            for name, rows in (("k", k), ("v", v)):
                cache[name][at + c: at + c + n] = rows[t: t + n]
            ks, vs = (cache[name][at: at + c + n].transpose(0, 1) for name in "kv")
            for i in range(0, n, 512):                            # some queries at a time
                m = min(512, n - i)
                qs = q[t + i: t + i + m].view(m, hkv, -1, d).permute(1, 2, 0, 3).reshape(hkv, -1, d)
                s = (qs @ ks.transpose(1, 2)).view(hkv, -1, m, c + n) * d ** -0.5
                ahead = torch.arange(c + n, device="cuda") > torch.arange(c + i, c + i + m, device="cuda")[:, None]
                p = torch.softmax(s.masked_fill_(ahead, float("-inf")), -1).view(hkv, -1, c + n)
                out[t + i: t + i + m] = (p @ vs).view(hkv, -1, m, d).permute(2, 0, 1, 3).reshape(m, hq, d)
            t += n
        if gate is not None:
            out = out * torch.sigmoid(gate)
        return out.reshape(-1, cfg.q_dim) @ self.w(pre + "attn_output.weight", h, cfg.q_dim).t()

    def delta_net(self, li, pre, x):
        cfg, h = self.cfg, self.cfg.hidden
        ng, hv, ds, taps, qd = cfg.ssm_n_heads_k, cfg.ssm_n_heads_v, cfg.ssm_head_dim, cfg.ssm_d_conv, cfg.ssm_qkv_dim
        rows = x @ self.w(pre + "attn_qkv.weight", qd, h).t()
        z = (x @ self.w(pre + "attn_gate.weight", cfg.ssm_d_inner, h).t()).view(-1, hv, ds)
        rate = torch.nn.functional.softplus(x @ self.w(pre + "ssm_alpha.weight", hv, h).t() + self.src.get(pre + "ssm_dt.bias", (hv,)).double())
        decay = torch.exp(rate * self.src.get(pre + "ssm_a", (hv,)).double())
        beta = torch.sigmoid(x @ self.w(pre + "ssm_beta.weight", hv, h).t())
        cw, cache, t, out = self.w(pre + "ssm_conv1d.weight", qd, taps), self.cache(li), 0, []
        for s, (n, _) in enumerate(self.spans):
            pad = torch.cat([cache["conv"][s], rows[t: t + n]])
            cache["conv"][s] = pad[n:]
            c = torch.nn.functional.silu(sum(pad[i: i + n] * cw[:, i] for i in range(taps)))
            q, k, v = c[:, : ng * ds].view(n, ng, ds), c[:, ng * ds: 2 * ng * ds].view(n, ng, ds), c[:, 2 * ng * ds:].view(n, hv, ds)
            q, k = (y * torch.rsqrt(y.pow(2).sum(-1, keepdim=True) + cfg.rms_eps) for y in (q * 1.0, k))
            which = torch.arange(hv, device="cuda") % ng
            q, k, state = q[:, which, :, None] * ds ** -0.5, k[:, which, :, None], cache["rec"][s].clone()
            for i in range(n):
                state *= decay[t + i, :, None, None]
                new = (v[i][..., None] - state @ k[i]) * beta[t + i, :, None, None]
                state += new @ k[i].transpose(1, 2)
                out.append((state @ q[i])[..., 0])
            cache["rec"][s] = state
            t += n
        o = _rms(torch.stack(out), self.w(pre + "ssm_norm.weight", ds), cfg.rms_eps) * torch.nn.functional.silu(z)
        return o.reshape(-1, hv * ds) @ self.w(pre + "ssm_out.weight", h, hv * ds).t()

    def ffn(self, pre, x):
        cfg, h = self.cfg, self.cfg.hidden
        silu = torch.nn.functional.silu
        if not cfg.is_moe:
            g, u = (x @ self.w(pre + n, cfg.ffn, h).t() for n in ("ffn_gate.weight", "ffn_up.weight"))
            return (silu(g) * u) @ self.w(pre + "ffn_down.weight", h, cfg.ffn).t()
        p, chosen = torch.softmax(x @ self.w(pre + "ffn_gate_inp.weight", cfg.n_experts, h).t(), -1).topk(cfg.n_experts_used, -1)
        p = p / p.sum(-1, keepdim=True)
        y = torch.zeros_like(x)
        for e in range(cfg.n_experts):
            tok, slot = (chosen == e).nonzero(as_tuple=True)
            g, u = (x[tok] @ self.src.get_expert(pre + n, e, (cfg.expert_ffn, h)).double().t() for n in ("ffn_gate_exps.weight", "ffn_up_exps.weight"))
            y.index_add_(0, tok, (silu(g) * u) @ self.src.get_expert(pre + "ffn_down_exps.weight", e, (h, cfg.expert_ffn)).double().t() * p[tok, slot, None])
        return y

    def logits(self):
        cfg, h = self.cfg, self.cfg.hidden
        ids = _ids(cfg, self.seed, sum(q for q, _ in self.spans)).long().cuda()
        x = self.src.get("token_embd.weight", (cfg.vocab, h))[ids].double()
        for li in range(cfg.n_layers):
            pre = "blk.%d." % li
            mix = self.delta_net if cfg.is_ssm_layer(li) else self.attention
            x = x + mix(li, pre, _rms(x, self.w(pre + "attn_norm.weight", h), cfg.rms_eps))
            x = x + self.ffn(pre, _rms(x, self.w(pre + "ffn_norm.weight", h), cfg.rms_eps))
        last = torch.tensor([q for q, _ in self.spans], device="cuda").cumsum(0) - 1
        x = _rms(x[last], self.w("output_norm.weight", h), cfg.rms_eps)
        return x @ self.w("token_embd.weight" if cfg.tie_embeddings else "output.weight", cfg.vocab, h).t()


@torch.no_grad()
def exact(case, seed):
    e = _Exact(case, seed)
    if any(e.cfg.is_ssm_layer(i) for i in range(e.cfg.n_layers)) and sum(q for q, _ in e.spans) > 3500:
        return None                                               # token by token: too long
    out = {"logits": e.logits()}
    if case["kind"] == "prefill":
        out.update(k=e.caches["k"], v=e.caches["v"])
    if e.caches["rec"]:
        out.update(conv=e.caches["conv"], rec=e.caches["rec"])
    return out
