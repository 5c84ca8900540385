"""The serving steps whose speed counts: decode and prefill of quantized decoders through ``GpuExecutor``.

A case is one step of a served model: every request of the batch brings its new tokens (one while it decodes, a portion of
its prompt while it is prefilled), the step runs the embedding, all layers, the output head and the sampler, and the sampled
ids are read back.  The sizes are those of the named configurations; a model is cut to its first layers and its vocabulary in
the same proportion, so that the layers and the output head keep their shares of a step.  The runner has the page pool, the
prefill budget of 8192 tokens and the decode graphs of a server.

A request that already has a context got it as in a server: its prompt was prefilled, and its pages are its own copies
(``shared`` tokens of them are one physical prefix, as the prefix cache hands out).
"""
from __future__ import annotations

import math
from dataclasses import replace

import torch

from cubic_serve_b200.executor.gpu_executor import GpuExecutor, Segment
from cubic_serve_b200.models.config import NAMED_CONFIGS, QuantSpec
from cubic_serve_b200.models.decoder import DecoderRunner, DecoderWeights, GdnWeights, LayerWeights
from cubic_serve_b200.models.moe import MoeLayer, stack_experts
from cubic_serve_b200.ops import wq_pack

PAGE = 16
BUDGET = 8192                    # prefill tokens of a step
PROMPTS = 2                      # distinct prompts behind the contexts of a batch

#: model -> (configuration, layers kept, vocabulary kept, weight format, bits of K and V)
MODELS = {
    "dense-8b": ("dense-8b", 12, 50688, QuantSpec("cubic", 4, 128), (8, 8)),
    "dense-8b-q4k": ("dense-8b", 12, 50688, QuantSpec("gguf", 4, 32), (8, 8)),
    "moe-30b-a3b": ("moe-30b-a3b", 6, 18944, QuantSpec("nvfp4", 4, 16), (4, 8)),
    "moe-235b-a22b": ("moe-235b-a22b", 2, 3200, QuantSpec("fp8_block", 8, 128), (6, 6)),
    "hybrid-8b": ("hybrid-8b", 8, 33792, QuantSpec("cubic", 4, 128), (8, 8)),
}


def _case(model, phase, requests, context, new, ragged=False, shared=0, name=None):
    c = {"model": model, "phase": phase, "requests": requests, "context": context, "new": new, "ragged": ragged, "shared": shared}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one user waits for every token: weights stream through a single row
        _case("dense-8b", "decode", 1, 700, 1, name="dense-decode-1"),
        # a handful of users at different points of their conversations, one of a bucket of eight rows stays empty
        _case("dense-8b", "decode", 7, 2100, 1, ragged=True, name="dense-decode-7-ragged"),
        # a server at part load
        _case("dense-8b", "decode", 48, 1500, 1, ragged=True, name="dense-decode-48-ragged"),
        # the headline workload at its mean context: 1024 input tokens, half of 512 output tokens
        _case("dense-8b", "decode", 256, 1280, 1, name="dense-decode-256"),
        # its prefill: prompts of 1024 tokens fill the step's budget
        _case("dense-8b", "prefill", 8, 0, 1024, name="dense-prefill-8x1024"),
        # one short question arrives on an idle server
        _case("dense-8b", "prefill", 1, 0, 331, name="dense-prefill-331"),
        # k-quant weights behind a prefix cache: eight requests decode after a common prefix of 2048 tokens
        _case("dense-8b-q4k", "decode", 8, 2432, 1, shared=2048, name="q4k-decode-8-prefix"),
        # ... and the 256 tokens of their own that they bring when they arrive
        _case("dense-8b-q4k", "prefill", 4, 2048, 256, shared=2048, name="q4k-extend-4x256-prefix"),
        # mixture of experts with 4-bit weights: decode of a busy server, prefill of two prompts
        _case("moe-30b-a3b", "decode", 96, 2176, 1, ragged=True, name="moe-decode-96-ragged"),
        _case("moe-30b-a3b", "prefill", 2, 0, 2048, name="moe-prefill-2x2048"),
        # large mixture of experts with block-scaled 8-bit weights and 6-bit cache, long contexts
        _case("moe-235b-a22b", "decode", 128, 4224, 1, name="moe-fp8-decode-128-long"),
        # recurrent layers: prompts of uneven length
        _case("hybrid-8b", "prefill", 5, 0, 1000, ragged=True, name="hybrid-prefill-5-ragged"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["dense-8b", "dense-8b", "dense-8b", "dense-8b-q4k", "moe-30b-a3b", "moe-30b-a3b", "moe-235b-a22b", "hybrid-8b"])
    phase = "prefill" if model == "hybrid-8b" else rng.choice(["decode", "decode", "prefill", "extend"])
    shared = 0
    if phase == "decode":
        most = {"dense-8b": 256, "dense-8b-q4k": 64, "moe-30b-a3b": 256, "moe-235b-a22b": 128}[model]
        requests = log(1, most)
        context = log(128, 4200 if model == "moe-235b-a22b" else 2400 if requests < 64 else 1280)
        new = 1
        if model == "dense-8b-q4k":
            shared = context // 2 // PAGE * PAGE
    else:
        requests = log(1, 8)
        most = {"moe-30b-a3b": 4096, "moe-235b-a22b": 2048, "hybrid-8b": 5000}.get(model, BUDGET if phase == "prefill" else 4096)
        new = log(17, min(2048, most // requests))
        context = 0
        if phase == "extend":
            context = log(64, 2048) // PAGE * PAGE
            shared = context
    return _case(model, "prefill" if phase == "extend" else phase, requests, context, new, rng.random() < 0.6, shared)


# ------------------------------------------------------------------------------------------------- sizes
def _config(case):
    name, layers, vocab, quant, _ = MODELS[case["model"]]
    return replace(NAMED_CONFIGS[name](), num_layers=layers, vocab_size=vocab, quant=quant)


def _lengths(case):
    """(tokens before the step, tokens of the step) of every request."""
    def spread(n, i, least):
        return max(least, int(n * (1 - 0.75 * ((i * 0.6180339887) % 1.0)))) if case["ragged"] else n

    out = []
    for i in range(case["requests"]):
        ctx = case["context"] if case["phase"] == "prefill" else max(case["shared"], spread(case["context"], i, 1))
        out.append((ctx, 1 if case["phase"] == "decode" else spread(case["new"], i, 1)))
    return out


def _generator(seed, *where):
    g = torch.Generator(device="cuda")
    n = seed
    for w in where:
        n = (n * 1000003 + w + 12345) % (1 << 40)
    return g.manual_seed(n)


def _tokens(case, cfg, seed):
    """The prompts behind the contexts and the new tokens of every request."""
    g = _generator(seed, 1)
    most = max(c for c, _ in _lengths(case))
    prompts = torch.randint(0, cfg.vocab_size, (PROMPTS, max(most, 1)), device="cuda", generator=g)
    if case["shared"]:
        prompts[:, :case["shared"]] = prompts[:1, :case["shared"]]
    new = [torch.randint(0, cfg.vocab_size, (n,), device="cuda", generator=g) for _, n in _lengths(case)]
    return prompts, new


# ------------------------------------------------------------------------------------------------- weights
STD = 0.02


def _raw(cfg, g, n, k, std=STD):
    """A random matrix of standard deviation ``std`` as its checkpoint stores it."""
    m = cfg.quant.method
    if m == "cubic":
        codes = (torch.randn(n, k, device="cuda", generator=g) * 2.6).round_().clamp_(-7, 7).to(torch.int8)
        u = torch.rand(3, n, k // 128, device="cuda", generator=g)
        return {"codes": codes, "scale": std * 7 / 2.6 * (0.8 + 0.4 * u[0]), "a": (0.9 + 0.2 * u[1]).half(), "b": (0.2 * u[2] - 0.1).half()}
    if m == "gguf":
        codes = (torch.randn(n, k, device="cuda", generator=g) * 2.6 + 8).round_().clamp_(0, 15).to(torch.uint8)
        u = torch.rand(2, n, k // 32, device="cuda", generator=g)
        scale = (std / 2.6 * (0.8 + 0.4 * u[0])).bfloat16().float()
        return {"codes": codes, "scale": scale, "offset": (std * (0.1 * u[1] - 0.05)).bfloat16().float() - 8 * scale}
    if m == "nvfp4":
        packed = torch.randint(0, 256, (n, k // 2), device="cuda", generator=g, dtype=torch.uint8)
        scale = (32 + 64 * torch.rand(n, k // 16, device="cuda", generator=g)).to(torch.float8_e4m3fn)
        return {"packed": packed, "scale": scale, "global": std / 2.9 / 64}
    w = (torch.randn(n, k, device="cuda", generator=g) * 100).clamp_(-448, 448).to(torch.float8_e4m3fn)
    return {"weight": w, "scale": std / 100 * (0.8 + 0.4 * torch.rand(-(-n // 128), -(-k // 128), device="cuda", generator=g))}


def _pack(cfg, r):
    m = cfg.quant.method
    if m == "cubic":
        return wq_pack.pack_cubic4(r["codes"], r["scale"], r["a"], r["b"], 128)
    if m == "gguf":
        return wq_pack.pack_affine4(r["codes"], r["scale"], r["offset"], 32)
    if m == "nvfp4":
        return wq_pack.pack_nvfp4(r["packed"], r["scale"], r["global"])
    return wq_pack.pack_fp8_block(r["weight"], r["scale"])


def _rows(cfg, r, lo, hi):
    return {k: v if isinstance(v, float) else v[lo // 128:hi // 128] if cfg.quant.method == "fp8_block" and k == "scale" else v[lo:hi] for k, v in r.items()}


def _values(cfg, r):
    """The matrix in 64 bits."""
    m = cfg.quant.method
    if m == "cubic":
        c = r["codes"].double()
        n, k = c.shape
        t = (c.abs() / 7).view(n, -1, 128)
        s, a, b = (r[x].double().unsqueeze(-1) for x in ("scale", "a", "b"))
        return (s * t * (a + t * (b + t * (1 - a - b)))).view(n, k) * c.sign()
    if m == "gguf":
        n, k = r["codes"].shape
        return (r["codes"].double().view(n, -1, 32) * r["scale"].double().unsqueeze(-1) + r["offset"].double().unsqueeze(-1)).view(n, k)
    if m == "nvfp4":
        p = r["packed"].long()
        code = torch.stack([p & 15, p >> 4], -1).view(p.shape[0], -1)
        level = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], device=p.device, dtype=torch.float64)
        return level[code] * r["scale"].double().repeat_interleave(16, 1) * r["global"]
    n, k = r["weight"].shape
    s = r["scale"].double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    return r["weight"].double() * s


def _bf16(g, n, k, std):
    return (torch.randn(n, k, device="cuda", generator=g) * std).bfloat16()


class _Layer:
    """The matrices of one layer, made when asked for."""

    def __init__(self, cfg, seed, i):
        self.cfg, self.seed, self.i = cfg, seed, i

    def raw(self, part, n, k, std=STD):
        return _raw(self.cfg, _generator(self.seed, 2, self.i, part), n, k, std)

    def added(self, part, n, k):
        """A matrix whose results join the residual stream: smaller with the depth of the whole model, as networks start out."""
        return self.raw(part, n, k, STD * (2 * NAMED_CONFIGS[self.cfg.name]().num_layers) ** -0.5)

    def small(self, part, *shape):
        return torch.randn(*shape, device="cuda", generator=_generator(self.seed, 3, self.i, part))

    def qkv(self):
        c = self.cfg
        return self.raw(0, c.q_size + 2 * c.kv_size, c.hidden_size)

    def o(self):
        return self.added(1, self.cfg.hidden_size, self.cfg.q_size)

    def gate(self):
        return self.raw(2, self.cfg.q_size, self.cfg.hidden_size)

    def gate_up(self):
        c = self.cfg
        return self.raw(3, 2 * (c.intermediate_size or c.num_experts * c.moe_intermediate_size), c.hidden_size)

    def down(self):
        c = self.cfg
        if c.is_moe:
            return self.added(4, c.num_experts * c.hidden_size, c.moe_intermediate_size)
        return self.added(4, c.hidden_size, c.intermediate_size)

    def router(self):
        return _bf16(_generator(self.seed, 4, self.i), self.cfg.num_experts, self.cfg.hidden_size, STD)

    def gdn(self):
        c = self.cfg
        hk, hv, H = c.gdn_k_heads, c.gdn_v_heads, c.hidden_size
        return {"in_proj": self.raw(5, (2 * hk + 2 * hv) * 128, H), "in_ba": self.small(6, 2 * hv, H).mul_(STD).bfloat16(),
                "conv": self.small(7, (2 * hk + hv) * 128, 4) * 0.3, "a_log": self.small(8, hv) * 0.5, "dt_bias": self.small(9, hv) * 0.5,
                "out": self.added(10, H, hv * 128)}


def _embedding(cfg, seed):
    e = torch.randn(cfg.vocab_size, cfg.hidden_size, device="cuda", generator=_generator(seed, 5))
    if cfg.is_moe:
        # a trained router knows its tokens: in every layer a token leans towards experts of its own
        for i in range(cfg.num_layers):
            r = _Layer(cfg, seed, i).router().float()
            pick = torch.rand(cfg.vocab_size, cfg.num_experts, device="cuda", generator=_generator(seed, 6, i)).topk(cfg.experts_per_token, -1).indices
            lean = torch.zeros(cfg.vocab_size, cfg.num_experts, device="cuda").scatter_(1, pick, 7.0 * (64 / cfg.hidden_size ** 0.5))
            e += lean @ (r / r.norm(dim=1, keepdim=True))
    return e.bfloat16()


def _head(cfg, seed):
    return _bf16(_generator(seed, 7), cfg.vocab_size, cfg.hidden_size, STD)


def _weights(cfg, seed):
    H, one = cfg.hidden_size, 0.0 if cfg.zero_centered_norm else 1.0

    def norm():
        return torch.full((H,), one, device="cuda", dtype=torch.bfloat16)

    layers = []
    for i in range(cfg.num_layers):
        l = _Layer(cfg, seed, i)
        w = LayerWeights(ln1=norm(), ln2=norm())
        if cfg.layer_is_gdn(i):
            r = l.gdn()
            w.gdn = GdnWeights(in_proj=_pack(cfg, r["in_proj"]), in_ba=wq_pack.pack_bf16(r["in_ba"]), conv_w=r["conv"], a_log=r["a_log"],
                               dt_bias=r["dt_bias"], norm_w=torch.ones(128, device="cuda"), out=_pack(cfg, r["out"]), hk=cfg.gdn_k_heads, hv=cfg.gdn_v_heads)
        else:
            w.qkv, w.o = _pack(cfg, l.qkv()), _pack(cfg, l.o())
            if cfg.attn_output_gate:
                w.attn_gate = _pack(cfg, l.gate())
            if cfg.qk_norm:
                w.q_norm = w.k_norm = torch.ones(128, device="cuda", dtype=torch.bfloat16)
        if cfg.is_moe:
            E, I = cfg.num_experts, cfg.moe_intermediate_size
            gu, dn = l.gate_up(), l.down()
            gu, gcs, gms = stack_experts([_pack(cfg, _rows(cfg, gu, e * 2 * I, (e + 1) * 2 * I)) for e in range(E)])
            dn, dcs, dms = stack_experts([_pack(cfg, _rows(cfg, dn, e * H, (e + 1) * H)) for e in range(E)])
            w.moe = MoeLayer(wq_pack.pack_bf16(l.router()), gu, dn, (gcs, gms, dcs, dms), E, cfg.experts_per_token, 0, E, cfg.norm_topk_prob)
        else:
            w.gate_up, w.down = _pack(cfg, l.gate_up()), _pack(cfg, l.down())
        layers.append(w)
    return DecoderWeights(embed=_embedding(cfg, seed), layers=layers, final_norm=norm(), lm_head=wq_pack.pack_bf16(_head(cfg, seed)))


# ------------------------------------------------------------------------------------------------- the framework
def prepare(case, seed):
    cfg = _config(case)
    k_bits, v_bits = MODELS[case["model"]][4]
    lengths = _lengths(case)
    prompts, new = _tokens(case, cfg, seed)
    most = max(c for c, _ in lengths)
    behind = -(-most // PAGE) if most else 0
    rows = 1 << (max(len(lengths), PROMPTS) - 1).bit_length()
    shared = case["shared"] // PAGE
    own = [-(-(c + n) // PAGE) - shared for c, n in lengths]
    pages = PROMPTS * behind + sum(own) + 1
    runner = DecoderRunner(cfg, _weights(cfg, seed), num_pages=pages, max_tokens=BUDGET, k_bits=k_bits, v_bits=v_bits, max_requests=rows)
    ex = GpuExecutor(runner, max_rows=rows, max_prefill_tokens=BUDGET, max_model_len=max(c + n for c, n in lengths) + PAGE)
    # the prompts, in portions that fit a step
    uid = 0
    for b in range(PROMPTS if most else 0):
        ids, first = prompts[b].cpu().numpy(), list(range(b * behind, (b + 1) * behind))
        for at in range(0, most, BUDGET):
            ex.execute([Segment(b, ids[at:at + BUDGET], at, first, uid=uid)])
        uid += 1
    segs, nxt, copies = [], PROMPTS * behind, []
    for i, ((c, n), ids) in enumerate(zip(lengths, new)):
        mine = list(range(nxt, nxt + own[i]))
        nxt += own[i]
        source = list(range(i % PROMPTS * behind, i % PROMPTS * behind + behind))
        copies += list(zip(source[shared:], mine))[:max(0, -(-c // PAGE) - shared)]
        table = list(range(shared)) + mine
        segs.append(Segment(i, ids.cpu().numpy() if n > 1 else [int(ids[0])], c, table, uid=uid + i))
    ex.copy_pages(copies)
    torch.cuda.synchronize()
    if case["phase"] == "decode":
        ex.capture_decode_graphs([1 << (len(segs) - 1).bit_length()])
    return {"executor": ex, "segments": segs}


def run(state):
    ex, segs = state["executor"], state["segments"]
    ex.execute(segs)
    return {"logits": ex.logits[:len(segs)]}


def work(case):
    cfg = _config(case)
    k_bits, v_bits = MODELS[case["model"]][4]
    H, D = cfg.hidden_size, 128
    lengths = _lengths(case)
    tokens = sum(n for _, n in lengths)
    per = {"cubic": 0.5 + 8 / 128, "gguf": 0.5 + 4 / 32, "nvfp4": 0.5 + 1 / 16, "fp8_block": 1.0}[cfg.quant.method]     # bytes of a weight
    byts, flops = 2 * H * cfg.vocab_size + 2 * len(lengths) * cfg.vocab_size + 2 * H * tokens, 2 * H * cfg.vocab_size * len(lengths)
    for i in range(cfg.num_layers):
        if cfg.layer_is_gdn(i):
            n = H * (2 * cfg.gdn_k_heads + 3 * cfg.gdn_v_heads) * D
            flops += tokens * cfg.gdn_v_heads * 7 * D * D
            byts += 2 * len(lengths) * cfg.gdn_v_heads * D * D * 4
        else:
            n = H * (2 * cfg.q_size + 2 * cfg.kv_size + (cfg.q_size if cfg.attn_output_gate else 0))
            seen = sum(m * c + m * (m + 1) // 2 for c, m in lengths)
            flops += 4 * seen * cfg.num_q_heads * D
            entry = cfg.num_kv_heads * (D * (k_bits + v_bits) / 8 + 2 * (D // 32) * 4)
            held = sum(c + m for c, m in lengths) - (len(lengths) - 1) * case["shared"]
            byts += (held + tokens) * entry
        if cfg.is_moe:
            each, top = 3 * H * cfg.moe_intermediate_size, cfg.experts_per_token
            flops += 2 * tokens * (each * top + H * cfg.num_experts)
            byts += 2 * H * cfg.num_experts + per * each * cfg.num_experts * (1 - (1 - top / cfg.num_experts) ** tokens)
        else:
            n += 3 * H * cfg.intermediate_size
        flops += 2 * tokens * n
        byts += per * n
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    # bf16 activations through all layers, and codes of the cache (and of 8-bit activations) that turn over: against ``exact``
    # the paths are 0.005 (two layers) to 0.011 (twelve) off, and about 0.7 of that against other orders of the same sums
    return {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------------------- in 64 bits
def _norm(x, eps=1e-6):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()


def _cached(x, bits):
    """What the cache gives back: codes with one scale for 32 channels of a head."""
    top = float((1 << (bits - 1)) - 1)
    g = x.view(*x.shape[:-1], -1, 32)
    s = g.abs().amax(-1, keepdim=True).clamp_min(1e-30) / top
    return ((g / s).round().clamp(-top, top) * s).view(x.shape)


def _rotate(x, pos, theta, width):
    half = width // 2
    f = theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    a = pos.double()[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    p, q, rest = x[..., :half], x[..., half:width], x[..., width:]
    return torch.cat([p * c - q * s, q * c + p * s, rest], -1)


def _attend(q, k, v, first):
    """Causal attention of one request: row ``r`` sees the first ``first + r + 1`` keys."""
    n, hq, d = q.shape
    g = hq // k.shape[1]
    out = torch.empty_like(q)
    for h in range(k.shape[1]):
        for r in range(0, n, 1024):
            z = torch.einsum("rgd,sd->rgs", q[r:r + 1024, h * g:(h + 1) * g], k[:, h]) * d ** -0.5
            sees = torch.arange(r, min(n, r + 1024), device=q.device)[:, None] + first + 1
            z.masked_fill_((torch.arange(k.shape[0], device=q.device)[None] >= sees)[:, None], -math.inf)
            out[r:r + 1024, h * g:(h + 1) * g] = torch.einsum("rgs,sd->rgd", z.softmax(-1), v[:, h])
    return out


def _delta(cfg, r, x, starts):
    """Gated delta rule over the rows of every request, in the order of its tokens."""
    hk, hv, d = cfg.gdn_k_heads, cfg.gdn_v_heads, 128
    proj, ba = x @ _values(cfg, r["in_proj"]).t(), x @ r["in_ba"].double().t()
    c, n = (2 * hk + hv) * d, len(starts) - 1
    conv = r["conv"].double()
    longest = max(starts[i + 1] - starts[i] for i in range(n))

    def padded(t):
        return torch.stack([torch.nn.functional.pad(t[starts[i]:starts[i + 1]], (0, 0, 0, longest - (starts[i + 1] - starts[i]))) for i in range(n)], 1)

    u = padded(proj[:, :c])
    past = torch.cat([u.new_zeros(3, n, c), u])
    mix = torch.nn.functional.silu(sum(conv[:, j] * past[j:j + longest] for j in range(4)))
    q, k, v = (t.view(longest, n, -1, d) for t in mix.split([hk * d, hk * d, hv * d], -1))
    q, k = ((t * (t.square().sum(-1, keepdim=True) + 1e-6).rsqrt()).repeat_interleave(hv // hk, 2) for t in (q, k))
    b, a = padded(ba).split(hv, -1)
    beta, decay = b.sigmoid(), (-r["a_log"].double().exp() * torch.nn.functional.softplus(a + r["dt_bias"].double())).exp()
    S, out = x.new_zeros(n, hv, d, d), torch.empty_like(v)
    for t in range(longest):
        S *= decay[t, :, :, None, None]
        step = (v[t] - (S @ k[t].unsqueeze(-1)).squeeze(-1)) * beta[t].unsqueeze(-1)
        S += step.unsqueeze(-1) * k[t].unsqueeze(-2)
        out[t] = (S @ q[t].unsqueeze(-1)).squeeze(-1) * d ** -0.5
    flat = torch.cat([out[:starts[i + 1] - starts[i], i] for i in range(n)])
    z = proj[:, c:].view(-1, hv, d)
    return (_norm(flat) * torch.nn.functional.silu(z)).view(-1, hv * d) @ _values(cfg, r["out"]).t()


def _as_fp8(cfg, x):
    """8-bit weights are multiplied with activations of 8 bits, one scale for a token."""
    if cfg.quant.method != "fp8_block":
        return x
    s = (x.abs().amax(-1, keepdim=True) / 448).clamp_min(1 / (448 * 512))
    return (x / s).float().to(torch.float8_e4m3fn).double() * s


def _experts(cfg, l, x):
    E, I, H = cfg.num_experts, cfg.moe_intermediate_size, cfg.hidden_size
    z, pick = (x @ l.router().double().t()).topk(cfg.experts_per_token, -1)
    share = z.softmax(-1)
    gu, dn, xq, out = l.gate_up(), l.down(), _as_fp8(cfg, x), torch.zeros_like(x)
    for e in range(E):
        row, at = (pick == e).nonzero(as_tuple=True)
        if row.numel():
            g, u = (xq[row] @ _values(cfg, _rows(cfg, gu, e * 2 * I, (e + 1) * 2 * I)).t()).chunk(2, -1)
            y = _as_fp8(cfg, torch.nn.functional.silu(g) * u) @ _values(cfg, _rows(cfg, dn, e * H, (e + 1) * H)).t()
            out.index_add_(0, row, y * share[row, at].unsqueeze(-1))
    return out


@torch.no_grad()
def exact(case, seed):
    cfg = _config(case)
    bits = MODELS[case["model"]][4]
    lengths = _lengths(case)
    prompts, new = _tokens(case, cfg, seed)
    most = max(c for c, _ in lengths)
    base = PROMPTS * most
    starts = [base]
    for _, n in lengths:
        starts.append(starts[-1] + n)
    ids = torch.cat([prompts[:, :most].reshape(-1), *new])
    pos = torch.cat([torch.arange(most, device="cuda")] * PROMPTS + [torch.arange(c, c + n, device="cuda") for c, n in lengths])
    h = _embedding(cfg, seed)[ids].double()
    Hq, Hk = cfg.num_q_heads, cfg.num_kv_heads
    for i in range(cfg.num_layers):
        l, x = _Layer(cfg, seed, i), _norm(h)
        if cfg.layer_is_gdn(i):
            h += _delta(cfg, l.gdn(), x, starts)
        else:
            x8 = _as_fp8(cfg, x)
            q, k, v = (t.unflatten(-1, (-1, 128)) for t in (x8 @ _values(cfg, l.qkv()).t()).split([cfg.q_size, cfg.kv_size, cfg.kv_size], -1))
            if cfg.qk_norm:
                q, k = _norm(q), _norm(k)
            q, k = (_rotate(t, pos, cfg.rope_theta, cfg.rotary_dim or 128) for t in (q, k))
            k, v, a = _cached(k, bits[0]), _cached(v.contiguous(), bits[1]), torch.empty_like(q)
            for b in range(PROMPTS if most else 0):
                s = slice(b * most, (b + 1) * most)
                a[s] = _attend(q[s], k[s], v[s], 0)
            for j, (c, _) in enumerate(lengths):
                s, p = slice(starts[j], starts[j + 1]), slice(j % PROMPTS * most, j % PROMPTS * most + c)
                a[s] = _attend(q[s], torch.cat([k[p], k[s]]), torch.cat([v[p], v[s]]), c)
            a = a.view(-1, cfg.q_size)
            if cfg.attn_output_gate:
                a = a * (x @ _values(cfg, l.gate()).t()).sigmoid()
            h += _as_fp8(cfg, a) @ _values(cfg, l.o()).t()
        x = _norm(h)
        if cfg.is_moe:
            h += _experts(cfg, l, x)
        else:
            for r in range(0, x.shape[0], 4096):
                g, u = (x[r:r + 4096] @ _values(cfg, l.gate_up()).t()).chunk(2, -1)
                h[r:r + 4096] += (torch.nn.functional.silu(g) * u) @ _values(cfg, l.down()).t()
    last = torch.tensor(starts[1:], device="cuda") - 1
    return {"logits": _norm(h[last]) @ _head(cfg, seed).double().t()}
