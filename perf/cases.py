"""What is measured: calls that users of this framework make, at the sizes of its own configurations and benchmark.

A case names a model, the call and its sizes:

* "request"  GPT.RunForwardOnSingleDevice: an empty cache, the prompts, then one token after the other;
* "prefill"  GPT.Prefill / PrefillRagged: the prompts of a batch and the first id of every sequence;
* "decode"   a parked cache is restored and the sequences continue for n tokens (GPT.CacheRestore, GPT.Decode), as a server does;
* "fed"      the same with the ids passed through the host at every step (GPT.StepHost), as a program that constrains or streams the text does.

Weights are seeded N(0, 0.02) like the benchmark's, embeddings larger where layers would drown them.  The language-model head also holds a clear successor for every token (id + 1), because a
trained model's next token is rarely a coin toss: the generated ids do not hang on rounding, and a nucleus holds a handful of candidates instead
of half the vocabulary.  The successors of a prompt's last id do not occur in the prompt, where the repeat penalty would change them.
(Models that share the head with the embedding, here the latent one, see the token itself as the likely successor.)
"""
import math
import zlib

import numpy as np
import torch

from seq2seqsharp_b200 import _native as N
from seq2seqsharp_b200.configs import CONFIGS
from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, DecodingStrategyEnums, GPT, MultiHeadAttentionTypeEnums, NormEnums,
                                   PositionEmbeddingEnums)
from seq2seqsharp_b200.layered import (BlockLayer, DenseGated, GroupedAttention, LatentAttention, LayeredConfig, LayeredGPT, MatrixMemory,
                                       TableExperts)

STD = 0.02
PEAK = 20.0      # logit of a token's successor; the other logits have a standard deviation of about 1.5
SHARE = 0.35
TOPP = {"c2_gpt2small_fp16": 0.9, "c5_llama7b_fp16": 0.95}     # the nuclei of the benchmark configurations
TINY, SMALL, M1B, M7B, LATENT, SANDWICH = "c1_tiny_fp32", "c2_gpt2small_fp16", "c3_llama1b_fp16", "c5_llama7b_fp16", "pepilix_2k", "gunuvik_2k"


def case_of(model, call, B, S, n=0, shortest=0):
    """B sequences with prompts of S tokens (shortest > 0: of lengths spread evenly from there to S), n tokens generated."""
    return {"model": model, "call": call, "B": B, "S": S, "n": n, "shortest": shortest or S}


def listed():
    named = lambda name, *a, **k: dict(case_of(*a, **k), name=name)  # noqa: E731
    return [
        # the smallest model, one user: all latency
        named("tiny_fp32_request", TINY, "request", 1, 32, 128),
        # a small model that samples for a handful of users
        named("small_topp_request_8", SMALL, "request", 8, 128, 64),
        # one user's prompt, a batch of users answered together, and the two halves of a long-document request
        named("1b_prefill_1k", M1B, "prefill", 1, 1024),
        named("1b_decode_32", M1B, "decode", 32, 1024, 32),
        named("1b_prefill_16k", M1B, "prefill", 1, 16384),
        named("1b_decode_16k_4", M1B, "decode", 4, 16384, 16),
        # the flagship: one user, a full server, and prompts of different lengths that arrive together
        named("7b_decode_1", M7B, "decode", 1, 512, 32),
        named("7b_decode_64", M7B, "decode", 64, 512, 16),
        named("7b_prefill_mixed_4", M7B, "prefill", 4, 509, shortest=127),
        # layered models in bf16: latent attention with experts (prompts; eight users fed by the host), windowed attention with matrix memories
        named("latent_prefill_3", LATENT, "prefill", 3, 1537),
        named("latent_fed_8", LATENT, "fed", 8, 2048, 32),
        named("sandwich_request_4", SANDWICH, "request", 4, 1024, 32),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.randrange(9)
    if kind == 0:
        return case_of(TINY, "request", spread(1, 8), spread(8, 200), spread(16, 128))
    if kind == 1:
        return case_of(SMALL, "request", spread(1, 32), spread(16, 512), spread(16, 64))
    if kind == 2:
        S = spread(48, 16384)
        return case_of(M1B, "prefill", spread(1, max(1, min(16, 16384 // S))), S)
    if kind == 3:
        B = spread(1, 32)
        return case_of(M1B, "decode", B, spread(48, min(16384, 65536 // B)), spread(8, 32))
    if kind == 4:
        B = spread(1, 64)
        return case_of(M7B, "decode", B, spread(48, min(2048, 32768 // B)), spread(8, 16))
    if kind == 5:
        S = spread(33, 2048)
        return case_of(M7B, "prefill", spread(1, max(1, min(16, 4096 // S))), S, shortest=spread(max(1, S // 8), S))
    if kind == 6:
        S = spread(32, 2048)
        return case_of(LATENT, "prefill", spread(1, max(1, min(16, 6144 // S))), S)
    if kind == 7:
        B = spread(1, 32)
        return case_of(LATENT, "fed", B, spread(32, min(2048, 32768 // B)), spread(8, 32))
    S = spread(32, 2048)
    return case_of(SANDWICH, "request", spread(1, max(1, min(16, 8192 // S))), S, spread(8, 32))


# ---- models ---------------------------------------------------------------------------------------------------------------------
def config(name):
    """The benchmark's configurations: the uniform decoders, and the 2048-wide sizes of the layered designs."""
    if name in CONFIGS:
        return CONFIGS[name]
    d, V = 2048, 32000
    if name == LATENT:
        experts = TableExperts(experts=32, top=4, ff=1408, limit=7.0, slope=1.702, shift=1.0)
        mixer = LatentAttention(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, rot_base=1e6, scale=192 ** -0.5)
        return LayeredConfig(name=name, d=d, V=V, norm_groups=8, conv_taps=4, embed_scale=d ** 0.5, layers=[BlockLayer(mixer, experts) for _ in range(12)])
    at = dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, window=1024, keep_first=4, bias_rows=32, bias_max=128,
              qk_norm=True, qkv_bias=True, sink=True, head_gate=True)
    return LayeredConfig(name=name, d=d, V=V, block="sandwich", embed_scale=d ** 0.5, tied_head=False,
                         layers=[BlockLayer(MatrixMemory(8, 128, 256, 15.0) if i % 4 == 2 else GroupedAttention(**at, kv_from=i - 2 if i % 4 == 3 else -1),
                                            dense=DenseGated(5632)) for i in range(12)])


def is_layered(cfg):
    return isinstance(cfg, LayeredConfig)


def embedding(cfg):
    """(standard deviation of the embedding table, share of the current token's embedding in the last normed row; the rest is what the layers
    added).  In a deep model weights of N(0, 0.02) would drown the token that is being read: the table is then scaled up to a share of SHARE."""
    scale = cfg.embed_scale if is_layered(cfg) else math.sqrt(cfg.d)
    if is_layered(cfg):
        added = 2.0 * cfg.L          # two normed sublayers
    else:
        s = cfg.d * STD ** 2
        added = cfg.L * cfg.F * STD ** 2 * {ActivateFuncEnums.ReLU: 0.5 * s, ActivateFuncEnums.GELU: 0.4 * s, ActivateFuncEnums.SwiGLU: s * s}[cfg.act]
    std = STD if cfg.name == LATENT else max(STD, math.sqrt(added * SHARE ** 2 / (1.0 - SHARE ** 2)) / scale)
    own = (std * scale) ** 2
    return std, math.sqrt(own / (own + added))


class Weights:
    """The model's tensors by the names that the engine takes, made from the seed one at a time, in the model's own type."""

    def __init__(self, cfg, seed, max_pos):
        self.cfg, self.seed = cfg, seed
        self.shapes = cfg.weight_shapes() if is_layered(cfg) else cfg.weight_shapes(max_pos)
        self.dtype = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}[cfg.dtype]

    def __call__(self, name):
        g = torch.Generator("cuda")
        g.manual_seed(zlib.crc32(name.encode()) * 1000003 + self.seed)
        shape, cfg = self.shapes[name], self.cfg
        if name.endswith("experts.table"):
            experts = cfg.layers[int(name.split(".")[1])].experts
            return torch.rand(shape[0], experts.experts, device="cuda", generator=g).argsort(dim=1)[:, :experts.top].int().contiguous()
        std, mean = embedding(cfg)[0] if name in ("embed", "TgtEmbeddings") else STD, 0.0
        if name.endswith(("m_alpha", "norm", "norm1", "norm2", "norm1b", "norm2b", "scale1", "scale2")):
            std, mean = 0.1, 1.0
        elif name.endswith("conv1"):
            std = 0.3
        elif name.endswith("mem.f.b"):
            std, mean = 0.5, 3.0      # memories start out remembering
        w = torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, std, generator=g)
        if name in ("FeedForward_Decoder_0.m_Whd", "head"):
            e = self("embed" if name == "head" else "TgtEmbeddings").float()
            e *= PEAK / (math.sqrt(cfg.d) * embedding(cfg)[1]) / e.norm(dim=1, keepdim=True)
            w += e.roll(1, 0) if name == "head" else e.roll(1, 0).t()
        return w.to(self.dtype)


def engine(cfg, seed, max_batch, max_tokens):
    gpt = (LayeredGPT if is_layered(cfg) else GPT)(cfg, max_batch=max_batch, max_tokens=max_tokens)
    weights = Weights(cfg, seed, max_tokens + 2)
    types = {torch.float32: N.F32, torch.float16: N.F16, torch.bfloat16: N.BF16, torch.int32: N.I32}
    for name, shape in weights.shapes.items():
        w = weights(name)
        torch.cuda.synchronize()     # the engine reads it on a stream of its own
        N.call("TSB200_GptSetWeight", gpt._h, name.encode(), w.data_ptr(), types[w.dtype], shape[0], shape[1], 1)
    return gpt


# ---- the calls ------------------------------------------------------------------------------------------------------------------
def lengths(case):
    B, S, lo = case["B"], case["S"], case["shortest"]
    return [S - (S - lo) * b // max(1, B - 1) for b in range(B)]


def prompts(case, seed):
    """Ids from the upper half of the vocabulary, the last one of every prompt from the lower half with room for its successors."""
    rng, V = np.random.default_rng(seed), config(case["model"]).V
    out = [rng.integers(V // 2, V, size=s).astype(np.int32) for s in lengths(case)]
    for p in out:
        p[-1] = rng.integers(5, V // 2 - case["n"] - 2)
    return out


def options(case, seed):
    o = DecodingOptions(MaxTgtSentLength=case["S"] + case["n"], Seed=seed)
    if case["model"] in TOPP:
        o.DecodingStrategy, o.TopP = DecodingStrategyEnums.Sampling, TOPP[case["model"]]
    return o


def prepare(case, seed):
    cfg = config(case["model"])
    p, o = prompts(case, seed), options(case, seed)
    gpt = engine(cfg, seed, case["B"], case["S"] + case["n"] + 2)
    s = {"case": case, "gpt": gpt, "prompts": p, "opts": o}
    if case["call"] in ("decode", "fed"):
        gpt.Prefill(np.stack(p), o)
        s["snap"] = gpt.CacheSnapshot()
        first = s["snap"].tokens[:, -1]
        s["feed"] = np.stack([first + i for i in range(case["n"])]).astype(np.int32)
    return s


def run(s):
    case, gpt, o = s["case"], s["gpt"], s["opts"]
    if case["call"] == "request":
        ids = gpt.RunForwardOnSingleDevice(np.stack(s["prompts"]), o)
    elif case["call"] == "prefill":
        gpt.Reset()
        ids = gpt.Prefill(np.stack(s["prompts"]), o) if case["shortest"] == case["S"] else gpt.PrefillRagged(s["prompts"], o)
    else:
        gpt.CacheRestore(s["snap"])
        if case["call"] == "decode":
            ids = gpt.Decode(case["n"], o)
        else:
            ids = np.stack([gpt.StepHost(f, o) for f in s["feed"]], axis=1)
    return {"ids": ids, "logits": gpt.Logits(want_probs=False)[0]}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def work(case):
    """Every weight once per forward pass (of a mixture of experts the ones that the batch's tokens name on average), the cached rows read and
    written, ids and logits; multiply-adds of the matrices and of the attended positions."""
    cfg, B, n = config(case["model"]), case["B"], case["n"]
    lens = lengths(case)
    size = 4 if cfg.dtype == "float32" else 2
    tokens = sum(lens)
    if is_layered(cfg):
        dense = dict((k, v) for k, v in cfg.weight_shapes().items() if v[0] > 1 and not k.endswith(("table", "conv1", "bias")) and k != "embed")
        fixed = sum(a * b for k, (a, b) in dense.items() if ".experts." not in k) + cfg.V * cfg.d * cfg.tied_head
        expert = sum(a * b for k, (a, b) in dense.items() if ".experts." in k)
        per_token = cfg.active_matmul_params()
        x = cfg.layers[0].experts
        weights = lambda t: size * (fixed + expert * (1.0 - (1.0 - x.top / x.experts) ** t if x else 0.0))  # noqa: E731
        row, pair, seen, state = 0, 0, [], 0
        for layer in cfg.layers:
            m = layer.mixer
            if isinstance(m, LatentAttention):
                row += m.kv_rank + m.rot_dim
                pair += m.heads * (m.dim + m.rot_dim + m.vdim)
            elif isinstance(m, GroupedAttention):
                row += m.kv_heads * (m.dim + m.vdim) * (m.kv_from < 0)
                pair += m.heads * (m.dim + m.vdim)
                seen.append(m.window + m.keep_first)
            else:
                state += 4 * m.heads * m.dim * (m.vdim + 1)
                per_token += 2 * m.heads * m.dim * m.vdim
        span = max(seen) if seen else 1 << 30
        read = row if not seen else sum(l.mixer.kv_heads * (l.mixer.dim + l.mixer.vdim) for l in cfg.layers if isinstance(l.mixer, GroupedAttention))
    else:
        per_token = cfg.matmul_params()
        weights = lambda t: size * per_token  # noqa: E731
        row = read = cfg.L * 2 * cfg.kv_heads() * cfg.hd
        pair, span, state = cfg.L * 2 * cfg.H * cfg.hd, 1 << 30, 0
    head = cfg.d * cfg.V
    bytes_ = flops = 0.0
    if case["call"] in ("request", "prefill"):
        bytes_ += weights(tokens) + size * row * tokens + 4 * tokens + 4 * B * cfg.V + state * B
        flops += 2.0 * (per_token - head) * tokens + 2.0 * head * B + 2.0 * pair * sum(min(i + 1, span) for s in lens for i in range(s))
    steps = n - 1 if case["call"] == "request" else n
    for i in range(steps):
        T = case["S"] + i
        bytes_ += weights(B) + size * B * (read * min(T, span) + row) + 2 * state * B
        flops += 2.0 * per_token * B + 2.0 * pair * B * min(T + 1, span)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the distance of the logits from exact(); a matrix memory's read-out that is nearly zero before its norm is the most
    sensitive.  The ids have clear winners."""
    rel = {TINY: 1e-5, LATENT: 0.011, SANDWICH: 0.03}.get(case["model"], 0.004)
    return {"rel": rel, "max": 8 * rel, "differ": 0.0}


# ---- the same in 64 bits, without the framework ------------------------------------------------------------------------------------
def _rms(x, w, eps, groups=1):
    p = x.reshape(*x.shape[:-1], groups, -1)
    return (p / torch.sqrt((p * p).mean(-1, keepdim=True) + eps)).reshape(x.shape) * w


def _attend(q, k, v, scale, heads_per_kv, bias=None, span=0, keep=0, sink=None):
    """Causal attention of one sequence: q [H, S, a], k [G, S, a], v [G, S, b] -> [S, H, b], a block of queries at a time."""
    H, S = q.shape[:2]
    kk, vv = k.repeat_interleave(heads_per_kv, 0), v.repeat_interleave(heads_per_kv, 0)
    out = torch.empty(S, H, v.shape[2], dtype=q.dtype, device=q.device)
    block = max(1, min(S, (1 << 27) // (H * S)))
    for a in range(0, S, block):
        b = min(S, a + block)
        z = torch.baddbmm(torch.zeros((), dtype=q.dtype, device=q.device), q[:, a:b], kk[:, :b].transpose(1, 2), beta=0, alpha=scale)
        back = torch.arange(a, b, device=q.device)[:, None] - torch.arange(b, device=q.device)[None]
        hidden = back < 0
        if span:
            hidden |= (back >= span) & (torch.arange(b, device=q.device)[None] >= keep)
        if bias is not None:
            z += bias[:, back.clamp_min(0)]
        z.masked_fill_(hidden, -math.inf)
        m = z.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink[:, None, None])
        z.sub_(m).exp_()
        total = z.sum(-1, keepdim=True)
        if sink is not None:
            total += (sink[:, None, None] - m).exp()
        out[a:b] = ((z @ vv[:, :b]) / total).transpose(0, 1)
    return out


def _sequences(flat, lens):
    return torch.split(flat, lens)


def _decoder(cfg, w, ids, lens, S):
    """Last normed rows of GPTDecoder for the concatenated sequences `ids` (all positions); S: prompt length, for the position table."""
    f = lambda name: w(name).double()  # noqa: E731
    rms = cfg.norm == NormEnums.RMSNorm

    def norm(x, key):
        g = f(key + ".m_alpha")[0]
        return _rms(x, g, cfg.eps) if rms else torch.nn.functional.layer_norm(x, (cfg.d,), g, f(key + ".m_beta")[0], cfg.eps)

    pos = torch.cat([torch.arange(n, device=ids.device) for n in lens])
    x = f("TgtEmbeddings")[ids] * math.sqrt(cfg.d)
    if cfg.pe == PositionEmbeddingEnums.APE:
        x = x + f("PosEmbedding")[torch.where(pos < S, pos, 0 if cfg.ape_decode_pos0 else pos)]
    H, G, hd = cfg.H, cfg.kv_heads(), cfg.hd
    half = torch.arange(hd // 2, device=ids.device, dtype=torch.float64)
    angle = pos[:, None].double() * cfg.rope_base ** (-2.0 * half / hd)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(t):
        if cfg.pe != PositionEmbeddingEnums.RoPE:
            return t
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack((a * cos - b * sin, b * cos + a * sin), -1).reshape(t.shape)

    for k in range(cfg.L):
        a, p = "GPTDecoder.SelfAttn_%d." % k, "GPTDecoder.PosFFN_%d." % k
        h = norm(x, a + "layerNormQ")
        if cfg.attn == MultiHeadAttentionTypeEnums.MHA:
            q, kk, v = (h @ f(a + "QKV") + f(a + "QKVb")).chunk(3, dim=1)
        else:
            q, kk, v = (h @ f(a + n) + f(a + n + "b") for n in ("Q", "K", "V"))
        q, kk, v = turn(q.reshape(-1, H, hd)), turn(kk.reshape(-1, G, hd)), v.reshape(-1, G, hd)
        o = torch.cat([_attend(*(t.transpose(0, 1) for t in s), hd ** -0.5, H // G) for s in zip(*(_sequences(t, lens) for t in (q, kk, v)))])
        x = x + o.reshape(-1, H * hd) @ f(a + "W0") + f(a + "b0")
        h = norm(x, p + "layerNorm2")
        up = h @ f(p + "feedForwardLayer1.m_Whd") + f(p + "feedForwardLayer1.m_Bd")
        if cfg.is_glu():
            up *= h @ f(p + "feedForwardLayer3.m_Whd") + f(p + "feedForwardLayer3.m_Bd")
        else:
            up = torch.relu(up) if cfg.act == ActivateFuncEnums.ReLU else torch.nn.functional.gelu(up)
        x = x + up @ f(p + "feedForwardLayer2.m_Whd") + f(p + "feedForwardLayer2.m_Bd")
    return norm(x, "GPTDecoder.layerNorm")


def _turn_halves(x, pos, dims, base):
    half = dims // 2
    angle = (pos[:, None].double() * base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / dims))[(slice(None),) + (None,) * (x.dim() - 2)]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat((u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin(), x[..., dims:]), -1)


def _latent(cfg, w, ids, lens):
    pos = torch.cat([torch.arange(n, device=ids.device) for n in lens])
    x = w("embed").double()[ids] * cfg.embed_scale
    for i, layer in enumerate(cfg.layers):
        f = lambda name: w("layer.%d.%s" % (i, name)).double()  # noqa: E731,B023
        m, e = layer.mixer, layer.experts
        h1, taps = _rms(x, f("norm1")[0], cfg.eps, cfg.norm_groups), f("conv1")
        hc = h1.clone()
        for j in range(cfg.conv_taps):
            back = cfg.conv_taps - 1 - j
            hc += torch.cat([torch.nn.functional.pad(s, (0, 0, back, 0))[:s.shape[0]] for s in _sequences(h1, lens)]) * taps[:, j]
        d = hc @ f("attn.dkv").t()
        c = _rms(d[:, :m.kv_rank], f("attn.dkv_norm")[0], cfg.eps)
        kr = _turn_halves(d[:, m.kv_rank:], pos, m.rot_dims, m.rot_base)
        q = (hc @ f("attn.q").t()).reshape(-1, m.heads, m.dim + m.rot_dim)
        q = torch.cat((q[..., :m.dim], _turn_halves(q[..., m.dim:], pos, m.rot_dims, m.rot_base)), -1)
        k = torch.cat(((c @ f("attn.uk").t()).reshape(-1, m.heads, m.dim), kr[:, None].expand(-1, m.heads, -1)), -1)
        v = (c @ f("attn.uv").t()).reshape(-1, m.heads, m.vdim)
        o = torch.cat([_attend(*(t.transpose(0, 1) for t in s), m.scale, 1) for s in zip(*(_sequences(t, lens) for t in (q, k, v)))])
        add = (o.reshape(-1, m.heads * m.vdim) @ f("attn.o").t()) * torch.sigmoid(h1 @ f("gate1.w").t() + f("gate1.b"))
        h2, table, y = _rms(x, f("norm2")[0], cfg.eps, cfg.norm_groups), w("layer.%d.experts.table" % i)[ids], torch.zeros_like(x)
        for n in range(e.experts):
            rows = (table == n).any(1).nonzero()[:, 0]
            g = (h2[rows] @ f("experts.%d.gate" % n).t()).clamp(max=e.limit)
            u = (h2[rows] @ f("experts.%d.up" % n).t()).clamp(-e.limit, e.limit)
            y[rows] += (g * torch.sigmoid(e.slope * g) * (u + e.shift)) @ f("experts.%d.down" % n).t() / e.top
        x = x + add + y * torch.sigmoid(h2 @ f("gate2.w").t() + f("gate2.b"))
    return _rms(x, w("final_norm").double()[0], cfg.eps, cfg.norm_groups)


def _memory(q, k, v, i, f):
    """Matrix memory of one sequence, all heads: q, k [S, H, a], v [S, H, b], log gates [S, H] -> [S, H, b]."""
    S, H, a = q.shape
    state, n, m = q.new_zeros(H, a, v.shape[2]), q.new_zeros(H, a), q.new_zeros(H)
    out = torch.empty_like(v)
    for t in range(S):
        new = torch.maximum(f[t] + m, i[t])
        keep, put, m = (f[t] + m - new).exp(), (i[t] - new).exp(), new
        state = keep[:, None, None] * state + put[:, None, None] * k[t][:, :, None] * v[t][:, None]
        n = keep[:, None] * n + put[:, None] * k[t]
        out[t] = (state * q[t][:, :, None]).sum(1) / (torch.maximum((n * q[t]).sum(1).abs(), (-m).exp()) + 1e-6)[:, None]
    return out


def _sandwich(cfg, w, ids, lens):
    x, kept = w("embed").double()[ids] * cfg.embed_scale, {}
    for i, layer in enumerate(cfg.layers):
        f = lambda name: w("layer.%d.%s" % (i, name)).double()  # noqa: E731,B023
        m, h = layer.mixer, _rms(x, f("norm1")[0], cfg.eps)
        if isinstance(m, GroupedAttention):
            def head_rows(name, heads, dim):
                return (h @ f("attn." + name).t() + f("attn.%s.b" % name)).reshape(-1, heads, dim)  # noqa: B023
            if m.kv_from < 0:
                kept[i] = (_rms(head_rows("k", m.kv_heads, m.dim), f("attn.k_norm")[0], cfg.eps), head_rows("v", m.kv_heads, m.vdim))
            k, v = kept[i if m.kv_from < 0 else m.kv_from]
            q = _rms(head_rows("q", m.heads, m.dim), f("attn.q_norm")[0], cfg.eps)
            rows, half = m.bias_rows, m.bias_rows // 2
            bucket = [n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(m.bias_max / half) * (rows - half))) for n in range(max(lens))]
            bias = f("attn.bias")[bucket].t().contiguous()
            o = torch.cat([_attend(*(t.transpose(0, 1) for t in s), m.scale, m.heads // m.kv_heads, bias, m.window, m.keep_first, f("attn.sink")[0])
                           for s in zip(*(_sequences(t, lens) for t in (q, k, v)))])
            y = (o * torch.sigmoid(h @ f("attn.gate").t())[:, :, None]).reshape(-1, m.heads * m.vdim) @ f("attn.o").t()
        else:
            q, k = ((h @ f("mem." + n).t()).reshape(-1, m.heads, m.dim) for n in ("q", "k"))
            v = (h @ f("mem.v").t()).reshape(-1, m.heads, m.vdim)
            gi = m.gate_cap * torch.tanh((h @ f("mem.i").t() + f("mem.i.b")) / m.gate_cap)
            gf = torch.nn.functional.logsigmoid(m.gate_cap * torch.tanh((h @ f("mem.f").t() + f("mem.f.b")) / m.gate_cap))
            o = torch.cat([_memory(*s) for s in zip(*(_sequences(t, lens) for t in (q * m.dim ** -0.5, k, v, gi, gf)))])
            o = _rms(o, 1.0, cfg.eps).reshape(-1, m.heads * m.vdim) * f("mem.norm")
            y = (o * torch.sigmoid(h @ f("mem.gate").t())) @ f("mem.o").t()
        x = x + _rms(y, f("norm1b")[0], cfg.eps) * f("scale1")
        h = _rms(x, f("norm2")[0], cfg.eps)
        y = (torch.nn.functional.silu(h @ f("ff.gate").t()) * (h @ f("ff.up").t())) @ f("ff.down").t()
        x = x + _rms(y, f("norm2b")[0], cfg.eps) * f("scale2")
    return _rms(x, w("final_norm").double()[0], cfg.eps)


def exact(case, seed):
    """One pass over the whole texts: the prompts and the tokens that the engine is fed, which are the successors of the prompts' last ids."""
    cfg, n = config(case["model"]), case["n"]
    latent = case["model"] == LATENT
    texts = []
    for p in prompts(case, seed):
        fed = {"request": n - 1, "prefill": 0, "decode": n, "fed": n}[case["call"]]
        first = p[-1] + (0 if latent else 1)
        texts.append(np.concatenate([p, np.arange(first, first + fed, dtype=np.int32)]))
    lens = [len(t) for t in texts]
    ids = torch.from_numpy(np.concatenate(texts)).long().cuda()
    w = Weights(cfg, seed, case["S"] + n + 4)
    with torch.no_grad():
        rows = (_latent if latent else _sandwich)(cfg, w, ids, lens) if is_layered(cfg) else _decoder(cfg, w, ids, lens, case["S"])
        made = max(1, n)         # the positions whose next id is returned
        rows = torch.stack([r[-made:] for r in _sequences(rows, lens)])
        if is_layered(cfg):
            logits = rows @ w("embed" if cfg.tied_head else "head").double().t() * cfg.logit_scale
        else:
            logits = rows @ w("FeedForward_Decoder_0.m_Whd").double() + w("FeedForward_Decoder_0.m_Bd").double()
    first = logits.argmax(-1).int()
    return {"ids": (first[:, 0] if case["call"] == "prefill" else first).cpu().numpy(), "logits": logits[:, -1].cpu().numpy()}
