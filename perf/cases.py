"""The work that this framework's speed is judged by.

Each case is a call that a program using the framework makes over and over:

  decode     one decode step of a running batch (``engine.step``): every sequence gets its next token
  prompt     the prompt pass of one sequence (``engine.prefill``), from nothing or on top of cached tokens
  attention  the paged decode attention operator alone (``ops.paged_attn_decode``), for callers with a model of their own
  experts    the FP8 mixture-of-experts operator alone (``ops.moe_fp8_forward``), likewise

for the three model families at the built-in shapes (qwen3-30b-a3b cut to 12 of its 48 equal layers, sulepel-2048 and
sefalorn-2048 whole).  Weights are random.  The embedding is large enough that a layer adds a small part to the residual
stream, as in a trained model, the router's logits have a trained router's spread, and row t + 1 of the output matrix points
along embedding row t, so that the next token has the clear lead over the others that a trained model gives most tokens.
Caches hold unit-variance keys and values on shuffled pages; the engines run with logits kept.

``exact`` restates each path in 64 bits with torch alone.  The e4m3 rounding of expert weights and of activations ahead of the
expert products is part of the operator (it defines what is multiplied), so it is restated too.
"""
from __future__ import annotations

import dataclasses
import importlib
import math
import zlib

import numpy as np
import torch

PAGE = 16
DEV = "cuda"
BF, F64 = torch.bfloat16, torch.float64
QWEN, SULEPEL, SEFALORN = "qwen3-30b-a3b", "sulepel-2048", "sefalorn-2048"
RESERVE = 256  # tokens a server keeps room for beyond the context of a row


def pkg(sub: str):
    return importlib.import_module("inference-server_b200." + sub)


# ---------------------------------------------------------------------- cases


def listed() -> list[dict]:
    return [
        # one user, one sequence: every launch and every dependent load shows
        dict(name="decode-1", kind="decode", model=QWEN, layers=12, rows=1, ctx_min=2000, ctx_max=2000),
        # a lightly loaded server: an odd number of short and longer chats, padded to the next graph size
        dict(name="decode-37", kind="decode", model=QWEN, layers=12, rows=37, ctx_min=60, ctx_max=2048),
        # the framework's headline workload: continuous batching of 256 sequences
        dict(name="decode-256", kind="decode", model=QWEN, layers=12, rows=256, ctx_min=512, ctx_max=4096),
        # a short question
        dict(name="prompt-91", kind="prompt", model=QWEN, layers=12, tokens=91, cached=0),
        # a prompt of the benchmark's length, two chunks
        dict(name="prompt-2048", kind="prompt", model=QWEN, layers=12, tokens=2048, cached=0),
        # the next turn of a long conversation: most of the prompt is found in the cache
        dict(name="prompt-deep", kind="prompt", model=QWEN, layers=12, tokens=1500, cached=14001),
        # the attention operator at the benchmark's shape: groups of rows share a system prompt's pages
        dict(name="attention-64", kind="attention", rows=64, q_heads=32, kv_heads=4, ctx_min=512, ctx_max=8192, group=8, shared=1024),
        # the expert layer at the size where it is arithmetic that counts
        dict(name="experts-4096", kind="experts", hidden=2048, inter=768, tokens=4096, tiled=True),
        # the other two families: a full batch, and a prompt
        dict(name="sulepel-decode-256", kind="decode", model=SULEPEL, layers=12, rows=256, ctx_min=512, ctx_max=4096),
        dict(name="sulepel-prompt-2048", kind="prompt", model=SULEPEL, layers=12, tokens=2048, cached=0),
        dict(name="sefalorn-decode-256", kind="decode", model=SEFALORN, layers=8, rows=256, ctx_min=512, ctx_max=4096),
        dict(name="sefalorn-prompt-1777", kind="prompt", model=SEFALORN, layers=8, tokens=1777, cached=0),
    ]


def draw(rng) -> dict:
    def spread(lo: int, hi: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("decode", "decode", "prompt", "prompt", "attention", "experts"))
    if kind in ("decode", "prompt"):
        model = rng.choice((QWEN, QWEN, SULEPEL, SEFALORN))
        layers = {QWEN: 12, SULEPEL: 12, SEFALORN: 8}[model]
        if kind == "decode":
            hi = spread(64, 4096)
            return dict(kind=kind, model=model, layers=layers, rows=spread(1, 256), ctx_min=max(1, int(hi * rng.uniform(0.02, 0.12))),
                        ctx_max=hi)
        cached = spread(1, 14000) if model == QWEN and rng.random() < 0.4 else 0
        return dict(kind=kind, model=model, layers=layers, tokens=spread(16, 1500 if cached else 2048), cached=cached)
    if kind == "attention":
        hi = spread(64, 8192)
        return dict(kind=kind, rows=spread(1, 96), q_heads=rng.choice((32, 64)), kv_heads=4, ctx_min=max(1, int(hi * rng.uniform(0.02, 1.0))),
                    ctx_max=hi, group=rng.choice((0, 4, 8)), shared=spread(16, 1024))
    hidden, inter = rng.choice(((2048, 768), (2048, 768), (4096, 1536)))
    return dict(kind=kind, hidden=hidden, inter=inter, tokens=spread(1, 4096 if hidden == 2048 else 1024), tiled=rng.random() < 0.7)


# --------------------------------------------------------------------- inputs


def key(seed: int, name: str) -> int:
    return (int(seed) * 1_000_003 + zlib.crc32(name.encode())) % (1 << 62)


def noise(seed: int, name: str, *shape: int, std: float = 1.0, mean: float = 0.0, dtype=BF) -> torch.Tensor:
    g = torch.Generator(device=DEV).manual_seed(key(seed, name))
    return torch.empty(shape, device=DEV, dtype=dtype).normal_(mean, std, generator=g)


def host_rng(seed: int, name: str):
    return np.random.default_rng(key(seed, name))


def vocab_tables(seed: int, vocab: int, width: int):
    embed = noise(seed, "embed", vocab, width, std=2.0)
    return embed, (torch.roll(embed, 1, 0) * 0.01).contiguous()


def quantize_blocks(w: torch.Tensor):
    """[E, rows, cols] -> e4m3 and an fp32 factor per 128 x 128 block."""
    E, R, C = w.shape
    t = w.float().view(E, R // 128, 128, C // 128, 128)
    scale = 448.0 / t.abs().amax(dim=(2, 4))
    q = t.mul_(scale[:, :, None, :, None]).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.view(E, R, C), (1.0 / scale).contiguous()


def expert_weights(seed: int, name: str, experts: int, hidden: int, inter: int):
    w13, s13 = quantize_blocks(noise(seed, name + "w13", experts, 2 * inter, hidden, std=0.02))
    w2, s2 = quantize_blocks(noise(seed, name + "w2", experts, hidden, inter, std=0.02))
    return w13, s13, w2, s2


def qwen_layer(seed: int, li: int, c) -> dict:
    n, H, D = f"l{li}.", c.hidden, c.head_dim
    w13, s13, w2, s2 = expert_weights(seed, n, c.experts, H, c.moe_inter)
    return dict(ln1=noise(seed, n + "ln1", H, std=0.1, mean=1.0), ln2=noise(seed, n + "ln2", H, std=0.1, mean=1.0),
                q_norm=noise(seed, n + "qn", D, std=0.1, mean=1.5), k_norm=noise(seed, n + "kn", D, std=0.1, mean=1.0),
                wqkv=noise(seed, n + "qkv", (c.q_heads + 2 * c.kv_heads) * D, H, std=0.02),
                wo=noise(seed, n + "o", H, c.q_heads * D, std=0.02), router=noise(seed, n + "router", c.experts, H, std=0.06),
                w13=w13, w13_scale=s13, w2=w2, w2_scale=s2)


def layered_tensors(seed: int, c, only: int | None = None) -> dict:
    """A checkpoint's tensors, or those of one layer."""
    out, W = {}, c.width
    for i, spec in enumerate(c.layer_list):
        if only is not None and i != only:
            continue
        p, m = f"l{i}.", spec.mixer
        for name, shape in c.tensor_shapes().items():
            if not name.startswith(p) or ".mlp.e" in name:
                continue
            std, mean = 0.02, 0.0
            tail = name[len(p):]
            if tail in ("norm1", "norm2", "mix.norm", "mix.right.norm", "mix.dkv.norm", "mix.temp"):
                std, mean = 0.1, 1.0
            elif "conv" in tail or tail == "canon1":
                std = 0.3
            elif tail.endswith(".dt_bias"):
                std, mean = 1.0, -4.0
            elif tail.endswith("A_log"):
                std, mean = 0.7, 1.5
            elif tail.endswith((".r1", ".r2")):
                std, mean = 0.05, 0.3
            t = noise(seed, name, *shape, std=std, mean=mean)
            if tail.endswith((".r1", ".r2")):
                t = t.abs()
            if tail.endswith(".talk"):
                t = t + torch.eye(shape[0], device=DEV, dtype=BF)
            out[name] = t
        if c.gated and spec.mlp is not None:
            e = spec.mlp
            for part, shape in (("gate", (e.inner, W)), ("up", (e.inner, W)), ("down", (W, e.inner))):
                every = noise(seed, f"{p}mlp.{part}", e.experts, *shape, std=0.02)
                out.update({f"{p}mlp.e{j}.{part}": every[j] for j in range(e.experts)})
    return out


def model_config(case: dict):
    if case["model"] == QWEN:
        return dataclasses.replace(pkg("engine").CONFIGS[QWEN], layers=case["layers"])
    c = pkg("layered").CONFIGS[case["model"]]
    return dataclasses.replace(c, layer_list=c.layer_list[:case["layers"]])


def row_lengths(case: dict, seed: int) -> np.ndarray:
    """Tokens already cached per row: evenly over the range, in any order."""
    if case["kind"] == "prompt":
        return np.array([case["cached"] + case["tokens"] - 1])
    return host_rng(seed, "lens").permutation(np.linspace(case["ctx_min"], case["ctx_max"], case["rows"]).round().astype(np.int64))


def page_lists(lens, seed: int) -> tuple[list[np.ndarray], int]:
    """Shuffled pages for rows of lens + 1 tokens, and their number."""
    n = [int(v) // PAGE + 1 for v in lens]
    perm = host_rng(seed, "pages").permutation(sum(n))
    return np.split(perm, np.cumsum(n)[:-1]), sum(n)


def build_engine(case: dict, seed: int, blocks: int, max_batch: int, max_pages: int):
    c = model_config(case)
    embed, head = vocab_tables(seed, c.vocab_size, c.hidden)
    if case["model"] == QWEN:
        em, quant, layers = pkg("engine"), pkg("quant"), []
        for li in range(c.layers):
            w = em.LayerWeights()
            for name, t in qwen_layer(seed, li, c).items():
                setattr(w, name, quant.tile_weight_blocks(t) if name in ("w13", "w2") else t)
            layers.append(w)
        e = em.DecodeEngine(c, blocks, max_batch, max_pages, layers=layers, embed=embed, lm_head=head,
                            final_norm=noise(seed, "final", c.hidden, std=0.1, mean=1.0), keep_logits=True)
    else:
        tensors = layered_tensors(seed, c)
        tensors.update({"embed": embed, "head": head, "final.norm": noise(seed, "final", c.width, std=0.1, mean=1.0)})
        e = pkg("layered").LayeredEngine(c, blocks, max_batch, max_pages, tensors=tensors, keep_logits=True)
    for kind, std in (("k_pools", 1.0), ("v_pools", 1.0), ("c_pools", 1.0), ("hist", 1.0), ("states", 0.1), ("rings", 1.0)):
        for li, t in enumerate(getattr(e, kind, [])):
            if t is not None:
                t.copy_(noise(seed, f"{kind}{li}", *t.shape, std=std, dtype=t.dtype))
    return e


def decode_batch(rows: int) -> int:
    """Rows a server that runs `rows` of them is set up for."""
    return max(16, 1 << (rows - 1).bit_length()) if rows > 1 else 1


def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "attention":
        return prepare_attention(case, seed)
    if case["kind"] == "experts":
        return prepare_experts(case, seed)
    lens = row_lengths(case, seed)
    pages, blocks = page_lists(lens, seed)
    vocab = model_config(case).vocab_size
    if case["kind"] == "prompt":
        n = case["cached"] + case["tokens"]
        e = build_engine(case, seed, blocks, 1, -(-(n + RESERVE) // PAGE))
        return dict(case=case, engine=e, blocks=blocks, tokens=host_rng(seed, "tokens").integers(0, vocab, size=n).tolist(),
                    pages=pages[0].tolist())
    B = case["rows"]
    e = build_engine(case, seed, blocks, decode_batch(B), -(-(case["ctx_max"] + RESERVE) // PAGE))
    table = np.zeros((B, e.max_pages), dtype=np.int32)
    for i, p in enumerate(pages):
        table[i, : len(p)] = p
    e.block_table[:B].copy_(torch.from_numpy(table))
    state = dict(case=case, engine=e, blocks=blocks, lens=torch.from_numpy(lens.astype(np.int32)).to(DEV),
                 tokens=torch.from_numpy(host_rng(seed, "tokens").integers(0, vocab, size=B)).to(DEV))
    run(state)  # a server has its graphs before its first request; a step may be run again from the same position
    return state


def shared_pages(case: dict, seed: int):
    """Block table of the attention operator: rows of a group share the full pages of their first tokens."""
    lens = row_lengths(case, seed)
    n = [-(-int(v) // PAGE) for v in lens]
    perm = host_rng(seed, "pages").permutation(sum(n)).tolist()
    table, shared, g = np.zeros((case["rows"], max(n)), dtype=np.int32), {}, case["group"]
    for b, v in enumerate(lens):
        for p in range(n[b]):
            if g and (p + 1) * PAGE <= min(int(v), case["shared"]):
                if (b // g, p) not in shared:
                    shared[b // g, p] = perm.pop()
                table[b, p] = shared[b // g, p]
            else:
                table[b, p] = perm.pop()
    return lens, table, sum(n)


def prepare_attention(case: dict, seed: int) -> dict:
    lens, table, blocks = shared_pages(case, seed)
    B, Hq, G, D = case["rows"], case["q_heads"], case["kv_heads"], 128
    ops = pkg("ops")
    split = ops.default_split_tokens(B, G, table.shape[1] * PAGE)
    return dict(case=case, q=noise(seed, "q", B, Hq, D, std=1.5), k=noise(seed, "k", blocks, G, PAGE, D), v=noise(seed, "v", blocks, G, PAGE, D),
                table=torch.from_numpy(table).to(DEV), lens=torch.from_numpy(lens.astype(np.int32)).to(DEV), split=split,
                ws=ops.paged_attn_workspace(B, Hq, D, table.shape[1], PAGE, split, DEV))


def prepare_experts(case: dict, seed: int) -> dict:
    H, I, T = case["hidden"], case["inter"], case["tokens"]
    ops, quant = pkg("ops"), pkg("quant")
    w13, s13, w2, s2 = expert_weights(seed, "", 128, H, I)
    if case["tiled"]:
        w13, w2 = quant.tile_weight_blocks(w13), quant.tile_weight_blocks(w2)
    return dict(case=case, x=noise(seed, "x", T, H), logits=noise(seed, "logits", T, 128, dtype=torch.float32), w13=w13, s13=s13, w2=w2, s2=s2,
                ws=ops.moe_fp8_workspace(T, 128, 8, H, I, DEV))


# ---------------------------------------------------------------------- calls


def run(s: dict):
    case = s["case"]
    if case["kind"] == "attention":
        return pkg("ops").paged_attn_decode(s["q"], s["k"], s["v"], s["table"], s["lens"], 128 ** -0.5, s["split"], s["ws"])
    if case["kind"] == "experts":
        return pkg("ops").moe_fp8_forward(s["x"], s["logits"], s["w13"], s["s13"], s["w2"], s["s2"], 8, True, s["ws"])
    e = s["engine"]
    if case["kind"] == "decode":
        B = case["rows"]
        e.tokens[:B].copy_(s["tokens"], non_blocking=True)
        e.ctx_lens[:B].copy_(s["lens"], non_blocking=True)
        out = dict(tokens=e.step(B), logits=e.last_logits[:B])
    else:
        first, logits = e.prefill(s["tokens"], s["pages"], cached_tokens=case["cached"])
        out = dict(tokens=first, logits=logits)
    # the caches of the last layers that have them, without the engine's scratch page and scratch slot
    for kind in ("k_pools", "v_pools", "c_pools"):
        pools = [t for t in getattr(e, kind, []) if t is not None]
        if pools:
            out[kind] = pools[-1][: s["blocks"]]
    if getattr(e, "num_slots", 0):
        out["states"] = e.states[-1][: case["rows"] if case["kind"] == "decode" else 1]
    return out


# ----------------------------------------------------------------- accounting


def seen_tokens(case: dict, window: int = 0, chunk: int = 0) -> tuple[float, float]:
    """(query, key) pairs, and tokens of cache read, of one attention layer; expected values over the lengths."""
    def of(pos):
        n = pos + 1
        n = n - pos // chunk * chunk if chunk else n
        return np.minimum(n, window) if window else n

    if case["kind"] == "prompt":
        pos = np.arange(case["cached"], case["cached"] + case["tokens"])
        return float(of(pos).sum()), float(min(case["cached"] + case["tokens"], window + case["tokens"] if window else 1 << 60))
    n = float(of(np.arange(case["ctx_min"], case["ctx_max"] + 1)).mean()) * case["rows"]
    return n, n


def experts_hit(tokens: int, experts: int, top: int) -> float:
    return experts * (1.0 - (1.0 - top / experts) ** tokens)


def work(case: dict) -> dict:
    if case["kind"] == "attention":
        B, Hq, G = case["rows"], case["q_heads"], case["kv_heads"]
        lens = np.arange(case["ctx_min"], case["ctx_max"] + 1)
        total = float(lens.mean()) * B
        again = float(np.minimum(lens, case["shared"]).mean()) // PAGE * PAGE * (B - -(-B // case["group"])) if case["group"] else 0.0
        return dict(bytes=(total - again) * G * 512 + B * Hq * 512, flops=4.0 * total * Hq * 128)
    if case["kind"] == "experts":
        T, H, I = case["tokens"], case["hidden"], case["inter"]
        return dict(bytes=experts_hit(T, 128, 8) * 3.0 * H * I + T * (4.0 * H + 512), flops=T * 8 * 6.0 * H * I)
    c = model_config(case)
    M = case["rows"] if case["kind"] == "decode" else case["tokens"]
    out = case["rows"] if case["kind"] == "decode" else 1
    nbytes = c.vocab_size * c.hidden * 2.0 + out * c.vocab_size * (2 if case["model"] == QWEN else 4) + M * c.hidden * 2.0
    flops = 2.0 * out * c.vocab_size * c.hidden
    if case["model"] == QWEN:
        H, hd = c.hidden, (c.q_heads + 2 * c.kv_heads) * c.head_dim
        pairs, read = seen_tokens(case)
        dense = H * (hd + c.q_heads * c.head_dim + c.experts)
        per = 3.0 * H * c.moe_inter
        nbytes += c.layers * (2.0 * dense + experts_hit(M, c.experts, c.top_k) * per + read * c.kv_heads * c.head_dim * 4)
        flops += c.layers * (2.0 * M * dense + 2.0 * M * c.top_k * per + 4.0 * pairs * c.q_heads * c.head_dim)
        return dict(bytes=nbytes, flops=flops)
    W = c.width
    for spec in c.layer_list:
        m = spec.mixer
        if not c.gated and hasattr(m, "kv_heads"):
            dense = W * (m.heads * (m.dim + m.vdim + 1) + m.kv_heads * (m.dim + m.vdim))
            pairs, read = seen_tokens(case, chunk=m.chunk)
            nbytes += read * m.kv_heads * (m.dim + m.vdim) * 2
            flops += 2.0 * pairs * m.heads * (m.dim + m.vdim)
        elif not c.gated:
            dense = W * (m.heads * (m.dim + m.vdim + 1) + m.rank) + m.rank * m.heads * (m.dim + m.vdim)
            pairs, read = seen_tokens(case)
            nbytes += read * m.rank * 2
            flops += (4.0 * pairs * m.heads * m.rank if case["kind"] == "decode" else 2.0 * pairs * m.heads * (m.dim + m.vdim))
        elif hasattr(m, "left"):
            a, r = m.left, m.right
            dense = W * (a.heads * (a.dim + a.vdim) + a.kv_heads * (a.dim + a.vdim) + 2 * r.kv_heads * r.dim + 3 * r.heads * r.vdim
                         + 2 * r.heads + W)
            pairs, read = seen_tokens(case, window=a.window)
            nbytes += read * a.kv_heads * (a.dim + a.vdim) * 2 + out * r.heads * r.dim * r.vdim * 8.0
            flops += 2.0 * pairs * a.heads * (a.dim + a.vdim) + 6.0 * M * r.heads * r.dim * r.vdim
        else:
            dense = W * (m.heads * (2 * m.dim + 3 * m.vdim) + W)
            nbytes += out * m.heads * m.dim * m.vdim * 8.0
            flops += 4.0 * M * m.heads * m.dim * m.vdim
        if c.gated:
            e = spec.mlp
            dense += W * (W + e.experts)
            nbytes += experts_hit(M, e.experts, e.top) * 6.0 * W * e.inner
            flops += M * e.top * 6.0 * W * e.inner
        elif spec.mlp is not None:
            dense += 3 * W * spec.mlp.inner
        nbytes += 2.0 * dense
        flops += 2.0 * M * dense
    return dict(bytes=nbytes, flops=flops)


def tolerance(case: dict) -> dict:
    """What bf16 (and, for the experts, e4m3) operands give; tokens have a lead far above it and stay the same."""
    if case["kind"] == "attention":
        return {"rel": 0.008, "max": 0.1}
    if case["kind"] == "experts":
        return {"rel": 0.01, "max": 0.2}
    return {"rel": 0.02, "max": 0.6}


# -------------------------------------------------------------- 64-bit oracle


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def quantized(x):
    """Rows as the expert products see them: e4m3 with a factor per 128 columns."""
    t = x.reshape(x.shape[0], -1, 128)
    s = t.abs().amax(-1, keepdim=True) / 448.0
    s = torch.where(s > 0, s, torch.ones_like(s))
    return ((t / s).float().to(torch.float8_e4m3fn).to(F64) * s).reshape(x.shape)


def dequantized(q, s):
    R, C = q.shape
    return (q.to(F64).view(R // 128, 128, C // 128, 128) * s.to(F64)[:, None, :, None]).view(R, C)


def fp8_experts(x, logits, w13, s13, w2, s2, top: int):
    p = torch.softmax(logits, -1)
    val, ids = torch.topk(p, top, -1)
    val = val / val.sum(-1, keepdim=True)
    xq, out, I = quantized(x), torch.zeros_like(x), w2.shape[2]
    for e in range(w13.shape[0]):
        at = (ids == e).nonzero()
        if len(at):
            gu = xq[at[:, 0]] @ dequantized(w13[e], s13[e]).T
            h = quantized(silu(gu[:, :I]) * gu[:, I:])
            out.index_add_(0, at[:, 0], (h @ dequantized(w2[e], s2[e]).T) * val[at[:, 0], at[:, 1], None])
    return out


def softmax_rows(q, k, v, scale, allowed=None):
    """One sequence: q [R, H, D], k and v [n, G, D]; allowed [R, n]."""
    R, H, _ = q.shape
    per = H // k.shape[1]
    out = torch.empty(R, H, v.shape[2], dtype=F64, device=q.device)
    for g in range(k.shape[1]):
        for lo in range(0, R, 512):
            s = torch.einsum("rhd,nd->rhn", q[lo:lo + 512, g * per:(g + 1) * per], k[:, g]) * scale
            if allowed is not None:
                s.masked_fill_(~allowed[lo:lo + 512, None], -math.inf)
            out[lo:lo + 512, g * per:(g + 1) * per] = torch.einsum("rhn,nd->rhd", torch.softmax(s, -1), v[:, g])
    return out


class Sequences:
    """The rows of one pass: groups of consecutive new positions of one sequence each (a decode row is a group of one)."""

    def __init__(self, case: dict, seed: int):
        lens = row_lengths(case, seed)
        self.pages, self.blocks = page_lists(lens, seed)
        self.pages = [torch.from_numpy(p).to(DEV) for p in self.pages]
        if case["kind"] == "prompt":
            self.groups = [(case["cached"], case["tokens"])]
        else:
            self.groups = [(int(n), 1) for n in lens]
        self.pos = torch.cat([torch.arange(f, f + n, device=DEV) for f, n in self.groups])
        self.starts = np.cumsum([0] + [n for _, n in self.groups])

    def __iter__(self):
        """(index, first position, new tokens, rows in the pass, pages)"""
        for i, (f, n) in enumerate(self.groups):
            yield i, f, n, slice(int(self.starts[i]), int(self.starts[i]) + n), self.pages[i]

    def write(self, pool, new):
        """pool [blocks, ..., page, D] with new [rows, ..., D] at the rows' places, in 64 bits."""
        out = pool.to(F64)
        page = torch.cat([p[torch.arange(f, f + n, device=DEV) // PAGE] for _, f, n, _, p in self])
        if out.dim() == 3:
            out[page, self.pos % PAGE] = new
        else:
            out[page, :, self.pos % PAGE] = new
        return out


def cached_rows(pool, pages, n: int):
    """The first n tokens [n, heads, D] of a sequence in [blocks, heads, page, D] (or [n, D] in [blocks, page, D])."""
    t = pool[pages[: -(-n // PAGE)]].to(F64)
    if t.dim() == 4:
        t = t.transpose(1, 2)
    return t.reshape(-1, *t.shape[2:])[:n]


def pool_noise(seed: int, kind: str, li: int, seqs: Sequences, *shape: int):
    return noise(seed, f"{kind}{li}", seqs.blocks + 1, *shape)[: seqs.blocks]


def new_tokens(case: dict, seed: int, vocab: int):
    n = case["rows"] if case["kind"] == "decode" else case["cached"] + case["tokens"]
    t = torch.from_numpy(host_rng(seed, "tokens").integers(0, vocab, size=n)).to(DEV)
    return t if case["kind"] == "decode" else t[case["cached"]:]


def answers(case: dict, head, h) -> dict:
    """Logits of decode rows, or of a prompt's last."""
    h = h if case["kind"] == "decode" else h[-1:]
    logits = torch.cat([h @ head[lo:lo + 16384].to(F64).T for lo in range(0, head.shape[0], 16384)], 1)
    first = logits.argmax(1)
    return dict(tokens=first, logits=logits) if case["kind"] == "decode" else dict(tokens=int(first[0]), logits=logits[0])


def exact_qwen(case: dict, seed: int) -> dict:
    c, seqs = model_config(case), Sequences(case, seed)
    D, Hq, G, eps = c.head_dim, c.q_heads, c.kv_heads, c.rms_eps
    embed, head = vocab_tables(seed, c.vocab_size, c.hidden)
    x = embed[new_tokens(case, seed, c.vocab_size)].to(F64)
    freq = c.rope_theta ** (-torch.arange(0, D, 2, dtype=F64, device=DEV) / D)
    ang = seqs.pos.to(F64)[:, None] * freq[None]
    cos, sin = (torch.cat([f, f], -1)[:, None] for f in (ang.cos(), ang.sin()))

    def rope(t):
        return t * cos + torch.cat([-t[..., D // 2:], t[..., : D // 2]], -1) * sin

    for li in range(c.layers):
        w = {n: t if n in ("w13", "w2", "w13_scale", "w2_scale") else t.to(F64) for n, t in qwen_layer(seed, li, c).items()}
        qkv = (rms(x, eps) * w["ln1"] @ w["wqkv"].T).view(len(x), -1, D)
        q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + G], qkv[:, Hq + G:]
        q, k = rope(rms(q, eps) * w["q_norm"]), rope(rms(k, eps) * w["k_norm"])
        kp, vp = (pool_noise(seed, n, li, seqs, G, PAGE, D) for n in ("k_pools", "v_pools"))
        o = torch.empty_like(q)
        for _, f, n, at, pages in seqs:
            ks, vs = (torch.cat([cached_rows(p, pages, f), t[at]]) for p, t in ((kp, k), (vp, v)))
            mask = None if n == 1 else torch.arange(f + n, device=DEV)[None] <= torch.arange(f, f + n, device=DEV)[:, None]
            o[at] = softmax_rows(q[at], ks, vs, D ** -0.5, mask)
        x = x + o.reshape(len(x), -1) @ w["wo"].T
        h = rms(x, eps) * w["ln2"]
        x = x + fp8_experts(h, h @ w["router"].T, w["w13"], w["w13_scale"], w["w2"], w["w2_scale"], c.top_k)
    out = answers(case, head, rms(x, eps) * noise(seed, "final", c.hidden, std=0.1, mean=1.0).to(F64))
    return dict(out, k_pools=seqs.write(kp, k), v_pools=seqs.write(vp, v))


def group_rms(x, w, eps, groups):
    return rms(x.view(len(x), groups, -1), eps).view(x.shape) * w


def exact_sulepel(case: dict, seed: int) -> dict:
    c, seqs = model_config(case), Sequences(case, seed)
    W, eps, taps = c.width, c.norm_eps, c.taps
    embed, head = vocab_tables(seed, c.vocab_size, W)
    i = torch.arange(W // 2, dtype=F64, device=DEV)
    ang = seqs.pos.to(F64)[:, None] * 10000.0 ** (-2.0 * i / W)[None]
    x = embed[new_tokens(case, seed, c.vocab_size)].to(F64) + torch.stack([ang.sin(), ang.cos()], -1).view(len(seqs.pos), W)
    out = {}
    for li, spec in enumerate(c.layer_list):
        m = spec.mixer
        w = {n[len(f"l{li}."):]: t.to(F64) for n, t in layered_tensors(seed, c, li).items()}
        normed = group_rms(x, w["norm1"], eps, c.norm_groups)
        hist, rows = pool_noise(seed, "hist", li, seqs, min(taps, PAGE), W), min(taps, PAGE)
        h = normed.clone()
        for _, f, n, at, pages in seqs:
            before = [hist[pages[p // PAGE], p % PAGE % rows].to(F64) if p >= 0 else torch.zeros(W, dtype=F64, device=DEV)
                      for p in range(f - taps + 1, f)]
            line = torch.cat([torch.stack(before), normed[at]]) if taps > 1 else normed[at]
            for j in range(taps):
                h[at] += w["canon1"][:, j] * line[j:j + n]
        gate = torch.sigmoid(h @ w["mix.g"].T)[..., None]
        q = (h @ w["mix.q"].T).view(len(x), m.heads, m.dim)
        o = torch.empty(len(x), m.heads, m.vdim, dtype=F64, device=DEV)
        if hasattr(m, "kv_heads"):
            q = q * w["mix.temp"][:, None]
            k, v = (h @ w["mix.k"].T).view(len(x), m.kv_heads, m.dim), (h @ w["mix.v"].T).view(len(x), m.kv_heads, m.vdim)
            kp, vp = (pool_noise(seed, n, li, seqs, m.kv_heads, PAGE, m.dim) for n in ("k_pools", "v_pools"))
            for _, f, n, at, pages in seqs:
                ks, vs = (torch.cat([cached_rows(p, pages, f), t[at]]) for p, t in ((kp, k), (vp, v)))
                a, b = torch.arange(f, f + n, device=DEV)[:, None], torch.arange(f + n, device=DEV)[None]
                o[at] = softmax_rows(q[at], ks, vs, m.scale, (b <= a) & ((a // m.chunk == b // m.chunk) if m.chunk else True))
            out.update(k_pools=seqs.write(kp, k), v_pools=seqs.write(vp, v))
        else:
            cp = pool_noise(seed, "c_pools", li, seqs, PAGE, m.rank)
            lat = rms(h @ w["mix.dkv"].T, eps) * w["mix.dkv.norm"]
            for _, f, n, at, pages in seqs:
                cs = torch.cat([cached_rows(cp, pages, f), lat[at]])
                if n == 1:
                    qc = torch.einsum("hd,hdr->hr", q[at][0], w["mix.uk"].view(m.heads, m.dim, m.rank))
                    oc = torch.softmax(qc @ cs.T * m.scale, -1) @ cs
                    o[at] = torch.einsum("hr,hdr->hd", oc, w["mix.uv"].view(m.heads, m.vdim, m.rank))[None]
                    continue
                ks, vs = (cs @ w["mix.uk"].T).view(-1, m.heads, m.dim), (cs @ w["mix.uv"].T).view(-1, m.heads, m.vdim)
                o[at] = softmax_rows(q[at], ks, vs, m.scale, torch.arange(f + n, device=DEV)[None] <= torch.arange(f, f + n, device=DEV)[:, None])
            out.update(c_pools=seqs.write(cp, lat))
        x = x + (o * gate).reshape(len(x), -1) @ w["mix.o"].T
        if spec.mlp is not None:
            h = group_rms(x, w["norm2"], eps, c.norm_groups)
            g, u = (h @ w["mlp.gate"].T).clamp(max=spec.mlp.limit), (h @ w["mlp.up"].T).clamp(-spec.mlp.limit, spec.mlp.limit)
            x = x + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w["mlp.down"].T
    return dict(answers(case, head, group_rms(x, noise(seed, "final", W, std=0.1, mean=1.0).to(F64), eps, c.norm_groups)), **out)


def layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return rms(d, eps) * w


def window_mixer(h, w: dict, a, seqs: Sequences, kp, vp):
    R, per = len(h), a.heads // a.kv_heads
    q = (h @ w["q"].T + w["q.b"]).view(R, a.heads, a.dim)
    k = (h @ w["k"].T + w["k.b"]).view(R, a.kv_heads, a.dim)
    v = (h @ w["v"].T + w["v.b"]).view(R, a.kv_heads, a.vdim)
    o = torch.empty(R, a.heads, a.vdim, dtype=F64, device=DEV)
    for _, f, n, at, pages in seqs:
        ks, vs = (torch.cat([cached_rows(p, pages, f), t[at]]) for p, t in ((kp, k), (vp, v)))
        lo = max(0, f - a.window + 1)
        ks, vs = ks[lo:].repeat_interleave(per, 1), vs[lo:].repeat_interleave(per, 1)
        for s in range(0, n, 256):
            qs = q[at][s:s + 256]
            d = torch.arange(f + s, f + s + len(qs), device=DEV)[:, None] - torch.arange(lo, f + n, device=DEV)[None]
            own = torch.einsum("rhd,nhd->hrn", qs, ks) * a.scale
            own -= w["r1"][:, None, None] * torch.log1p(w["r2"][:, None, None] * d.clamp(min=0).to(F64)[None])
            mixed = torch.einsum("hg,grn->hrn", w["talk"], own).masked_fill_(((d < 0) | (d >= a.window))[None], -math.inf)
            o[at.start + s:at.start + s + len(qs)] = torch.einsum("hrn,nhd->rhd", torch.softmax(mixed, -1), vs)
    return o.reshape(R, -1) @ w["o"].T + w["o.b"], k, v


def delta_mixer(h, w: dict, r, seqs: Sequences, state, ring, eps):
    """`state` [slots, 2, H, d, dv] in 64 bits is brought up to date."""
    R, per = len(h), r.heads // r.kv_heads
    pre = torch.cat([h @ w["q"].T, h @ w["k"].T, h @ w["v"].T], 1)
    conv = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
    act = torch.zeros_like(pre)
    for i, f, n, at, _ in seqs:
        before = [ring[i, p % r.taps].to(F64) if p >= 0 else torch.zeros_like(pre[0]) for p in range(f - r.taps + 1, f)]
        line = torch.cat([torch.stack(before), pre[at]]) if r.taps > 1 else pre[at]
        for j in range(r.taps):
            act[at] += conv[:, j] * line[j:j + n]
    act = silu(act)
    q, k, v = act.split([r.kv_heads * r.dim, r.kv_heads * r.dim, r.heads * r.vdim], 1)

    def unit(t):
        t = t.view(R, r.kv_heads, r.dim)
        return (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(per, 1)

    q, k, v = unit(q) * r.dim ** -0.5, unit(k), v.view(R, r.heads, r.vdim)
    beta = torch.sigmoid(h @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))

    def step(S, t):
        S = S * decay[t][..., None, None]
        e = beta[t][..., None] * (v[t] - torch.einsum("...kv,...k->...v", S, k[t]))
        S = S + k[t][..., None] * e[..., None, :]
        return S, torch.einsum("...kv,...k->...v", S, q[t])

    o = recur(seqs, state, step, R, r.heads, r.vdim)
    o = rms(o, eps) * w["norm"] * silu(h @ w["g"].T).view(o.shape)
    return o.reshape(R, -1) @ w["o"].T


def recur(seqs: Sequences, state, step, R: int, heads: int, vdim: int):
    """Runs `step` over the new tokens; state half (p & 1) holds the state after position p."""
    o = torch.empty(R, heads, vdim, dtype=F64, device=DEV)
    if all(n == 1 for _, n in seqs.groups):
        slot, pos = torch.arange(R, device=DEV), seqs.pos
        S, out = step(state[slot, (pos - 1) & 1] * (pos > 0)[:, None, None, None], slice(None))
        state[slot, pos & 1] = S
        return out
    (_, f, n, at, _), = list(seqs)
    S = state[0, (f - 1) & 1] if f else torch.zeros_like(state[0, 0])
    for t in range(n):
        S, o[t] = step(S, t)
    state[0, (f + n - 1) & 1] = S
    return o


def lightning_mixer(h, w: dict, m, seqs: Sequences, state, eps):
    R = len(h)
    q, k = silu(h @ w["q"].T).view(R, m.heads, m.dim), silu(h @ w["k"].T).view(R, m.heads, m.dim)
    v = silu(h @ w["v"].T).view(R, m.heads, m.vdim)
    decay = torch.tensor(m.decay, dtype=F64, device=DEV)[:, None, None]

    def step(S, t):
        S = S * decay + k[t][..., None] * v[t][..., None, :]
        return S, torch.einsum("...kv,...k->...v", S, q[t])

    o = recur(seqs, state, step, R, m.heads, m.vdim).reshape(R, -1)
    return (rms(o, eps) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def routed_experts(h, w: dict, e):
    val, ids = torch.topk(torch.sigmoid(h @ w["router"].T), e.top, -1)
    val = val / (val.sum(-1, keepdim=True) + 1e-20) * e.scale
    out = torch.zeros_like(h)
    for j in range(e.experts):
        at = (ids == j).nonzero()
        if len(at):
            t = h[at[:, 0]]
            y = (silu(t @ w[f"e{j}.gate"].to(F64).T) * (t @ w[f"e{j}.up"].to(F64).T)) @ w[f"e{j}.down"].to(F64).T
            out.index_add_(0, at[:, 0], y * val[at[:, 0], at[:, 1], None])
    return out


def below(w: dict, prefix: str) -> dict:
    return {n[len(prefix):]: t for n, t in w.items() if n.startswith(prefix)}


def exact_sefalorn(case: dict, seed: int) -> dict:
    c, seqs = model_config(case), Sequences(case, seed)
    W, eps = c.width, c.norm_eps
    slots = (decode_batch(case["rows"]) if case["kind"] == "decode" else 1) + 5
    embed, head = vocab_tables(seed, c.vocab_size, W)
    x = embed[new_tokens(case, seed, c.vocab_size)].to(F64)
    out = {}
    for li, spec in enumerate(c.layer_list):
        m = spec.mixer
        w = {n[len(f"l{li}."):]: t if ".mlp.e" in n else t.to(F64) for n, t in layered_tensors(seed, c, li).items()}
        r = getattr(m, "right", m)
        state = noise(seed, f"states{li}", slots, 2, r.heads, r.dim, r.vdim, std=0.1, dtype=torch.float32)[: len(seqs.groups)].to(F64)
        h = layer_norm(x, w["norm1"], eps)
        if r is not m:
            a = m.left
            ring = noise(seed, f"rings{li}", slots, r.taps, 2 * r.kv_heads * r.dim + r.heads * r.vdim)
            # 64-wide columns of all kv heads of a page lie one after the other
            kp, vp = (pool_noise(seed, n, li, seqs, a.kv_heads * d // 64, PAGE, 64) for n, d in (("k_pools", a.dim), ("v_pools", a.vdim)))
            ks, vs = (p.view(-1, a.kv_heads, d // 64, PAGE, 64).transpose(2, 3).reshape(-1, a.kv_heads, PAGE, d)
                      for p, d in ((kp, a.dim), (vp, a.vdim)))
            left, k, v = window_mixer(h, below(w, "mix.left."), a, seqs, ks, vs)
            y = m.left_scale * left + m.right_scale * delta_mixer(h, below(w, "mix.right."), r, seqs, state, ring, eps)
            out.update({n: seqs.write(p, t.reshape(len(x), -1, 64)) for n, p, t in (("k_pools", kp, k), ("v_pools", vp, v))})
        else:
            y = lightning_mixer(h, below(w, "mix."), m, seqs, state, eps)
        out["states"] = state
        x = x + torch.sigmoid(h @ w["rg1"].T + w["rg1.b"]) * y
        if spec.mlp is not None:
            h = layer_norm(x, w["norm2"], eps)
            x = x + torch.sigmoid(h @ w["rg2"].T + w["rg2.b"]) * routed_experts(h, below(w, "mlp."), spec.mlp)
    h = layer_norm(x, noise(seed, "final", W, std=0.1, mean=1.0).to(F64), eps) * c.logit_scale
    return dict(answers(case, head, h), **out)


def exact(case: dict, seed: int):
    if case["kind"] == "attention":
        s = prepare_attention(case, seed)
        out = torch.empty(s["q"].shape, dtype=F64, device=DEV)
        for b, n in enumerate(row_lengths(case, seed).tolist()):
            ks, vs = (cached_rows(s[p], s["table"][b].long(), n) for p in ("k", "v"))
            out[b] = softmax_rows(s["q"][b:b + 1].to(F64), ks, vs, 128 ** -0.5)[0]
        return out
    if case["kind"] == "experts":
        w = expert_weights(seed, "", 128, case["hidden"], case["inter"])
        x = noise(seed, "x", case["tokens"], case["hidden"]).to(F64)
        return fp8_experts(x, noise(seed, "logits", case["tokens"], 128, dtype=torch.float32).to(F64), *w, 8)
    return {QWEN: exact_qwen, SULEPEL: exact_sulepel, SEFALORN: exact_sefalorn}[case["model"]](case, seed)
