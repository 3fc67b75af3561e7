"""The passes a serving user has this framework run, as measurable cases.

The engine serves requests with three kinds of pass over packed rows: a decode step (one row per request, replayed
from a CUDA graph), a speculative step (verify rows, MTP block and draft chain, replayed from a CUDA graph as well)
and a ragged chunked-prefill pass (launched kernel by kernel). A case is one such pass through ``Model``'s public
methods at the full widths of the served architecture, tile-packed as the server packs them, over one period of its
layer pattern (three Gated-DeltaNet layers and one gated-attention layer, every tenth part of the stack being the
same) plus the LM head. ``listed`` covers one request alone up to the largest batch buckets, short to very long
contexts, a short follow-up turn up to a full 8192-row prefill pass; ``draw`` picks others from the same ranges.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from b200serve.config import PAGE_SIZE, ModelConfig
from b200serve.models.checkpoint import LayerWeights, MTPWeights, Weights
from b200serve.models.qwen36 import Model, PackedBatch
from b200serve.ops import cuda_ops

LAYERS = 4           # one period: three Gated-DeltaNet layers, one attention layer
WIDTHS = (64, 512, 4096)  # page-table widths of the decode graphs (contexts up to 4k / 32k / 256k tokens)
DEV = "cuda"


def listed() -> list[dict]:
    return [
        # one interactive request: launches, the weight stream of one row's experts and the LM head
        {"name": "decode_1", "kind": "decode", "seqs": 1, "context": 900, "spread": 0.0, "head": "greedy"},
        # a few coding-agent sessions with long contexts
        {"name": "decode_4_long", "kind": "decode", "seqs": 4, "context": 90000, "spread": 0.5, "head": "greedy"},
        # a small service whose requests sample: the logits of every row are formed
        {"name": "decode_13_sampled", "kind": "decode", "seqs": 13, "context": 3000, "spread": 0.8, "head": "logits"},
        # the benchmark's batch: 128 requests of 1024 prompt tokens
        {"name": "decode_128", "kind": "decode", "seqs": 128, "context": 1088, "spread": 0.06, "head": "greedy"},
        # the largest batch bucket: 256 requests of about 2048 tokens each
        {"name": "decode_256", "kind": "decode", "seqs": 256, "context": 2300, "spread": 0.1, "head": "greedy"},
        # speculative steps: three drafts per request, a few requests and a busy server
        {"name": "verify_3", "kind": "verify", "seqs": 3, "drafts": 3, "context": 2500, "spread": 0.4, "head": "greedy"},
        {"name": "verify_40", "kind": "verify", "seqs": 40, "drafts": 3, "context": 1500, "spread": 0.7, "head": "greedy"},
        # a session's next turn: a short span on top of a cached context
        {"name": "prefill_turn", "kind": "prefill", "seqs": 1, "rows": 61, "context": 3584, "spread": 0.0, "head": "greedy"},
        # several short prompts of different lengths packed into one pass
        {"name": "prefill_ragged", "kind": "prefill", "seqs": 7, "rows": 1531, "context": 0, "spread": 0.8, "head": "logits"},
        # one prompt alone up to the chunk limit
        {"name": "prefill_2048", "kind": "prefill", "seqs": 1, "rows": 2048, "context": 0, "spread": 0.0, "head": "greedy"},
        # the benchmark's prefill: a full pass of eight 1024-token prompts
        {"name": "prefill_8x1024", "kind": "prefill", "seqs": 8, "rows": 8192, "context": 0, "spread": 0.0, "head": "greedy"},
        # a full pass of chunks in the middle of long prompts
        {"name": "prefill_4x2048_long", "kind": "prefill", "seqs": 4, "rows": 8192, "context": 28672, "spread": 0.9, "head": "greedy"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "verify", "prefill", "prefill"))
    spread = round(rng.uniform(0.0, 0.9), 3)
    head = rng.choice(("greedy", "greedy", "logits"))
    if kind == "decode":
        seqs = _log_int(rng, 1, 256)
        return {"kind": kind, "seqs": seqs, "context": _log_int(rng, 64, min(100000, 500000 // seqs)), "spread": spread,
                "head": head}
    if kind == "verify":
        seqs = _log_int(rng, 1, 64)
        return {"kind": kind, "seqs": seqs, "drafts": rng.choice((1, 3, 3)),
                "context": _log_int(rng, 64, min(30000, 200000 // seqs)), "spread": spread, "head": "greedy"}
    rows = _log_int(rng, 16, 8192)
    seqs = rng.randint(max(1, -(-rows // 2048)), max(1, min(16, -(-rows // 2048) * 2 + rows // 200)))
    context = rng.choice((0, 0, PAGE_SIZE * _log_int(rng, 1, 448)))
    return {"kind": kind, "seqs": seqs, "rows": rows, "context": context, "spread": spread, "head": head}


# ------------------------------------------------------------------ the shape of a case
def _config(case: dict) -> ModelConfig:
    return ModelConfig(num_hidden_layers=LAYERS, mtp_num_hidden_layers=int(case["kind"] == "verify"))


def _vary(n: int, spread: float) -> list[float]:
    """``n`` fixed factors in ``[1 - spread, 1]`` that cover the interval evenly."""
    return [1.0 - spread * ((i * 0.6180339887) % 1.0) for i in range(n)]


def _spans(case: dict) -> tuple[list[int], list[int]]:
    """``(rows, position of the first row)`` of every sequence of the pass."""
    n = case["seqs"]
    f = _vary(n, case["spread"])
    if case["kind"] != "prefill":
        g = case.get("drafts", 0) + 1
        return [g] * n, [max(1, int(case["context"] * x)) for x in f]
    rows = [max(1, min(2048, int(case["rows"] * x / sum(f)))) for x in f]  # a span is a chunk of at most 2048 rows
    for i in range(n):
        rows[i] += min(2048 - rows[i], max(0, case["rows"] - sum(rows)))
    # chunks start on a page; a spread of contexts also has a sequence's first chunk among them
    return rows, [int(case["context"] * (x if i else 1.0)) // PAGE_SIZE * PAGE_SIZE for i, x in enumerate(f)]


def _width(case: dict, pages: int) -> int:
    return pages if case["kind"] == "prefill" else next(w for w in WIDTHS if w >= pages)


def work(case: dict) -> dict:
    cfg, (rows, pos0) = _config(case), _spans(case)
    T, n, H, V = sum(rows), len(rows), cfg.hidden_size, cfg.vocab_size
    drafts = case.get("drafts", 0)
    expert = 3 * H * cfg.moe_intermediate_size
    gdn = (cfg.gdn_in_rows + cfg.gdn_value_dim) * H
    attn = (cfg.attn_q_rows + 2 * cfg.attn_kv_rows + cfg.num_attention_heads * cfg.head_dim) * H
    kv_row = 2 * cfg.attn_kv_rows * 2
    state = cfg.linear_num_value_heads * cfg.linear_key_head_dim * cfg.linear_value_head_dim
    conv = cfg.gdn_conv_dim * (cfg.linear_conv_kernel_dim - 1)

    def moe_bytes(t: int) -> float:  # experts that at least one of t rows picks, the shared one and the router
        hit = cfg.num_experts * (1.0 - (1.0 - cfg.num_experts_per_tok / cfg.num_experts) ** t)
        return 2 * (expert * (hit + 1) + H * (cfg.num_experts + 1))

    def moe_flops(t: int) -> float:
        return 2.0 * t * (expert * (cfg.num_experts_per_tok + 1) + H * (cfg.num_experts + 1))

    keys = sum(p + r for p, r in zip(pos0, rows))                       # distinct cached positions of the pass
    pairs = sum(r * p + r * (r + 1) / 2 for p, r in zip(pos0, rows))    # (query, visible key) pairs
    score = 4.0 * cfg.num_attention_heads * cfg.head_dim
    n_gdn, n_attn = len(cfg.gdn_layers), len(cfg.attention_layers)
    picked = T if case["kind"] != "prefill" else n
    b = n_gdn * (2 * gdn + n * 2 * (4 * state + 2 * conv)) + n_attn * (2 * attn + keys * kv_row) + LAYERS * moe_bytes(T)
    f = n_gdn * T * (2.0 * gdn + 8.0 * state) + n_attn * (2.0 * T * attn + pairs * score) + LAYERS * moe_flops(T)
    b += 2 * V * H + T * (2 * H * 2 + 8) + (picked * V * 4 if case["head"] == "logits" else picked * 8)
    f += 2.0 * picked * V * H
    if case["kind"] == "verify":
        # the MTP block over all rows, then one head per draft and one block per later link of the chain
        b += 2 * attn + 4 * H * H + keys * kv_row + moe_bytes(T) + 2 * V * H
        f += T * (2.0 * attn + 4.0 * H * H) + pairs * score + moe_flops(T) + 2.0 * n * V * H
        b += (drafts - 1) * (2 * attn + 4 * H * H + keys * kv_row + moe_bytes(n) + 2 * V * H)
        f += (drafts - 1) * (n * (2.0 * attn + 4.0 * H * H + 2.0 * V * H) + keys * score + moe_flops(n))
        b += n * n_gdn * (4 * state + 2 * conv)  # the committed states
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case: dict) -> dict:
    # bf16 activations between kernels: two passes whose sums are ordered differently round differently, and a few rows
    # then take another eighth expert. Against 64 bits the hidden states are off by 0.007 to 0.014 (norm), and a row that
    # took another expert by a good part of a standard deviation at single elements.
    return {"rel": 0.03, "max": 0.9, "differ": 0.01}


# ------------------------------------------------------------------ inputs
def _normal(gen, shape, std: float, dtype=torch.bfloat16) -> torch.Tensor:
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=gen)


def _layer(cfg: ModelConfig, kind: str, gen) -> LayerWeights:
    H, E, inter = cfg.hidden_size, cfg.num_experts + 1, cfg.moe_intermediate_size
    if kind == "linear_attention":
        nv = cfg.linear_num_value_heads
        # decay rates and time steps over the ranges such layers are initialised with: memories of tens to thousands of rows
        a = torch.empty(nv, device=DEV).uniform_(1.0, 16.0, generator=gen)
        dt = torch.exp(torch.empty(nv, device=DEV).uniform_(math.log(1e-3), math.log(1e-1), generator=gen))
        mixer = dict(in_proj=_normal(gen, (cfg.gdn_in_rows, H), 0.02), out_proj=_normal(gen, (H, cfg.gdn_value_dim), 0.02),
                     conv_w=_normal(gen, (cfg.gdn_conv_dim, cfg.linear_conv_kernel_dim), 0.4), A_log=torch.log(a),
                     dt_bias=torch.log(torch.expm1(dt)), gnorm_w=1.0 + _normal(gen, (cfg.linear_value_head_dim,), 0.1))
    else:
        mixer = dict(in_proj=_normal(gen, (cfg.attn_q_rows + 2 * cfg.attn_kv_rows, H), 0.02),
                     out_proj=_normal(gen, (H, cfg.num_attention_heads * cfg.head_dim), 0.02),
                     q_norm=_normal(gen, (cfg.head_dim,), 0.1), k_norm=_normal(gen, (cfg.head_dim,), 0.1))
    return LayerWeights(kind=kind, input_norm=_normal(gen, (H,), 0.1), post_norm=_normal(gen, (H,), 0.1), **mixer,
                        router=_normal(gen, (E, H), 0.04), w_gate_up=_normal(gen, (E, 2 * inter, H), 0.02),
                        w_down=_normal(gen, (E, H, inter), 0.02), shared_merged=True)


def _weights(cfg: ModelConfig, gen) -> Weights:
    """Random weights of the architecture whose head is as decided as a trained model's: token ``t`` predicts ``t + 1``."""
    H = cfg.hidden_size
    embed = _normal(gen, (cfg.vocab_size, H), 1.0)
    layers = [_layer(cfg, kind, gen) for kind in cfg.layer_types]
    lm_head = _normal(gen, (cfg.vocab_size, H), 0.02).add_(torch.roll(embed, 1, 0), alpha=0.02)
    mtp = None
    if cfg.mtp_num_hidden_layers:
        fc = _normal(gen, (H, 2 * H), 0.01)
        fc[:, :H].add_(torch.eye(H, dtype=fc.dtype, device=DEV))
        mtp = MTPWeights(fc=fc, pre_fc_norm_embedding=_normal(gen, (H,), 0.1), pre_fc_norm_hidden=_normal(gen, (H,), 0.1),
                         norm=_normal(gen, (H,), 0.1), layer=_layer(cfg, "full_attention", gen))
    return Weights(cfg, embed, lm_head, _normal(gen, (H,), 0.1), layers, mtp)


def _tokens(case: dict, cfg: ModelConfig, seed: int, rows: list[int]) -> list[list[int]]:
    """Uniform-random tokens; in a speculative step, the first drafts of a sequence are the ones the model will pick."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for i, n in enumerate(rows):
        t = torch.randint(0, cfg.vocab_size, (n,), generator=gen).tolist()
        if case["kind"] == "verify":
            for j in range(1, 1 + i % n):
                t[j] = (t[j - 1] + 1) % cfg.vocab_size
        out.append(t)
    return out


def _inputs(case: dict, seed: int) -> dict:
    cfg, (rows, pos0) = _config(case), _spans(case)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    weights = _weights(cfg, gen)
    n = len(rows)
    drafts = case.get("drafts", 0)
    pages = [(p + r + drafts + PAGE_SIZE - 1) // PAGE_SIZE for p, r in zip(pos0, rows)]
    total = sum(pages)
    ids = torch.randperm(total, generator=torch.Generator().manual_seed(seed + 1), dtype=torch.int64) + 1  # page 0 is scratch
    table = torch.zeros(n, _width(case, max(pages)), dtype=torch.int32)
    at = 0
    for i, k in enumerate(pages):
        table[i, :k] = ids[at:at + k].int()
        at += k
    kv = _normal(gen, (cfg.num_kv_layers, total + 1, 2, cfg.num_key_value_heads, PAGE_SIZE, cfg.head_dim), 1.0)
    nv, dk, dv = cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
    rec = _normal(gen, (len(cfg.gdn_layers), n + 1, nv, dk, dv), 0.05, torch.float32)
    conv = _normal(gen, (len(cfg.gdn_layers), n + 1, cfg.gdn_conv_dim, cfg.linear_conv_kernel_dim - 1), 1.0)
    return {"cfg": cfg, "weights": weights, "rows": rows, "pos0": pos0, "table": table, "kv": kv, "rec": rec, "conv": conv,
            "tokens": _tokens(case, cfg, seed + 2, rows), "slots": list(range(1, n + 1)), "pages": total + 1}


def prepare(case: dict, seed: int) -> dict:
    """A loaded model with its caches in the middle of serving the case's requests, and the captured step."""
    x = _inputs(case, seed)
    cuda_ops.pack_weights(x["weights"])
    n = len(x["rows"])
    model = Model(x["weights"], x["pages"], n + 1, ops=cuda_ops)
    s = {"case": case, "model": model, "tokens": x["tokens"], "slots": x["slots"], "pos0": x["pos0"], "table": x["table"]}
    starts = [sum(x["rows"][:i]) for i in range(n + 1)]
    if case["kind"] == "prefill":
        s["last"] = torch.tensor([a - 1 for a in starts[1:]], device=DEV)
        s["fresh"] = [slot for slot, p in zip(x["slots"], x["pos0"]) if p == 0]
    else:
        G = x["rows"][0]
        tokens = [t for ts in x["tokens"] for t in ts]
        positions = [p + j for p in x["pos0"] for j in range(G)]
        s["host"] = torch.tensor([tokens, positions], dtype=torch.int64).pin_memory()
        s["dev"] = s["host"].to(DEV)
        s["batch"] = PackedBatch.uniform(s["dev"][0], s["dev"][1], x["slots"], x["table"], G, DEV)
        s["batch"].tokens, s["batch"].positions = s["dev"][0], s["dev"][1]
        if case["kind"] == "verify":
            s["ring"] = model.new_ring(n, G)
            s["valid"] = torch.full((n,), case["drafts"], dtype=torch.int32, device=DEV)
            s["seq1"] = torch.arange(n, dtype=torch.int32, device=DEV)
        _step(s)  # first use of the kernels stays outside the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["out"] = _step(s)
        s["graph"] = graph
    # the caches as the requests left them (the warm-up step above wrote to them)
    for name, mine in (("kv", model.kv), ("rec", model.rec_state), ("conv", model.conv_state)):
        mine.copy_(x[name])
    return s


def _head(s: dict, hidden: torch.Tensor) -> torch.Tensor:
    return s["model"].logits(hidden) if s["case"]["head"] == "logits" else s["model"].greedy(hidden)


def _step(s: dict) -> dict:
    """A decode step, or a speculative step: verify, MTP block, accepted prefix, draft chain, state commit."""
    m, batch = s["model"], s["batch"]
    if s["case"]["kind"] == "decode":
        hidden = m.forward(batch)
        return {"hidden": hidden, "head": _head(s, hidden)}
    drafts = s["case"]["drafts"]
    hidden = m.forward(batch, ring=s["ring"])
    picks = m.greedy(hidden)
    y = m.mtp_forward(hidden, picks, batch)
    accepted, h, link_pos = m.ops.chain_accept(batch.tokens, picks, s["valid"], batch.positions, y, batch.G, drafts - 1)
    chain, ys = [m.draft_pick(h)], []
    for j in range(1, drafts):
        link = PackedBatch(chain[-1], link_pos[j - 1], s["seq1"], batch.slots, batch.block_tables, 1)
        h = m.mtp_forward(h, chain[-1], link)
        ys.append(h)
        chain.append(m.draft_pick(h))
    m.commit_ring(s["ring"], batch.slots, accepted)
    return {"hidden": hidden, "head": picks, "mtp": y, "links": ys, "accepted": accepted, "drafts": chain}


def run(s: dict) -> dict:
    m = s["model"]
    if s["case"]["kind"] == "prefill":
        for slot in s["fresh"]:  # a new request starts from an empty state
            m.reset_slot(slot)
        batch = PackedBatch.prefill(s["tokens"], s["slots"], s["pos0"], s["table"], DEV)
        hidden = m.forward(batch)
        out = {"hidden": hidden, "head": _head(s, hidden[s["last"]])}
    else:
        s["dev"].copy_(s["host"], non_blocking=True)
        s["graph"].replay()
        out = dict(s["out"])
    out.update(kv=m.kv, rec=m.rec_state, conv=m.conv_state)
    return out


# ------------------------------------------------------------------ the same pass in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * (1.0 + w.double())


def _mm(x, w):
    return x @ w.double().t()


class _Rows:
    """Packed rows in 64 bits: row ``r`` belongs to sequence ``seq[r]`` at position ``pos[r]``."""

    def __init__(self, x: dict, rows: list[int], pos: torch.Tensor) -> None:
        self.rows, self.pos = rows, pos
        self.starts = [sum(rows[:i]) for i in range(len(rows) + 1)]
        self.seq = torch.repeat_interleave(torch.arange(len(rows)), torch.tensor(rows)).to(DEV)
        self.table = x["table"].to(DEV).long()


def _moe64(cfg, lw, h):
    logits = _mm(h, lw.router)
    E, I = cfg.num_experts, cfg.moe_intermediate_size
    top, idx = torch.softmax(logits[:, :E], -1).topk(cfg.num_experts_per_tok, -1)
    out = torch.zeros_like(h)
    wts = torch.cat([top / top.sum(-1, keepdim=True), torch.sigmoid(logits[:, E:])], -1)
    idx = torch.cat([idx, torch.full_like(idx[:, :1], E)], -1)
    for e in torch.unique(idx).tolist():
        r, j = (idx == e).nonzero(as_tuple=True)
        gu = _mm(h[r], lw.w_gate_up[e])
        out.index_add_(0, r, _mm(F.silu(gu[:, :I]) * gu[:, I:], lw.w_down[e]) * wts[r, j][:, None])
    return out


def _attention64(cfg, lw, kv, h, b: _Rows):
    D, nq, nkv = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    T = h.shape[0]
    qkv = _mm(h, lw.in_proj)
    qg = qkv[:, : 2 * nq * D].view(T, nq, 2 * D)
    q, gate = qg[..., :D], qg[..., D:]
    k, v = (qkv[:, 2 * nq * D + i * nkv * D:2 * nq * D + (i + 1) * nkv * D].view(T, nkv, D) for i in (0, 1))
    half = cfg.rotary_dim // 2
    inv = cfg.rope_theta ** (-torch.arange(half, dtype=torch.float64, device=DEV) * 2 / cfg.rotary_dim)
    ang = b.pos.double()[:, None, None] * inv

    def rope(t, w):
        t = _norm(t, w, cfg.rms_norm_eps)
        a, c = t[..., :half], t[..., half:2 * half]
        return torch.cat([a * ang.cos() - c * ang.sin(), c * ang.cos() + a * ang.sin(), t[..., 2 * half:]], -1)

    q, k = rope(q, lw.q_norm), rope(k, lw.k_norm)
    page, at = b.table[b.seq, b.pos // PAGE_SIZE], b.pos % PAGE_SIZE
    kv[page, 0, :, at], kv[page, 1, :, at] = k, v
    out = torch.empty_like(q)
    for i in range(len(b.rows)):
        r0, r1 = b.starts[i], b.starts[i + 1]
        n_keys = int(b.pos[r1 - 1]) + 1
        pages = kv[b.table[i, : -(-n_keys // PAGE_SIZE)]]
        ks, vs = (pages[:, j].transpose(0, 1).reshape(nkv, -1, D)[:, :n_keys] for j in (0, 1))
        for c0 in range(r0, r1, 512):  # bounds the score matrix
            c1 = min(r1, c0 + 512)
            qs = q[c0:c1].view(c1 - c0, nkv, nq // nkv, D).permute(1, 2, 0, 3)
            sc = qs @ ks[:, None].transpose(-1, -2) * D ** -0.5
            sc = sc.masked_fill(torch.arange(n_keys, device=DEV) > b.pos[c0:c1, None], -math.inf)
            out[c0:c1] = (torch.softmax(sc, -1) @ vs[:, None]).permute(2, 0, 1, 3).reshape(c1 - c0, nq, D)
    return _mm((out * torch.sigmoid(gate)).reshape(T, nq * D), lw.out_proj)


def _gdn64(cfg, lw, rec, conv, h, b: _Rows, keep):
    """Row by row over all sequences at once; ``keep[i]``: the row of sequence ``i`` whose state stays behind."""
    nk, nv, dk, dv = (cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim,
                      cfg.linear_value_head_dim)
    C = cfg.gdn_conv_dim
    mixed = _mm(h, lw.in_proj)
    z = mixed[:, C:C + nv * dv].view(-1, nv, dv)
    beta = torch.sigmoid(mixed[:, C + nv * dv:C + nv * dv + nv])
    decay = torch.exp(-lw.A_log.double().exp() * F.softplus(mixed[:, C + nv * dv + nv:] + lw.dt_bias.double()))
    w = lw.conv_w.double()
    out = torch.zeros(h.shape[0], nv, dv, dtype=torch.float64, device=DEV)
    S, win = rec[1:].clone(), conv[1:].clone()
    n_rows = torch.tensor(b.rows)
    for j in range(max(b.rows)):
        live = (n_rows > j).nonzero().flatten().to(DEV)
        r = torch.tensor(b.starts[:-1], device=DEV)[live] + j
        full = torch.cat([win[live], mixed[r, :C, None]], -1)
        x = F.silu((full * w).sum(-1))
        win[live] = full[..., 1:]
        q, k = (x[:, i * nk * dk:(i + 1) * nk * dk].view(-1, nk, dk) for i in (0, 1))
        q, k = (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(nv // nk, 1) for t in (q * dk ** -0.5, k))
        v = x[:, 2 * nk * dk:].view(-1, nv, dv)
        s = S[live] * decay[r][..., None, None]
        delta = (v - (k[:, :, None] @ s)[:, :, 0]) * beta[r][..., None]
        s += k[..., None] * delta[:, :, None]
        out[r] = (q[:, :, None] @ s)[:, :, 0]
        S[live] = s
        done = (keep[live] == j).nonzero().flatten()
        rec[1 + live[done]], conv[1 + live[done]] = s[done], full[done][..., 1:]
    o = out * torch.rsqrt(out.pow(2).mean(-1, keepdim=True) + cfg.rms_norm_eps) * lw.gnorm_w.double() * F.silu(z)
    return _mm(o.reshape(-1, nv * dv), lw.out_proj)


def _mtp64(x, kv, hidden, nxt, b: _Rows):
    cfg, w, m = x["cfg"], x["weights"], x["weights"].mtp
    eps = cfg.rms_norm_eps
    res = _mm(torch.cat([_norm(w.embed[nxt].double(), m.pre_fc_norm_embedding, eps),
                         _norm(hidden, m.pre_fc_norm_hidden, eps)], -1), m.fc)
    res = res + _attention64(cfg, m.layer, kv, _norm(res, m.layer.input_norm, eps), b)
    res = res + _moe64(cfg, m.layer, _norm(res, m.layer.post_norm, eps))
    return _norm(res, m.norm, eps)


def _logits64(x, h):
    head = x["weights"].lm_head
    return torch.cat([_mm(h, head[i:i + 32768]) for i in range(0, head.shape[0], 32768)], -1)


def exact(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    cfg, w, rows = x["cfg"], x["weights"], x["rows"]
    n, eps = len(rows), cfg.rms_norm_eps
    kv, rec, conv = x["kv"].double(), x["rec"].double(), x["conv"].double()
    for i, p in enumerate(x["pos0"]):
        if case["kind"] == "prefill" and p == 0:
            rec[:, 1 + i], conv[:, 1 + i] = 0.0, 0.0
    pos = torch.tensor([p + j for p, r in zip(x["pos0"], rows) for j in range(r)], device=DEV)
    b = _Rows(x, rows, pos)
    tokens = torch.tensor([t for ts in x["tokens"] for t in ts], device=DEV)
    keep = torch.tensor([r - 1 for r in rows], device=DEV)
    if case["kind"] == "verify":  # the head predicts t + 1: a draft is accepted where it is that
        keep = torch.tensor([next((j for j in range(r - 1) if t[j + 1] != (t[j] + 1) % cfg.vocab_size), r - 1)
                             for t, r in zip(x["tokens"], rows)], device=DEV)
    res = w.embed[tokens].double()
    gi = ai = 0
    for lw in w.layers:
        h = _norm(res, lw.input_norm, eps)
        if lw.kind == "linear_attention":
            res = res + _gdn64(cfg, lw, rec[gi], conv[gi], h, b, keep)
            gi += 1
        else:
            res = res + _attention64(cfg, lw, kv[ai], h, b)
            ai += 1
        res = res + _moe64(cfg, lw, _norm(res, lw.post_norm, eps))
    hidden = _norm(res, w.final_norm, eps)
    last = torch.tensor(b.starts[1:], device=DEV) - 1
    top = hidden if case["kind"] != "prefill" else hidden[last]
    logits = _logits64(x, top)
    out = {"hidden": hidden, "head": logits if case["head"] == "logits" else logits.argmax(-1)}
    if case["kind"] == "verify":
        y = _mtp64(x, kv[ai], hidden, out["head"], b)
        at = torch.tensor(b.starts[:-1], device=DEV) + keep
        h, p = y[at], pos[at]
        chain, ys = [_logits64(x, h).argmax(-1)], []
        for _ in range(1, case["drafts"]):
            p = p + 1
            h = _mtp64(x, kv[ai], h, chain[-1], _Rows(x, [1] * n, p))
            ys.append(h)
            chain.append(_logits64(x, h).argmax(-1))
        out.update(mtp=y, links=ys, accepted=keep, drafts=chain)
    out.update(kv=kv, rec=rec, conv=conv)
    return out
