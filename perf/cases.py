"""What a user of this package has it do, as sizes that can be timed: decode steps, prefill batches and the
preparation of a decode step's metadata, through the package's public entry points.

Every case is one call pattern of the serving engine the layer belongs to:

  decode        one layer of an eager decode step: Attention.forward (cache store, then paged attention)
  decode_graph  the attention of a whole decode step as the engine replays it: `layers` layers of the fused producer
                (QK-norm, rotary embedding, store) and paged attention, captured once into a CUDA graph
  prefill       one layer of a prefill step, always eager in the engine: Attention.forward, or the fused producer and
                the attention behind it (`fused`); with `prefix` part of every other sequence is already in the cache
                and all keys come from there through the block tables
  metadata      the host side of a decode step: scheduler state -> pinned record -> device -> graph buffers

Lengths are spread evenly over [lo, hi] (so the work of a case is known), their order, the block tables and all
values come from the seed.  The cache has 256-token blocks scattered at random, bf16 throughout.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nanovllm_b200
from nanovllm_b200.engine.decode_metadata import DecodeMetadataStager
from nanovllm_b200.layers.qk_norm_rope import qk_norm_rope_store
from nanovllm_b200.utils.context import reset_context, set_context

BLOCK = 256
D = 128                      # head dimension of every supported model
MAX_POSITION = 40960         # rows of the rotary table, as the model's configuration has it
EPS = 1e-6
# (query heads, kv heads) of one GPU: Qwen3-0.6B and Qwen3-8B geometry at tensor parallelism 1, 2, 4, 8
HEADS = ((16, 8), (8, 4), (4, 2), (2, 1), (32, 8), (16, 4), (8, 2), (4, 1))


def listed():
    return [
        # a single request being served: the smallest call there is, eager (enforce_eager) and as the engine's graph
        dict(name="decode_one", kind="decode", H=16, Hkv=8, batch=1, lo=562, hi=562),
        dict(name="decode_one_graph", kind="decode_graph", H=16, Hkv=8, batch=1, lo=562, hi=562, layers=28),
        # a lightly loaded server: an odd number of chats, prompts and answers of 100 to 1024 tokens
        dict(name="decode_chat_graph", kind="decode_graph", H=16, Hkv=8, batch=37, lo=100, hi=1024, layers=28),
        # a busy server (the headline benchmark's decode shape), and one GPU's part of it under 8-way tensor parallelism
        dict(name="decode_busy", kind="decode", H=16, Hkv=8, batch=256, lo=100, hi=2048),
        dict(name="decode_busy_tp8_graph", kind="decode_graph", H=2, Hkv=1, batch=256, lo=100, hi=2048, layers=28),
        # the largest decode: the 8B geometry, full batch, long contexts
        dict(name="decode_8b", kind="decode", H=32, Hkv=8, batch=512, lo=512, hi=8192),
        # one short prompt arriving at an idle server
        dict(name="prefill_one", kind="prefill", H=16, Hkv=8, batch=1, lo=137, hi=137, fused=False, prefix=False),
        # what fits the engine's limit of 16384 tokens per prefill step, through the fused producer
        dict(name="prefill_step", kind="prefill", H=16, Hkv=8, batch=29, lo=100, hi=1024, fused=True, prefix=False),
        # the prefill benchmark's batch, dense and with cached prefixes
        dict(name="prefill_many", kind="prefill", H=16, Hkv=8, batch=256, lo=100, hi=1024, fused=False, prefix=False),
        dict(name="prefill_prefix", kind="prefill", H=16, Hkv=8, batch=256, lo=100, hi=1024, fused=False, prefix=True),
        # long documents on the 8B geometry: the largest attention
        dict(name="prefill_long", kind="prefill", H=32, Hkv=8, batch=4, lo=8192, hi=8192, fused=False, prefix=False),
        # what the host does in front of every decode step of the busy server
        dict(name="metadata_busy", kind="metadata", batch=256, lo=100, hi=2048),
    ]


def draw(rng):
    def logint(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    def span(most):
        a, b = logint(1, most), logint(16, most)
        return min(a, b), max(a, b)

    kind = rng.choice(("decode", "decode", "decode_graph", "decode_graph", "prefill", "prefill", "prefill", "metadata"))
    if kind == "metadata":
        lo, hi = span(4096)
        return dict(kind=kind, batch=logint(1, 512), lo=lo, hi=hi)
    h, hkv = rng.choice(HEADS)
    if kind == "prefill":
        case = dict(kind=kind, H=h, Hkv=hkv, batch=logint(1, 256))
        case["lo"], case["hi"] = span(8192)
        case["fused"], case["prefix"] = rng.random() < 0.4, rng.random() < 0.35
        while sum(lengths(case)) > 147456 or work(case)["flops"] > 2.19e12:
            case["batch"] = max(1, case["batch"] * 2 // 3)
        return case
    case = dict(kind=kind, H=h, Hkv=hkv, batch=logint(1, 512))
    case["lo"], case["hi"] = span(8192)
    if kind == "decode_graph":
        case["layers"] = 28 if h == 2 * hkv else 36
    while work(case)["bytes"] > (8e9 if kind == "decode" else 4e9):
        case["batch"] = max(1, case["batch"] * 2 // 3)
    return case


# ---- sizes ---------------------------------------------------------------------------------------------------
def lengths(case):
    """Context lengths, spread evenly over [lo, hi]."""
    n, lo, hi = case["batch"], case["lo"], case["hi"]
    return [lo + int((hi - lo) * (i + 0.5) / n + 0.5) for i in range(n)]


def prefixes(case, lens):
    """Cached tokens in front of every sequence: whole blocks, at least one token left to compute."""
    return [BLOCK * (i % ((n - 1) // BLOCK + 1)) if case["prefix"] and i % 2 else 0 for i, n in enumerate(lens)]


def work(case):
    """Bytes and operations of one pass that no implementation can do without."""
    lens = lengths(case)
    n = case["batch"]
    if case["kind"] == "metadata":
        width = -(-max(lens) // BLOCK)
        return {"bytes": 2 * (24 * n + 4 * n * width), "flops": 0}
    h, hkv = case["H"], case["Hkv"]
    kv_row, q_row = 2 * hkv * D * 2, h * D * 2          # bytes of a token's K and V, of its query heads
    if case["kind"] == "prefill":
        pre = prefixes(case, lens)
        new = sum(lens) - sum(pre)
        pairs = sum((k - p) * p + (k - p) * (k - p + 1) // 2 for k, p in zip(lens, pre))
        # new q, k, v read; output and cache rows written; cached prefixes read
        return {"bytes": new * (2 * q_row + 2 * kv_row) + sum(pre) * kv_row, "flops": 4 * D * h * pairs}
    # every cached token's K and V read, the new one's read from the step's input and written; q read, output written
    layer = sum(lens) * kv_row + n * kv_row + 2 * n * q_row
    layers = case.get("layers", 1)
    return {"bytes": layers * layer, "flops": layers * 4 * D * h * sum(lens)}


def tolerance(case):
    """Attention in bf16 with fp32 sums: outputs are rounded to 8 bits, and so are the probabilities."""
    return "exact" if case["kind"] == "metadata" else {"rel": 1e-2, "max": 0.1}


# ---- inputs --------------------------------------------------------------------------------------------------
class Sequence:
    """What the scheduler hands the model runner: the fields of nano-vllm's Sequence that a decode step reads."""

    def __init__(self, length, block_table, last_token):
        self.length, self.block_table, self.last_token = length, block_table, last_token

    def __len__(self):
        return self.length


def tables(lens, rng):
    """Block tables (rows padded with -1) over blocks scattered at random, and the number of blocks."""
    nblk = [-(-n // BLOCK) for n in lens]
    blocks = sum(nblk) + 8
    perm = rng.permutation(blocks).astype(np.int32)
    bt = np.full((len(lens), max(nblk)), -1, dtype=np.int32)
    at = 0
    for i, k in enumerate(nblk):
        bt[i, :k] = perm[at:at + k]
        at += k
    return bt, blocks


def slots(bt, row, token):
    return (bt[row, token // BLOCK] * BLOCK + token % BLOCK).astype(np.int32)


def rotary_table(dev):
    freq = 1.0 / (1e6 ** (torch.arange(0, D, 2, dtype=torch.float, device=dev) / D))
    angle = torch.arange(MAX_POSITION, dtype=torch.float, device=dev)[:, None] * freq
    return torch.cat((angle.cos(), angle.sin()), dim=-1).unsqueeze_(1)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    n, lens = case["batch"], lengths(case)
    order = rng.permutation(n)
    pre = prefixes(case, lens) if case["kind"] == "prefill" else [0] * n
    lens, pre = [lens[i] for i in order], [pre[i] for i in order]
    bt, blocks = tables(lens, rng)
    dev = torch.device("cuda")
    if case["kind"] == "metadata":
        return prepare_metadata(lens, bt, rng, dev)

    h, hkv = case["H"], case["Hkv"]
    gen = torch.Generator(device=dev).manual_seed(seed)
    normal = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=dev).normal_(generator=gen)  # noqa: E731
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    layers = case.get("layers", 1)
    s = dict(case=case, kv_cache=normal(2, layers, blocks, BLOCK, hkv, D).mul_(0.5))
    s["layers"] = []
    for i in range(layers):
        att = nanovllm_b200.Attention(h, D, D ** -0.5, hkv)
        att.k_cache, att.v_cache = s["kv_cache"][0, i], s["kv_cache"][1, i]
        s["layers"].append(att)
    lens_np, pre_np = np.array(lens), np.array(pre)
    rows = np.arange(n)
    if case["kind"] == "prefill":
        new = lens_np - pre_np
        tokens = int(new.sum())
        row = np.repeat(rows, new)
        pos = np.arange(tokens) - np.repeat(np.cumsum(new) - new, new) + np.repeat(pre_np, new)
        cu = lambda a: to(np.concatenate([[0], np.cumsum(a)]).astype(np.int32))  # noqa: E731
        s["context"] = dict(is_prefill=True, cu_seqlens_q=cu(new), cu_seqlens_k=cu(lens_np), max_seqlen_q=int(new.max()),
                            max_seqlen_k=int(lens_np.max()), slot_mapping=to(slots(bt, row, pos)),
                            block_tables=to(bt) if case["prefix"] else None)
    else:
        tokens, pos = n, lens_np - 1
        s["context"] = dict(is_prefill=False, slot_mapping=to(slots(bt, rows, pos)), context_lens=to(lens_np.astype(np.int32)),
                            block_tables=to(bt))
    # the fused projection's rows; q and k are what the rotary embedding returns (contiguous), v stays a view of the row
    qkv = normal(layers, tokens, (h + 2 * hkv) * D)
    if case["kind"] == "decode_graph" or case.get("fused"):
        s.update(qkv=qkv, positions=to(pos.astype(np.int64)), table=rotary_table(dev), q_weight=normal(D).mul_(0.1).add_(1.0),
                 k_weight=normal(D).mul_(0.1).add_(1.0))
    else:
        q, k, v = qkv[0].mul_(0.5 if case["kind"] == "decode" else 1.0).split([h * D, hkv * D, hkv * D], dim=-1)
        s.update(q=q.reshape(tokens, h, D).contiguous(), k=k.reshape(tokens, hkv, D).contiguous(), v=v.view(tokens, hkv, D))
    if case["kind"] == "decode_graph":
        # as the engine captures a batch size: one eager pass, then the capture; replays write the same output buffers
        set_context(**s["context"])
        with torch.inference_mode():
            fused_layer(s, 0)
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["out"] = [fused_layer(s, i) for i in range(layers)]
        reset_context()
    return s


def prepare_metadata(lens, bt, rng, dev):
    tokens = rng.integers(0, 151936, len(lens))
    seqs = [Sequence(n, [int(b) for b in bt[i, :-(-n // BLOCK)]], int(tokens[i])) for i, n in enumerate(lens)]
    rows, cols = 512, 16
    ints = lambda *shape: torch.zeros(shape, dtype=torch.int32, device=dev)  # noqa: E731
    wide = lambda: torch.zeros(rows, dtype=torch.int64, device=dev)  # noqa: E731
    buffers = dict(input_ids=wide(), positions=wide(), slot_mapping=ints(rows), context_lens=ints(rows),
                   block_tables=ints(rows, cols))
    return dict(case=dict(kind="metadata"), seqs=seqs, stager=DecodeMetadataStager(rows, cols, BLOCK, dev), buffers=buffers)


def fused_layer(s, i):
    att = s["layers"][i]
    q, k, v = qk_norm_rope_store(s["qkv"][i], s["positions"], s["q_weight"], s["k_weight"], s["table"], EPS, att.num_heads,
                                 att.num_kv_heads, att.k_cache, att.v_cache, s["context"]["slot_mapping"])
    return att.forward(q, k, v, already_stored=True)


# ---- one pass ------------------------------------------------------------------------------------------------
def run(s):
    kind = s["case"]["kind"]
    if kind == "metadata":
        stager, b = s["stager"], s["buffers"]
        stager.pack(s["seqs"])
        stager.unpack_into(stager.to_device(), b["input_ids"], b["positions"], b["slot_mapping"], b["context_lens"],
                           b["block_tables"])
        return b
    if kind == "decode_graph":
        s["graph"].replay()
        out = s["out"]
    else:
        set_context(**s["context"])
        if s["case"].get("fused"):
            out = fused_layer(s, 0)
        else:
            out = s["layers"][0](s["q"], s["k"], s["v"])
        reset_context()
    return {"out": out, "kv_cache": s["kv_cache"]}
