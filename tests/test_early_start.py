"""What the kernels read while the kernel in front of them still runs.  GPU: a kernel that lets its dependents start early
(griddepcontrol.launch_dependents) and writes its arrays only afterwards stands in front of every call; the call must see what
it wrote.  The same call on the same values with nothing running is the reference, bit for bit."""
import os
import re

import pytest
import torch

from workloads import cu_seqlens, decode_slots, default_scale, make_block_tables

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanovllm_b200", "csrc")
DEV = "cuda:0"
DELAY = 200_000                  # cycles between the early trigger and the writes (0.1 ms)
SOURCE = r"""
extern "C" __global__ void late_copy(const int* src, int* dst, int words, int cycles) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long t0 = clock64();
  while (clock64() - t0 < cycles) {}
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}
"""


def test_rows_are_not_read_through_the_read_only_path():
    """__ldg and const __restrict__ let the compiler move a load ahead of griddepcontrol.wait (and the hardware serve it from a
    cache that nobody invalidates): in kernels that start early only for arrays that no kernel in front may write."""
    early = [f for f in sorted(os.listdir(CSRC)) if "griddepcontrol" in open(os.path.join(CSRC, f)).read()]
    assert len(early) >= 5
    for f in early + ["decode_common.cuh"]:
        code = re.sub(r"//.*", "", open(os.path.join(CSRC, f)).read())
        assert "__restrict__" not in code, f
        for arg in re.findall(r"__ldg\((.{20})", code):
            allowed = ("p.cu_q", "p.cu_k") if f == "prefill_attn_tc2.cu" else ("p.st_slots",) if f == "decode_attn.cu" else ()
            assert arg.startswith(allowed) if allowed else False, (f, arg)


@pytest.fixture(scope="module")
def late_copy():
    kernel = torch.cuda._compile_kernel(SOURCE, "late_copy")
    return lambda src, dst: kernel(grid=(1, 1, 1), block=(1024, 1, 1), args=[src, dst, src.numel(), DELAY])


def _packed(tensors):
    """The tensors in one buffer of 32-bit words on the device (each at a multiple of 16 bytes), and views of them in it."""
    sizes = [-(-t.numel() * t.element_size() // 16) * 4 for t in tensors.values()]
    buf = torch.zeros(sum(sizes), dtype=torch.int32, device=DEV)
    views, at = {}, 0
    for (name, t), size in zip(tensors.items(), sizes):
        words = t.numel() * t.element_size() // 4
        views[name] = buf[at:at + words].view(t.dtype).view(t.shape)
        views[name].copy_(t)
        at += size
    return buf, views


def _compare(late_copy, before, after, prepare, call):
    """call(views, state) -> the tensors it wrote: with `after` in place and nothing running, and with `before` in place until a
    kernel that is still running when the call's kernel starts puts `after` there.  `state` is made ahead of that kernel, so
    that nothing is launched between it and the call's."""
    with torch.inference_mode():
        quiet, views = _packed(after)
        state = prepare()
        torch.cuda.synchronize()
        want = call(views, state)
        for _ in range(3):
            buf, views = _packed(before)
            state = prepare()
            torch.cuda.synchronize()
            late_copy(quiet, buf)
            got = call(views, state)
            torch.cuda.synchronize()
            assert torch.equal(buf, quiet) and len(got) == len(want)
            for a, b in zip(got, want):
                assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def _rows(seed, **shapes):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return {k: torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for k, s in shapes.items()}


def _caches(blocks, hkv):
    return lambda: tuple(torch.zeros(blocks, 256, hkv, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2))


def _layer(h, hkv, caches, call, **context):
    import nanovllm_b200
    from nanovllm_b200.utils.context import reset_context, set_context
    att = nanovllm_b200.Attention(h, 128, default_scale(128), hkv)
    att.k_cache, att.v_cache = caches
    set_context(**context)
    out = call(att)
    reset_context()
    return (out, *caches)


@pytest.mark.gpu
@pytest.mark.parametrize("n,hkv", [(1, 8), (7, 1), (256, 8), (20000, 8)])                  # the last: two passes
def test_store_behind_a_kernel_that_writes_its_rows(late_copy, n, hkv):
    import nanovllm_b200
    slots = torch.arange(n, dtype=torch.int32, device=DEV).flip(0)
    shape = dict(k=(n, hkv, 128), v=(n, hkv, 128))

    def call(m, caches):
        nanovllm_b200.store_kvcache(m["k"], m["v"], *caches, slots)
        return caches
    _compare(late_copy, _rows(1, **shape), _rows(2, **shape), _caches(n // 256 + 1, hkv), call)


def _slots(n, total, seed):
    """n slots of `total` in an order of their own, a fifth of them skipped."""
    g = torch.Generator().manual_seed(seed)
    s = torch.randperm(total, generator=g)[:n].to(torch.int32)
    s[torch.randperm(n, generator=g)[:n // 5]] = -1
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("n,hkv", [(1, 8), (7, 1), (256, 8), (3000, 2), (20000, 8)])
def test_store_behind_a_kernel_that_writes_its_slots(late_copy, n, hkv):
    import nanovllm_b200
    blocks = n // 256 + 2
    rows = _rows(1, k=(n, hkv, 128), v=(n, hkv, 128))

    def call(m, caches):
        nanovllm_b200.store_kvcache(rows["k"], rows["v"], *caches, m["slots"])
        return caches
    _compare(late_copy, dict(slots=_slots(n, blocks * 256, 2)), dict(slots=_slots(n, blocks * 256, 3)), _caches(blocks, hkv), call)


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,hkv", [(1, 16, 8), (3, 8, 8), (37, 16, 8), (200, 4, 2)])     # clusters, store inside, store in front
def test_layer_decode_behind_a_kernel_that_writes_its_rows(late_copy, n, h, hkv):
    g = torch.Generator().manual_seed(n)
    lens = torch.randint(1, 700, (n,), generator=g).tolist()
    bt, blocks = make_block_tables(lens, 256, g)
    ctx = dict(is_prefill=False, slot_mapping=decode_slots(lens, bt, 256).to(DEV), block_tables=bt.to(DEV),
               context_lens=torch.tensor(lens, dtype=torch.int32, device=DEV))
    shape = dict(q=(n, h, 128), k=(n, hkv, 128), v=(n, hkv, 128))
    _compare(late_copy, _rows(1, **shape), _rows(2, **shape), _caches(blocks, hkv),
             lambda m, caches: _layer(h, hkv, caches, lambda att: att(m["q"], m["k"], m["v"]), **ctx))


@pytest.mark.gpu
@pytest.mark.parametrize("h,hkv,lens", [(16, 8, [137]), (16, 8, [1, 63, 64, 65]), (5, 1, [100, 200]), (16, 8, [700, 31, 2000]),
                                        (2, 2, [900] * 40)])                               # mma.sync, tcgen05 in both forms
def test_layer_prefill_behind_a_kernel_that_writes_its_rows(late_copy, h, hkv, lens):
    n = sum(lens)
    cu = cu_seqlens(lens).to(DEV)
    ctx = dict(is_prefill=True, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens),
               slot_mapping=torch.arange(n, dtype=torch.int32, device=DEV))
    shape = dict(q=(n, h, 128), k=(n, hkv, 128), v=(n, hkv, 128))
    _compare(late_copy, _rows(1, **shape), _rows(2, **shape), _caches(n // 256 + 1, hkv),
             lambda m, caches: _layer(h, hkv, caches, lambda att: att(m["q"], m["k"], m["v"]), **ctx))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 37, 3000])                                               # one head a pass, four heads a pass
def test_producer_behind_a_kernel_that_writes_its_rows(late_copy, n):
    from nanovllm_b200.layers.qk_norm_rope import qk_norm_rope_store
    h, hkv = 16, 8
    w = _rows(3, q=(128,), k=(128,))
    table = torch.randn(4096, 1, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4))
    pos, slots = torch.arange(n, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    shape = dict(qkv=(n, (h + 2 * hkv) * 128))

    def call(m, caches):
        q, k, _ = qk_norm_rope_store(m["qkv"], pos, w["q"], w["k"], table, 1e-6, h, hkv, *caches, slots)
        return (q, k, *caches)
    _compare(late_copy, _rows(1, **shape), _rows(2, **shape), _caches(n // 256 + 1, hkv), call)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 4])                       # the table at a multiple of 32 bytes, and of 16 only
@pytest.mark.parametrize("n,h,hkv", [(1, 16, 8), (37, 16, 8), (256, 2, 1), (3000, 16, 8)])
def test_producer_behind_a_kernel_that_writes_everything_else(late_copy, n, h, hkv, shift):
    from nanovllm_b200.layers.qk_norm_rope import qk_norm_rope_store
    blocks = n // 256 + 2
    qkv = _rows(1, qkv=(n, (h + 2 * hkv) * 128))["qkv"]

    def metadata(seed):
        g = torch.Generator().manual_seed(seed)
        pos = torch.randint(0, 1000, (n,), generator=g)
        pos[::5] = torch.arange(0, n, 5) % 1000                  # some stay as they were
        return dict(pad=torch.zeros(4 + shift, dtype=torch.int32), table=torch.randn(1000, 1, 128, generator=g),
                    pos=pos, slots=_slots(n, blocks * 256, seed), **_rows(seed, q=(128,), k=(128,)))

    def call(m, caches):
        assert m["table"].data_ptr() % 32 == (4 + shift) * 4 % 32
        q, k, _ = qk_norm_rope_store(qkv, m["pos"], m["q"], m["k"], m["table"], 1e-6, h, hkv, *caches, m["slots"])
        return (q, k, *caches)
    _compare(late_copy, metadata(2), metadata(3), _caches(blocks, hkv), call)

@pytest.mark.gpu
@pytest.mark.parametrize("h,hkv,lq,paged", [(16, 8, [137], False), (16, 8, [60] * 8, False), (5, 1, [1, 200, 30, 0, 7], False),
                                            (16, 8, [33, 70, 1], True), (4, 2, [20] * 100, False)])
def test_mma_prefill_behind_a_kernel_that_writes_its_metadata(late_copy, h, hkv, lq, paged):
    """Before: other lengths of the same number of tokens, other slots, another block table."""
    import nanovllm_b200
    n = sum(lq)
    g = torch.Generator().manual_seed(n)
    before = list(reversed(lq)) if len(set(lq)) > 1 else [n - len(lq) + 1] + [1] * (len(lq) - 1)
    assert sum(before) == n
    rows = _rows(1, q=(n, h, 128), k=(n, hkv, 128), v=(n, hkv, 128))
    blocks = len(lq) * 2 + 2

    def metadata(lens, seed):
        m = dict(cu=cu_seqlens(lens), slots=_slots(n, blocks * 256, seed))
        if paged:
            m["bt"] = torch.randperm(blocks, generator=torch.Generator().manual_seed(seed))[:2 * len(lq)].to(torch.int32).view(-1, 2)
        return m

    def call(m, caches):
        if paged:
            return (nanovllm_b200.prefill_attention(rows["q"], *cache, m["cu"], m["cu"], n, n, default_scale(128), hkv, m["bt"], 1),)
        out = nanovllm_b200.prefill_attention(rows["q"], rows["k"], rows["v"], m["cu"], m["cu"], n, n, default_scale(128), hkv, None, 1)
        return (out, *caches)

    def layer(m, caches):
        return _layer(h, hkv, caches, lambda att: att(rows["q"], rows["k"], rows["v"]), is_prefill=True, cu_seqlens_q=m["cu"],
                      cu_seqlens_k=m["cu"], max_seqlen_q=n, max_seqlen_k=n, slot_mapping=m["slots"])
    cache = tuple(torch.randn(blocks, 256, hkv, 128, device=DEV).to(torch.bfloat16) for _ in range(2))
    for f in (call, layer) if n < 500 and not paged else (call,):          # (the layer takes the other kernel for more)
        _compare(late_copy, metadata(before, 2), metadata(lq, 3), _caches(blocks, hkv), f)


@pytest.mark.gpu
@pytest.mark.parametrize("bucket,bs,h,hkv", [(4, 3, 16, 8), (48, 37, 16, 8), (64, 64, 2, 1)])     # a cluster per pair, whole pairs
def test_graph_of_unpack_producer_and_decode_on_changing_metadata(bucket, bs, h, hkv):
    """A decode step as one graph, two layers: the record's unpack, then producer and attention of each layer, which start early one
    behind the other.  Positions, slots, lengths and tables change with every replay; the same calls with a
    synchronisation behind each are the reference, bit for bit, and the oracles within their tolerances."""
    import random
    import nanovllm_b200
    from nanovllm_b200.engine.decode_metadata import DecodeMetadataStager
    from nanovllm_b200.layers.qk_norm_rope import qk_norm_rope_store
    from nanovllm_b200.utils.context import reset_context, set_context
    from oracle.attention_oracle import decode_attn_ref
    from oracle.metadata_oracle import prepare_decode_ref
    from oracle.qk_norm_rope_oracle import qk_norm_rope_ref, rope_cos_sin_cache
    from test_decode_metadata import FakeSeq, _fake_batch
    from test_qk_norm_rope import _one_step
    cols, blocks, layers = 8, 600, 2
    ints = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype, device=DEV)  # noqa: E731
    gv = dict(input_ids=ints(bucket, dtype=torch.int64), positions=ints(bucket, dtype=torch.int64), slot_mapping=ints(bucket) - 1,
              context_lens=ints(bucket), block_tables=ints(bucket, cols))
    w = _rows(1, q=(128,), k=(128,))
    table = rope_cos_sin_cache(128, 4096, 1e6).to(DEV)
    qkv = torch.zeros(layers, bucket, (h + 2 * hkv) * 128, dtype=torch.bfloat16, device=DEV)
    shape = (layers, blocks, 256, hkv, 128)
    stager = DecodeMetadataStager(bucket, cols, 256, DEV)
    att = nanovllm_b200.Attention(h, 128, default_scale(128), hkv)

    def step(record, kv, sync):
        stager.unpack_into(record, **gv)
        sync()
        out = []
        for i in range(layers):
            att.k_cache, att.v_cache = kv["k"][i], kv["v"][i]
            q, k, v = qk_norm_rope_store(qkv[i], gv["positions"], w["q"], w["k"], table, 1e-6, h, hkv, kv["k"][i], kv["v"][i],
                                         gv["slot_mapping"])
            sync()
            out += [q, k, att(q, k, v, already_stored=True)]
            sync()
        return out

    rng = random.Random(bucket)

    def batch():                                                     # (one sequence with a full row of the table: one record size)
        seqs = _fake_batch(rng, bs - 1, 2000, blocks - cols)
        return seqs + [FakeSeq(rng.randint(7 * 256 + 1, 8 * 256), list(range(blocks - cols, blocks)), 1)]

    set_context(False, slot_mapping=gv["slot_mapping"], context_lens=gv["context_lens"], block_tables=gv["block_tables"])
    with torch.inference_mode():
        replayed, stepped = _rows(2, k=shape, v=shape), _rows(2, k=shape, v=shape)
        stager.pack(batch())
        record = stager.to_device().clone()
        step(record, _rows(2, k=shape, v=shape), lambda: None)       # warm-up, on caches of its own
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = step(record, replayed, lambda: None)
        for turn in range(4):
            seqs = batch()
            stager.pack(seqs)
            record.copy_(stager.to_device())
            qkv.copy_(_rows(turn + 3, x=qkv.shape)["x"])
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            want = step(record, stepped, torch.cuda.synchronize)
            for x, y in zip(got + list(replayed.values()), want + list(stepped.values())):
                assert torch.equal(x.view(torch.int16), y.view(torch.int16))
            _, pos, _, lens, bt = prepare_decode_ref(seqs, 256)
            ref = qk_norm_rope_ref(qkv[0, :bs].cpu(), pos, w["q"].cpu(), w["k"].cpu(), table.cpu(), 1e-6, h, hkv, 128)
            _one_step(got[0][:bs].cpu(), ref[0])
            out = decode_attn_ref(got[0][:bs].cpu(), replayed["k"][0].cpu(), replayed["v"][0].cpu(), lens, bt, default_scale(128))
            torch.testing.assert_close(got[2][:bs].float().cpu(), out.float(), atol=2e-2, rtol=1e-2)
            assert not got[2][bs:].any()                             # padded rows
    reset_context()
