"""GPU: how the tcgen05 prefill kernel hands out its work -- few items, whose keys the two halves share tile by tile (one tile,
odd and even numbers of them, rows that see nothing of a half's only tile), and many, in the order of their lengths
(batches up to the sort's limit, beyond it, and beyond the slot table) -- dense and paged, against the oracle."""
import pytest
import torch

from oracle.attention_oracle import prefill_attn_ref
from workloads import cu_seqlens, default_scale

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EDGES = [1, 127, 128, 129, 255, 256, 257, 384, 385, 513, 640, 900]


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("h,hkv,lq,lk", [
    (2, 1, EDGES, None), (1, 1, [1], None), (4, 1, [33], None), (8, 1, [130], None), (16, 8, [1500], None), (128, 1, [70], None),
    (4, 2, [1, 64, 65, 200], [129, 320, 1000, 201]),         # cached prefixes
    (2, 1, [300, 0, 70, 300], [100, 50, 1, 257]),            # rows without a visible key
    (32, 8, EDGES * 4, None), (16, 8, (EDGES * 22)[:256], None), (16, 8, (EDGES * 22)[:257], None),
    (4, 2, [1 + i % 150 for i in range(1100)], None),
])
def test_tcgen05_items(paged, h, hkv, lq, lk):
    from nanovllm_b200.layers.attention import prefill_attention
    lk = lk or lq
    g = torch.Generator().manual_seed(sum(lk) + h)
    n = sum(lk)
    q = torch.randn(sum(lq), h, 128, generator=g).to(torch.bfloat16)
    k = torch.randn(n, hkv, 128, generator=g).to(torch.bfloat16)
    v = torch.randn(n, hkv, 128, generator=g).to(torch.bfloat16)
    cu_q, cu_k = cu_seqlens(lq), cu_seqlens(lk)
    args, bt = (k.to(DEV), v.to(DEV)), None
    if paged:
        cols = -(-max(lk) // 256)
        blocks = sum(-(-m // 256) for m in lk) + 1
        perm = torch.randperm(blocks, generator=g).tolist()
        bt = torch.full((len(lk), cols), -1, dtype=torch.int32)
        kc = torch.full((blocks, 256, hkv, 128), float("nan"), dtype=torch.bfloat16)     # what is not the sequence's own
        vc = torch.full((blocks, 256, hkv, 128), float("nan"), dtype=torch.bfloat16)
        at = 0
        for i, m in enumerate(lk):
            for c in range(-(-m // 256)):
                rows = min(256, m - 256 * c)
                b = perm.pop()
                bt[i, c] = b
                kc[b, :rows], vc[b, :rows] = k[at:at + rows], v[at:at + rows]
                at += rows
        args, bt = (kc.to(DEV), vc.to(DEV)), bt.to(DEV)
    scale = default_scale(128)
    out = prefill_attention(q.to(DEV), *args, cu_q.to(DEV), cu_k.to(DEV), max(lq), max(lk), scale, hkv, bt, kernel_variant=2)
    torch.cuda.synchronize()
    ref = prefill_attn_ref(q, k, v, cu_q, cu_k, scale).float()
    torch.testing.assert_close(out.float().cpu(), ref, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("h,hkv", [(2, 1), (64, 1)])                 # 64 query tokens to a CTA, one or two
@pytest.mark.parametrize("batch", [1, 2, 30, 31, 32, 33, 63, 64, 961, 962, 1023, 1100])
def test_mma_finds_its_sequence(batch, h, hkv):
    """The mma.sync kernel's search, 32 places at a time: batches around a power of 32, sequences without queries first, last and
    in a row, a query tile of several sequences and sequences of several tiles."""
    from nanovllm_b200.layers.attention import prefill_attention
    g = torch.Generator().manual_seed(batch)
    lq = [0 if i % 7 in (0, 5, 6) and batch > 2 else 1 + (i * 37) % 3 for i in range(batch)]
    lq[batch // 2] = 70
    lk = [m + i % 3 for i, m in enumerate(lq)]
    n = sum(lk)
    q = torch.randn(sum(lq), h, 128, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(n, hkv, 128, generator=g).to(torch.bfloat16) for _ in range(2))
    cu_q, cu_k = cu_seqlens(lq), cu_seqlens(lk)
    out = prefill_attention(q.to(DEV), k.to(DEV), v.to(DEV), cu_q.to(DEV), cu_k.to(DEV), max(lq), max(lk), default_scale(128), hkv, None, 1)
    want = prefill_attn_ref(q, k, v, cu_q, cu_k, default_scale(128))
    torch.testing.assert_close(out.float().cpu(), want.float(), atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("h,hkv,lens", [(16, 8, [60, 70]), (2, 1, [700, 31, 2000]), (2, 2, [900] * 40)])     # mma.sync, tcgen05 in both forms
def test_store_ends_with_the_rows_of_k(h, hkv, lens):
    """cu_seqlens_k that run past total_k, in a sequence without queries: rows there are not read, whatever kernel takes the call.
    (k, v and slots go on behind total_k, so that a store of these rows would show in the cache.)"""
    from nanovllm_b200 import _lib
    n, beyond = sum(lens) + 40, 60
    g = torch.Generator(device=DEV).manual_seed(n)
    q = torch.randn(sum(lens), h, 128, device=DEV, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(n + beyond, hkv, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    kc, vc = (torch.zeros(-(-(n + beyond) // 256), 256, hkv, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    slots = torch.arange(n + beyond, dtype=torch.int32, device=DEV)
    cu_q, cu_k = cu_seqlens(lens + [0]).to(DEV), cu_seqlens(lens + [40 + beyond]).to(DEV)
    out = torch.empty_like(q)
    _lib.check(_lib.load().b200_store_prefill_attn(
        q.data_ptr(), h * 128, k.data_ptr(), v.data_ptr(), hkv * 128, hkv * 128, n, kc.data_ptr(), vc.data_ptr(), slots.data_ptr(),
        kc.shape[0] * 256, cu_q.data_ptr(), cu_k.data_ptr(), len(lens) + 1, sum(lens), max(lens), max(lens + [40 + beyond]), out.data_ptr(), h, hkv, 128,
        default_scale(128), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for cache, rows in ((kc, k), (vc, v)):
        flat = cache.view(-1, hkv, 128)
        assert torch.equal(flat[:n], rows[:n]) and not flat[n:].any()
