"""GPU: the dense prefill step of the layer, whose cache store rides along in the attention launch: slots that run on and
slots that do not, skipped and out-of-range slots, ragged tiles, every split of a query block over key tiles, sequences
without queries, keys that start before the queries -- attention against the oracle, the cache bit for bit."""
import pytest
import torch

from oracle.attention_oracle import prefill_attn_ref, store_kvcache_ref
from workloads import cu_seqlens, default_scale

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("slots", ["blocks", "scattered", "holes"])
@pytest.mark.parametrize("h,hkv,lq,lk", [
    (16, 8, [1, 127, 128, 129, 31, 32, 33, 700, 2000], None), (16, 8, [1, 63, 64, 65, 33], None), (2, 1, [70], None),
    (2, 2, [255, 256, 257, 600], None),                      # one query head per kv head: two key tiles per query block
    (32, 8, [63, 64, 65, 500], None), (8, 1, [300, 17], None),
    (5, 1, [100, 200], None), (3, 1, [2000, 7], None),       # not tcgen05 head ratios
    (4, 2, [100, 0, 300, 64], [150, 90, 300, 400]), (8, 8, [900, 0, 1300, 64, 2000], [950, 90, 1300, 400, 2000]),
])
def test_layer_prefill_with_store(slots, h, hkv, lq, lk):
    import nanovllm_b200
    from nanovllm_b200 import _lib
    from nanovllm_b200.utils.context import reset_context, set_context
    lk = lk or lq
    g = torch.Generator().manual_seed(sum(lq) + h)
    n = sum(lk)
    blocks = n // 256 + len(lk) + 2
    q = torch.randn(sum(lq), h, 128, generator=g).to(torch.bfloat16)
    fused = torch.randn(n, 2 * hkv * 128, generator=g).to(torch.bfloat16)
    k, v = fused[:, :hkv * 128].reshape(n, hkv, 128).contiguous(), fused[:, hkv * 128:].view(n, hkv, 128)
    kc = torch.randn(blocks, 256, hkv, 128, generator=g).to(torch.bfloat16)
    vc = torch.randn(blocks, 256, hkv, 128, generator=g).to(torch.bfloat16)
    if slots == "scattered":
        sm = torch.randperm(blocks * 256, generator=g)[:n].to(torch.int32)
    else:
        perm, rows = torch.randperm(blocks, generator=g).tolist(), []
        for m in lk:
            for t in range(m):
                if t % 256 == 0:
                    b = perm.pop()
                rows.append(b * 256 + t % 256)
        sm = torch.tensor(rows, dtype=torch.int32)
        if slots == "holes":
            sm[::9] = -1
            sm[5] = blocks * 256 + 3                          # outside the cache: skipped
    cu_q, cu_k = cu_seqlens(lq), cu_seqlens(lk)
    att = nanovllm_b200.Attention(h, 128, default_scale(128), hkv)
    att.k_cache, att.v_cache = kc.to(DEV), vc.to(DEV)
    fd = fused.to(DEV)
    set_context(True, cu_q.to(DEV), cu_k.to(DEV), max(lq), max(lk), sm.to(DEV))
    out = att(q.to(DEV), k.to(DEV), fd[:, hkv * 128:].view(n, hkv, 128))
    torch.cuda.synchronize()
    reset_context()
    torch.testing.assert_close(out.float().cpu(), prefill_attn_ref(q, k, v, cu_q, cu_k, default_scale(128)).float(), atol=2e-2, rtol=1e-2)
    ok = sm < blocks * 256
    store_kvcache_ref(k[ok], v[ok], kc, vc, sm[ok])
    assert torch.equal(att.k_cache.cpu().view(torch.int16), kc.view(torch.int16))
    assert torch.equal(att.v_cache.cpu().view(torch.int16), vc.view(torch.int16))
    _lib.check(_lib.load().b200_device_status())
