"""GPU: how the two decode kernels share out a batch, at the sizes where it can go wrong -- clusters of every size
(fewer tiles than CTAs, ragged shares), whole pairs just below and above one per CTA, cut pairs (one long sequence
among short ones; few long ones, whose parts get a CTA each), rows without context -- against the CPU oracle."""
import pytest
import torch

from oracle.attention_oracle import decode_attn_ref
from workloads import default_scale, make_block_tables

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _lens(kind, n):
    g = torch.Generator().manual_seed(n)
    if kind == "equal":
        return [200] * n
    if kind == "ragged":
        return torch.randint(0, 700, (n,), generator=g).tolist()
    if kind == "one long":
        return [6000 if i == n // 2 else 1 + i % 130 for i in range(n)]
    if kind == "spread":
        return [100 + 2900 * i // n for i in range(n)]
    return [int(kind)] * n                                    # one length


@pytest.mark.parametrize("kind,n,h,hkv", [
    ("1", 1, 16, 8), ("64", 1, 2, 1), ("65", 1, 2, 1), ("129", 2, 8, 8), ("513", 1, 16, 2), ("1000", 2, 16, 8),     # clusters of up to 8
    ("ragged", 3, 16, 8), ("ragged", 17, 2, 2), ("ragged", 60, 4, 1), ("ragged", 130, 4, 1), ("one long", 5, 16, 8),
    ("513", 3, 32, 2), ("ragged", 9, 5, 1),                                  # 16 and 5 query heads per kv head
    ("equal", 37, 16, 8), ("equal", 149, 4, 2), ("ragged", 296, 1, 1), ("ragged", 297, 1, 1), ("ragged", 512, 4, 1),
    ("spread", 20, 16, 4), ("spread", 100, 2, 1), ("spread", 148, 4, 2), ("9000", 2, 4, 2), ("9000", 1, 2, 1),   # a CTA per part
    ("one long", 40, 16, 8), ("one long", 300, 4, 1), ("one long", 513, 2, 1), ("0", 200, 2, 1),
])
def test_decode_shares(kind, n, h, hkv):
    import nanovllm_b200
    from nanovllm_b200 import _lib
    lens = _lens(kind, n)
    g = torch.Generator().manual_seed(n + h)
    bt, nb = make_block_tables(lens, 256, g)
    kc = (torch.randn(nb, 256, hkv, 128, generator=g) * 0.5).to(torch.bfloat16)
    vc = (torch.randn(nb, 256, hkv, 128, generator=g) * 0.5).to(torch.bfloat16)
    q = torch.randn(n, h, 128, generator=g).to(torch.bfloat16)
    cl = torch.tensor(lens, dtype=torch.int32)
    want = decode_attn_ref(q, kc, vc, cl, bt.clamp_min(0), default_scale(128))
    d = [x.to(DEV) for x in (q, kc, vc, cl, bt)]
    for _ in range(2):                                        # the counters are back at zero after the first call
        out = nanovllm_b200.decode_attention(*d, default_scale(128), hkv)
        torch.testing.assert_close(out.float().cpu(), want.float(), atol=2e-2, rtol=1e-2)
    _lib.check(_lib.load().b200_device_status())


@pytest.mark.parametrize("kind,n,h,hkv", [("562", 33, 2, 1), ("562", 17, 4, 2), ("ragged", 37, 4, 1), ("ragged", 37, 2, 1), ("3000", 17, 4, 2)])
def test_decode_between_cluster_sizes(kind, n, h, hkv):
    """The last pairs on clusters of 4, the first on clusters of 2, and a table too wide for those."""
    test_decode_shares(kind, n, h, hkv)


@pytest.mark.parametrize("kind,n,h,hkv", [("ragged", 15, 4, 1), ("ragged", 16, 4, 1), ("8000", 15, 2, 1), ("4000", 33, 2, 1), ("1200", 74, 2, 1),
                                          ("1300", 74, 2, 1), ("1000", 75, 2, 1), ("1100", 75, 2, 1), ("700", 148, 2, 1), ("700", 149, 2, 1), ("1", 15, 8, 1)])
def test_decode_at_the_lines_of_the_cluster_rule(kind, n, h, hkv):
    """The last and the first number of pairs on clusters of a size, the last and the first width of a table."""
    test_decode_shares(kind, n, h, hkv)


@pytest.mark.parametrize("slots", ["own", "anywhere", "holes"])
@pytest.mark.parametrize("n,h,hkv", [(1, 16, 8), (3, 8, 8), (9, 2, 1), (70, 4, 2), (140, 2, 1), (20, 16, 8), (37, 16, 8), (160, 8, 4),
                                     (161, 4, 2), (513, 2, 1)])
def test_layer_decode_with_store(slots, n, h, hkv):
    """The step's rows stored in the attention launch: at the sequences' ends, in other sequences' blocks (whoever reads such
    a row must see the new one), skipped and outside the cache; a row without context is stored all the same."""
    import nanovllm_b200
    from nanovllm_b200.utils.context import reset_context, set_context
    from oracle.attention_oracle import AttentionRef, Context
    from workloads import decode_slots
    g = torch.Generator().manual_seed(n * 7 + h)
    lens = torch.randint(1, 700, (n,), generator=g).tolist()
    bt, nb = make_block_tables(lens, 256, g)
    if slots == "own":
        sm = decode_slots(lens, bt, 256)
    else:
        sm = torch.randperm(nb * 256, generator=g)[:n].to(torch.int32)
        if slots == "holes":
            sm[::3] = -1
            sm[n // 2] = nb * 256 + 7
            lens[0] = 0
            sm[0] = 5 if not (sm == 5).any() else sm[0]
    kc = (torch.randn(nb, 256, hkv, 128, generator=g) * 0.5).to(torch.bfloat16)
    vc = (torch.randn(nb, 256, hkv, 128, generator=g) * 0.5).to(torch.bfloat16)
    q = torch.randn(n, h, 128, generator=g).to(torch.bfloat16)
    fused = torch.randn(n, 2 * hkv * 128, generator=g).to(torch.bfloat16)
    k, v = fused[:, :hkv * 128].reshape(n, hkv, 128).contiguous(), fused[:, hkv * 128:].view(n, hkv, 128)
    cl = torch.tensor(lens, dtype=torch.int32)
    att = nanovllm_b200.Attention(h, 128, default_scale(128), hkv)
    att.k_cache, att.v_cache = kc.to(DEV), vc.to(DEV)
    set_context(False, slot_mapping=sm.to(DEV), context_lens=cl.to(DEV), block_tables=bt.to(DEV))
    out = att(q.to(DEV), k.to(DEV), fused.to(DEV)[:, hkv * 128:].view(n, hkv, 128))
    torch.cuda.synchronize()
    reset_context()
    ref = AttentionRef(h, 128, default_scale(128), hkv)
    ref.k_cache, ref.v_cache = kc, vc
    inside = torch.where(sm < nb * 256, sm, torch.full_like(sm, -1))
    want = ref.forward(q, k, v, Context(False, slot_mapping=inside, context_lens=cl, block_tables=bt.clamp_min(0)))
    torch.testing.assert_close(out.float().cpu(), want.float(), atol=2e-2, rtol=1e-2)
    assert torch.equal(att.k_cache.cpu().view(torch.int16), kc.view(torch.int16))
    assert torch.equal(att.v_cache.cpu().view(torch.int16), vc.view(torch.int16))


@pytest.mark.parametrize("kind,n,h,hkv", [("one long", 40, 64, 8), ("spread", 256, 2, 1), ("spread", 20, 16, 4), ("spread", 60, 16, 2),
                                          ("9000", 6, 32, 4), ("one long", 300, 16, 1)])
def test_cut_pairs_repeat_bit_for_bit(kind, n, h, hkv):
    """Which CTA brings a pair's last part depends on timing; the order in which its parts are summed must not."""
    import nanovllm_b200
    lens = _lens(kind, n)
    g = torch.Generator().manual_seed(n + 3 * h)
    bt, nb = make_block_tables(lens, 256, g)
    gd = torch.Generator(device=DEV).manual_seed(n)
    kc, vc = (torch.randn(nb, 256, hkv, 128, device=DEV, generator=gd).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(n, h, 128, device=DEV, generator=gd).to(torch.bfloat16)
    cl, bt = torch.tensor(lens, dtype=torch.int32, device=DEV), bt.to(DEV)
    scratch = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    first = nanovllm_b200.decode_attention(q, kc, vc, cl, bt, default_scale(128), hkv)
    for i in range(60):
        scratch[:(i % 5) << 25].fill_(i)                      # another state of L2 every time, so other CTAs are late
        out = nanovllm_b200.decode_attention(q, kc, vc, cl, bt, default_scale(128), hkv)
        assert torch.equal(out.view(torch.int16), first.view(torch.int16)), f"run {i}"
