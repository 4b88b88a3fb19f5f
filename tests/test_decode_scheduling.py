"""GPU: how the two decode kernels share out a batch, at the sizes where it can go wrong -- clusters of every size
(fewer tiles than CTAs, ragged shares), whole pairs just below and above one per CTA, cut pairs (one long sequence
among short ones), rows without context -- against the CPU oracle."""
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
    return [int(kind)] * n                                    # one length


@pytest.mark.parametrize("kind,n,h,hkv", [
    ("1", 1, 16, 8), ("64", 1, 2, 1), ("65", 1, 2, 1), ("129", 2, 8, 8), ("513", 1, 16, 2), ("1000", 2, 16, 8),     # clusters of up to 8
    ("ragged", 3, 16, 8), ("ragged", 17, 2, 2), ("ragged", 60, 4, 1), ("ragged", 130, 4, 1), ("one long", 5, 16, 8),
    ("513", 3, 32, 2), ("ragged", 9, 5, 1),                                  # 16 and 5 query heads per kv head
    ("equal", 37, 16, 8), ("equal", 149, 4, 2), ("ragged", 296, 1, 1), ("ragged", 297, 1, 1), ("ragged", 512, 4, 1),
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
