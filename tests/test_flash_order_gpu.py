"""The order of products that the attention kernels rely on: a product may write over tensor memory that
an earlier product of the same thread reads, with no wait in between (S over P in the forward for heads
wider than 64, S over P and dP over dS in the dK / dV pass).  Were it broken, rows of a result would hold
parts of other tiles: calls with many tiles per CTA, repeated next to other work on the GPU, equal the first
to the bit, and a call of the same kind is compared with 64 bits.  Head sizes at which the two products have
different widths."""
import pytest
import torch

from slapo_b200.ops import native
from test_flash_paths_gpu import BF, FP, test_flash_attention_paths as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [40, 64, 72, 80, 112, 128])
@pytest.mark.parametrize("b,s,h,how,p", [(4, 1000, 16, "", 0.0), (2, 1500, 12, "c", 0.1)])
def test_products_in_order(b, s, h, how, p, d):
    ops = native.ops()
    dtype = FP if d == 80 else BF
    check(1, s, s, h, d, dtype, how, p)
    torch.manual_seed(d)
    q, k, v, do = (torch.randn(b, s, h, d, device="cuda", dtype=dtype) for _ in range(4))
    rng = torch.tensor([7, 4, 0, 0], dtype=torch.int64) if p else None
    causal, scale = "c" in how, d ** -0.5
    out, lse = ops.flash_attn_fwd(q, k, v, None, None, causal, scale, p, rng)
    grads = ops.flash_attn_bwd(do, q, k, v, out, lse, None, None, causal, scale, p, rng, False)[:3]
    side, other = torch.cuda.Stream(), torch.randn(2048, 2048, device="cuda").to(BF)
    for i in range(12):
        if i % 3 == 0:      # another stream's kernels take some of the SMs
            with torch.cuda.stream(side):
                for _ in range(4):
                    other @ other
        again, lse2 = ops.flash_attn_fwd(q, k, v, None, None, causal, scale, p, rng)
        assert torch.equal(again, out) and torch.equal(lse2, lse), i
        g = ops.flash_attn_bwd(do, q, k, v, out, lse, None, None, causal, scale, p, rng, False)[:3]
        assert all(torch.equal(x, y) for x, y in zip(g, grads)), i
    torch.cuda.synchronize()
    assert ops.device_status() == 0
