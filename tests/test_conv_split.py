"""Convs and linear layers with few output tiles, whose reduction runs over a cluster of CTAs, against the oracle."""
import pytest
import torch

from oracle import snn_oracle as orc
from util import check_parity

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    # cluster size; T, B, cin, cout, k, stride, H, W, residual, carried state
    (8, 4, 1, 512, 512, 3, 1, 7, 7, True, False),     # one image in a tile that holds two
    (8, 4, 3, 256, 200, 3, 1, 7, 7, True, True),      # two images and one; the last channel tile is ragged
    (8, 4, 1, 256, 512, 3, 2, 14, 14, False, False),  # stride 2: four phase tiles per slab
    (8, 4, 2, 256, 128, 3, 2, 29, 31, True, True),    # odd strided map, last tiles shifted back inside the image
    (8, 1, 2, 256, 256, 3, 1, 8, 8, False, True),     # one step
    (8, 3, 1, 256, 256, 3, 1, 13, 11, True, True),    # odd T: a pair and a single step in one window
    (8, 6, 1, 256, 128, 3, 1, 16, 9, True, True),     # windows of four and two steps
    (8, 7, 1, 384, 128, 3, 1, 15, 8, False, False),   # windows of four and three
    (8, 4, 1, 1152, 136, 1, 1, 14, 14, False, True),  # 1x1, ragged channels out
    (8, 2, 1, 1160, 256, 1, 1, 9, 8, False, False),   # 1x1, the last slab is partly filled
    (8, 12, 1, 512, 128, 3, 1, 5, 3, True, False),    # three windows, map smaller than half a tile row
    (4, 6, 24, 192, 100, 3, 1, 8, 8, True, True),        # windows of four and two steps
    (4, 3, 9, 256, 256, 3, 1, 9, 8, True, True),         # odd T
    (4, 4, 21, 1024, 256, 1, 1, 7, 8, False, True),      # 1x1, two images per tile and one
    (2, 1, 4, 512, 512, 3, 1, 16, 16, True, True),       # a CTA owns seven rows, all that its warps have room for
    (2, 4, 99, 512, 128, 3, 1, 7, 7, True, False),       # the same with two images per tile and one
    (2, 5, 40, 512, 128, 3, 1, 8, 8, False, True),       # windows of four steps and one
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_the_oracle(case, dtype):
    S, T, B, cin, cout, k, s, H, W, residual, carry = case
    from triton_snn_fusion_b200 import _lib
    from triton_snn_fusion_b200.runtime import triton_convlif_backend as be
    assert _lib.conv_kernel_name(T, B, cin, H, W, cout, k, s, k // 2, dtype, residual=residual) == f"conv_split/{S}"
    g = torch.Generator().manual_seed(T * 1000 + cin + cout)
    xs = [(torch.rand(B, cin, H, W, generator=g) < 0.2).to(dtype) for _ in range(T)]
    w = (torch.randn(cout, cin, k, k, generator=g) * 2.5 / (0.2 * cin * k * k) ** 0.5).to(dtype)
    b = (torch.randn(cout, generator=g) * 0.1).to(dtype)
    ho, wo = (H - 1) // s + 1, (W - 1) // s + 1
    v0 = (torch.randn(B, cout, ho, wo, generator=g) * 0.3).to(dtype) if carry else torch.tensor(0.0, dtype=dtype)
    res = [(torch.rand(B, cout, ho, wo, generator=g) < 0.2).to(dtype) for _ in range(T)] if residual else None
    rs, rv = orc.temporal_conv_lif([orc.widen(x) for x in xs], orc.widen(w), orc.widen(b), orc.widen(v0) if carry else None,
                                   [s, s], [k // 2] * 2, [1, 1], 1, 1.0, 0.0, 2.0,
                                   residuals=[orc.widen(r) for r in res] if res else None)
    r = be._run_temporal(None, [x.to(DEV) for x in xs], [q.to(DEV) for q in res] if res else None, w.to(DEV), b.to(DEV),
                         v0.to(DEV), s, k // 2, 1, 1, 1.0, 0.0, 2.0, True, True, False, None)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    check_parity(r.spikes, r.v_next, rs, rv, dtype, what=str(case))
    assert 0.02 < float(rs.mean()) < 0.6


def test_soft_reset_membrane_in_place_one_byte_spikes():
    """fp32 membrane updated in place on a map whose tiles overlap, in two chained calls; tau no power of two."""
    from triton_snn_fusion_b200 import _lib as L
    B, cin, cout, H, W, T = 1, 256, 128, 17, 13, 6
    g = torch.Generator().manual_seed(4)
    x = (torch.rand(T, B, H, W, cin, generator=g) < 0.2).bfloat16()
    w = (torch.randn(cout, 3, 3, cin, generator=g) * 0.1).bfloat16()
    b = (torch.randn(cout, generator=g) * 0.1).bfloat16()
    nchw = lambda t: orc.widen(t).permute(0, 3, 1, 2)
    rs, rv = orc.temporal_conv_lif([nchw(x[t]) for t in range(T)], nchw(w), orc.widen(b), None, [1, 1], [1, 1], [1, 1], 1,
                                   0.8, -1.0, 3.0)
    xd, wd, bd = x.to(DEV), w.to(DEV), b.to(DEV)
    sp = torch.empty(T, B, H, W, cout, dtype=torch.uint8, device=DEV)
    v = torch.empty(B, H, W, cout, dtype=torch.float32, device=DEV)
    for t0, n in ((0, 4), (4, 2)):
        L.check(L.lib.snnb_conv_lif(xd[t0].data_ptr(), xd.stride(0), wd.data_ptr(), bd.data_ptr(), None,
                                    v.data_ptr() if t0 else None, sp[t0].data_ptr(), v.data_ptr(), n, B, cin, H, W, cout, 3, 3, 1,
                                    1, 1, L.BF16, L.U8, L.F32, 0.8, -1.0, 3.0, L.PATH_AUTO, None), "conv")
    torch.cuda.synchronize()
    assert L.device_status() == 0
    check_parity(sp.permute(0, 1, 4, 2, 3), v.permute(0, 3, 1, 2), rs, rv, torch.float32, what="in place")


@pytest.mark.parametrize("T,M,K,N", [(4, 32, 3072, 768), (2, 56, 1024, 130), (4, 72, 1024, 256), (3, 8, 768, 100)])
def test_linear_with_few_tokens(T, M, K, N):
    from triton_snn_fusion_b200.runtime import triton_temporal_linear_lif_backend as be
    g = torch.Generator().manual_seed(M + N)
    x = (torch.rand(T, M, K, generator=g) < 0.2).bfloat16()
    w = (torch.randn(N, K, generator=g) * 2.5 / (0.2 * K) ** 0.5).bfloat16()
    b = (torch.randn(N, generator=g) * 0.1).bfloat16()
    rs, rv = orc.temporal_linear_lif(orc.widen(x), orc.widen(w), orc.widen(b), None, 1.0, 0.0, 2.0)
    r = be.run_triton_fused_temporal_linear_lif_state_packed(x.to(DEV), w.to(DEV), b.to(DEV),
                                                             torch.tensor(0.0, device=DEV, dtype=torch.bfloat16), 1.0, 0.0, 2.0, True)
    check_parity(r.spikes, r.v_next, rs, rv, torch.bfloat16)


@pytest.mark.parametrize("form,B,cin,H,W", [("conv_split/8", 6, 256, 7, 7), ("conv_split/8", 5, 256, 3, 4),
                                           ("conv_split/4", 40, 256, 7, 7), ("conv_split/8", 3, 256, 17, 13)])
def test_an_image_comes_out_the_same_wherever_it_stands_in_the_batch(form, B, cin, H, W):
    """Copies of one image (dense values, whose sums depend on the order of the additions) in all places of a batch, two
    to a tile or one."""
    from triton_snn_fusion_b200 import _lib as L
    T, cout = 4, 128
    assert L.conv_kernel_name(T, B, cin, H, W, cout, 3, 1, 1, torch.bfloat16) == form
    g = torch.Generator().manual_seed(B)
    x = torch.randn(T, 1, H, W, cin, generator=g).bfloat16().expand(T, B, H, W, cin).contiguous().to(DEV)
    w = (torch.randn(cout, 3, 3, cin, generator=g) * 0.06).bfloat16().to(DEV)
    b = (torch.randn(cout, generator=g) * 0.1).bfloat16().to(DEV)
    sp, v = torch.empty(T, B, H, W, cout, dtype=torch.bfloat16, device=DEV), torch.empty(B, H, W, cout, device=DEV)
    L.check(L.lib.snnb_conv_lif(x.data_ptr(), x.stride(0), w.data_ptr(), b.data_ptr(), None, None, sp.data_ptr(), v.data_ptr(), T, B,
                                cin, H, W, cout, 3, 3, 1, 1, 1, L.BF16, L.BF16, L.F32, 1.0, 0.0, 2.0, L.PATH_AUTO, None), "conv")
    for i in range(1, B):
        assert torch.equal(v[i], v[0]) and torch.equal(sp[:, i], sp[:, 0])
    assert 0.02 < float(sp.float().mean()) < 0.6
