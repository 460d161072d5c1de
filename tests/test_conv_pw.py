"""The GEMM kernel of 1x1 convs and linear layers at the edges of its tiles, against the oracle."""
import pytest
import torch

from oracle import snn_oracle as orc
from util import check_parity

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    # T, pixels, cin, cout, residual, carried state, (v_th, v_reset, tau)
    (4, 1, 64, 130, False, False, (1.0, 0.0, 2.0)),       # one pixel; the last channel tile holds two channels
    (4, 127, 72, 128, False, True, (1.0, 0.0, 2.0)),      # one pixel short of a tile; a partly filled slab
    (4, 129, 64, 64, True, True, (1.0, 0.0, 2.0)),        # a shifted last tile; duplicated weight rows
    (1, 300, 128, 40, False, False, (1.0, 0.0, 2.0)),     # one step, ragged channels
    (3, 257, 192, 200, True, True, (1.0, 0.0, 2.0)),      # odd T: the last pair holds one step
    (2, 20000, 64, 256, False, False, (1.0, 0.0, 2.0)),   # more tiles than SMs: blocks walk tiles with resident weights
    (6, 3000, 640, 384, False, True, (1.0, 0.0, 2.0)),    # weights streamed
    (5, 200, 512, 136, True, False, (0.8, -1.0, 2.0)),    # soft reset
    (4, 200, 64, 128, False, True, (1.0, 0.2, 3.0)),      # reset to a value, tau no power of two
    (7, 150, 320, 72, True, True, (1.0, 0.2, 3.0)),       # the same with a residual, odd T
    (3, 131, 72, 33, True, False, (0.8, -1.0, 3.0)),      # 33 channels: the residual is not copied ahead
    (6, 5, 128, 200, True, True, (1.0, 0.0, 0.9)),        # tau at most 1; five pixels
    (4, 300, 128, 64, False, False, (1.0, -1.0, 0.9)),    # tau at most 1, soft reset
    (8, 40, 576, 136, True, False, (1.0, 0.0, 2.0)),      # residual, weights streamed
    (2, 19000, 64, 200, True, False, (1.0, 0.0, 2.0)),    # residual, blocks walk tiles
    (9, 70, 320, 24, True, True, (1.0, 0.0, 2.0)),        # residual, duplicated weight rows, odd T
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_the_oracle(case, dtype):
    T, P, cin, cout, residual, carry, lif = case
    from triton_snn_fusion_b200 import _lib
    from triton_snn_fusion_b200.runtime import triton_convlif_backend as be
    assert _lib.conv_kernel_name(T, 1, cin, 1, P, cout, 1, 1, 0, dtype, residual=residual) == "conv_pw"
    g = torch.Generator().manual_seed(P + cin)
    xs = [(torch.rand(1, cin, 1, P, generator=g) < 0.2).to(dtype) for _ in range(T)]
    w = (torch.randn(cout, cin, 1, 1, generator=g) * 2.5 / (0.2 * cin) ** 0.5).to(dtype)
    b = (torch.randn(cout, generator=g) * 0.1).to(dtype)
    v0 = (torch.randn(1, cout, 1, P, generator=g) * 0.3).to(dtype) if carry else torch.tensor(0.0, dtype=dtype)
    res = [(torch.rand(1, cout, 1, P, generator=g) < 0.2).to(dtype) for _ in range(T)] if residual else None
    rs, rv = orc.temporal_conv_lif([orc.widen(x) for x in xs], orc.widen(w), orc.widen(b), orc.widen(v0) if carry else None,
                                   [1, 1], [0, 0], [1, 1], 1, *lif, residuals=[orc.widen(r) for r in res] if res else None)
    r = be._run_temporal(None, [x.to(DEV) for x in xs], [q.to(DEV) for q in res] if res else None, w.to(DEV), b.to(DEV),
                         v0.to(DEV), 1, 0, 1, 1, *lif, True, True, False, None)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    check_parity(r.spikes, r.v_next, rs, rv, dtype, what=str(case))


def test_membrane_in_place_on_a_shifted_tile_and_no_lif():
    from triton_snn_fusion_b200 import _lib as L
    P, cin, cout, T = 321, 64, 96, 4
    g = torch.Generator().manual_seed(5)
    x = (torch.rand(T, P, cin, generator=g) < 0.2).bfloat16()
    w = (torch.randn(cout, cin, generator=g) * 0.6).bfloat16()
    b = (torch.randn(cout, generator=g) * 0.1).bfloat16()
    rs, rv = orc.temporal_linear_lif(orc.widen(x), orc.widen(w), orc.widen(b), None, 1.0, 0.0, 2.0)
    xd, wd, bd = x.to(DEV), w.to(DEV), b.to(DEV)
    sp = torch.empty(T, P, cout, dtype=torch.uint8, device=DEV)
    v = torch.empty(P, cout, device=DEV)
    for t0 in (0, 2):
        L.check(L.lib.snnb_linear_lif(xd[t0].data_ptr(), xd.stride(0), wd.data_ptr(), bd.data_ptr(), v.data_ptr() if t0 else None,
                                      sp[t0].data_ptr(), v.data_ptr(), 2, P, cin, cout, L.BF16, L.U8, L.F32, 1.0, 0.0, 2.0,
                                      L.PATH_AUTO, None), "linear")
    check_parity(sp, v, rs, rv, torch.float32)
    out = torch.empty(T, P, cout, dtype=torch.bfloat16, device=DEV)
    L.check(L.lib.snnb_conv_lif(xd.data_ptr(), xd.stride(0), wd.data_ptr(), bd.data_ptr(), None, None, out.data_ptr(), None, T, 1,
                                cin, 1, P, cout, 1, 1, 1, 0, 0, L.BF16, L.BF16, L.BF16, 1.0, 0.0, 2.0, L.PATH_AUTO, None), "conv")
    ref = orc.widen(x) @ orc.widen(w).t() + orc.widen(b)
    torch.testing.assert_close(out.float().cpu(), ref, rtol=1e-2, atol=1e-2)   # one rounding to bf16: 2^-9 relative


def test_no_lif_with_a_residual():
    from triton_snn_fusion_b200 import _lib as L
    P, cin, cout, T = 200, 96, 104, 5
    g = torch.Generator().manual_seed(6)
    x = (torch.rand(T, P, cin, generator=g) < 0.2).bfloat16()
    w, b = (torch.randn(cout, cin, generator=g) * 0.4).bfloat16(), (torch.randn(cout, generator=g) * 0.1).bfloat16()
    res = torch.randn(T, P, cout, generator=g).bfloat16()
    xd, wd, bd, rd = x.to(DEV), w.to(DEV), b.to(DEV), res.to(DEV)
    out = torch.empty(T, P, cout, dtype=torch.bfloat16, device=DEV)
    L.check(L.lib.snnb_conv_lif(xd.data_ptr(), xd.stride(0), wd.data_ptr(), bd.data_ptr(), rd.data_ptr(), None, out.data_ptr(), None,
                                T, 1, cin, 1, P, cout, 1, 1, 1, 0, 0, L.BF16, L.BF16, L.BF16, 1.0, 0.0, 2.0, L.PATH_AUTO, None), "conv")
    ref = orc.widen(x) @ orc.widen(w).t() + orc.widen(b) + orc.widen(res)
    torch.testing.assert_close(out.float().cpu(), ref, rtol=1e-2, atol=1e-2)   # one rounding to bf16: 2^-9 relative
