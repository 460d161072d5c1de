"""The fp32 conv / linear + LIF kernel at the edges of its tiles against the oracle."""
import pytest
import torch

from oracle import snn_oracle as orc
from util import check_parity

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    # T, B, cin, cout, k, stride, pad, H, W
    (4, 1, 4, 1, 3, 1, 1, 5, 7),        # one channel out, K = 36: the last K chunk is partly filled
    (4, 3, 20, 33, 3, 1, 1, 9, 11),     # a chunk spans taps; channels one past a 32-channel tile, not a multiple of 4
    (8, 2, 8, 65, 3, 2, 1, 13, 9),      # eight steps per tile, one channel past 64
    (1, 5, 16, 64, 1, 1, 0, 8, 8),      # one step in a window of eight
    (3, 4, 12, 36, 3, 1, 1, 10, 10),    # odd T, the rest of the window is idle
    (6, 2, 16, 128, 3, 1, 1, 12, 12),   # T even and no power of two
    (16, 1, 32, 64, 1, 1, 0, 7, 5),     # two windows of eight, membrane in shared memory
    (4, 40, 64, 128, 3, 1, 1, 14, 14),  # more 64-channel tiles than SMs
    (4, 2, 4, 16, 11, 4, 2, 35, 35),    # 121 taps
    (2, 1, 28, 8, 5, 1, 2, 6, 6),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("residual", [False, True])
def test_against_the_oracle(case, residual):
    T, B, cin, cout, k, s, pad, H, W = case
    from triton_snn_fusion_b200.runtime import triton_convlif_backend as be
    g = torch.Generator().manual_seed(T * 100 + cin + cout)
    xs = [torch.randn(B, cin, H, W, generator=g) for _ in range(T)]
    w = torch.randn(cout, cin, k, k, generator=g) * (2.0 / (cin * k * k)) ** 0.5
    b = torch.randn(cout, generator=g) * 0.1
    ho, wo = (H + 2 * pad - k) // s + 1, (W + 2 * pad - k) // s + 1
    v0 = torch.randn(B, cout, ho, wo, generator=g) * 0.3
    res = [(torch.rand(B, cout, ho, wo, generator=g) < 0.2).float() for _ in range(T)] if residual else None
    rs, rv = orc.temporal_conv_lif(xs, w, b, v0, [s, s], [pad, pad], [1, 1], 1, 1.0, 0.0, 2.0, residuals=res)
    args = (w.to(DEV), b.to(DEV), v0.to(DEV), s, pad, 1, 1, 1.0, 0.0, 2.0, True)
    xd = [x.to(DEV) for x in xs]
    run = be._run_temporal
    r = run(None, xd, [q.to(DEV) for q in res] if res else None, *args, True, False, None)
    check_parity(r.spikes, r.v_next, rs, rv, torch.float32, what=str(case))


@pytest.mark.parametrize("cin,kernel", [(8, "conv_lif_simt"), (24, "conv_lif_f32/1x32")])
def test_one_frame_for_all_steps_one_byte_spikes_soft_reset_in_place(cin, kernel):
    from triton_snn_fusion_b200 import _lib as L
    B, cout, H, W, T = 2, 24, 9, 9, 5
    assert L.conv_kernel_name(T, B, cin, H, W, cout, 3, 1, 1, torch.float32, one_frame=True, path=L.PATH_SIMT) == kernel
    g = torch.Generator().manual_seed(3)
    x = torch.randn(B, H, W, cin, generator=g)
    w = torch.randn(cout, cin, 3, 3, generator=g) * 0.3
    b = torch.randn(cout, generator=g) * 0.1
    v0 = torch.randn(B, H, W, cout, generator=g) * 0.3
    rs, rv = orc.temporal_conv_lif([x.permute(0, 3, 1, 2)] * T, w, b, v0.permute(0, 3, 1, 2), [1, 1], [1, 1], [1, 1], 1, 0.8, -1.0, 3.0)
    xd, wd, bd, v = x.to(DEV), w.permute(0, 2, 3, 1).contiguous().to(DEV), b.to(DEV), v0.to(DEV)
    sp = torch.empty(T, B, H, W, cout, dtype=torch.uint8, device=DEV)
    L.check(L.lib.snnb_conv_lif(xd.data_ptr(), 0, wd.data_ptr(), bd.data_ptr(), None, v.data_ptr(), sp.data_ptr(), v.data_ptr(),
                                T, B, cin, H, W, cout, 3, 3, 1, 1, 1, L.F32, L.U8, L.F32, 0.8, -1.0, 3.0, L.PATH_SIMT, None), "conv")
    torch.cuda.synchronize()
    check_parity(sp.permute(0, 1, 4, 2, 3), v.permute(0, 3, 1, 2), rs, rv, torch.float32)


@pytest.mark.parametrize("M,K,N,T", [(1, 4, 4, 4), (22, 1024, 100, 4), (33, 36, 130, 2), (130, 64, 64, 1)])
def test_linear(M, K, N, T):
    from triton_snn_fusion_b200.runtime import triton_temporal_linear_lif_backend as be
    g = torch.Generator().manual_seed(M + N)
    x, w, b = torch.randn(T, M, K, generator=g), torch.randn(N, K, generator=g) / K ** 0.5 * 2, torch.randn(N, generator=g) * 0.1
    rs, rv = orc.temporal_linear_lif(x, w, b, None, 1.0, 0.0, 2.0)
    r = be.run_triton_fused_temporal_linear_lif_state_packed(x.to(DEV), w.to(DEV), b.to(DEV), torch.tensor(0.0, device=DEV), 1.0, 0.0, 2.0, True)
    check_parity(r.spikes, r.v_next, rs, rv, torch.float32)


TILES = [
    # steps of a window, channels of a block; T, B, H, cout (1x1, 36 channels in): a window and several, ragged pixels, the
    # last channel past the block's first
    (8, 32, 6, 1, 5, 9), (8, 32, 9, 3, 5, 9), (8, 64, 5, 3, 20, 33), (8, 64, 11, 3, 20, 35),
    (4, 32, 4, 32, 9, 9), (4, 32, 9, 96, 9, 9), (4, 64, 3, 96, 5, 33), (4, 64, 9, 96, 5, 33),
    (2, 32, 2, 12, 20, 9), (2, 32, 5, 192, 9, 9), (2, 64, 2, 12, 20, 33), (2, 64, 5, 96, 9, 36),
    (1, 32, 1, 24, 20, 9), (1, 32, 3, 191, 14, 9), (1, 64, 1, 24, 20, 33), (1, 64, 3, 191, 9, 33),
]


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("residual", [False, True])
def test_every_tile_of_the_kernel(tile, residual):
    steps, channels, T, B, H, cout = tile
    from triton_snn_fusion_b200 import _lib as L
    assert L.conv_kernel_name(T, B, 36, H, H, cout, 1, 1, 0, torch.float32, residual=residual) == f"conv_lif_f32/{steps}x{channels}"
    g = torch.Generator().manual_seed(T * 100 + B)
    x, w = torch.randn(T, B, H, H, 36, generator=g), torch.randn(cout, 1, 1, 36, generator=g) / 3
    b, v0 = torch.randn(cout, generator=g) * 0.1, torch.randn(B, H, H, cout, generator=g) * 0.3
    res = (torch.rand(T, B, H, H, cout, generator=g) < 0.2).float() if residual else None
    nchw = lambda t: t.permute(0, 3, 1, 2)
    rs, rv = orc.temporal_conv_lif([nchw(x[t]) for t in range(T)], nchw(w), b, nchw(v0), [1, 1], [0, 0], [1, 1], 1, 1.0, 0.0, 2.0,
                                   residuals=[nchw(res[t]) for t in range(T)] if residual else None)
    xd, wd, bd, v = x.to(DEV), w.to(DEV), b.to(DEV), v0.to(DEV)
    rd = res.to(DEV) if residual else None
    sp = torch.empty(T, B, H, H, cout, device=DEV)
    L.check(L.lib.snnb_conv_lif(xd.data_ptr(), xd.stride(0), wd.data_ptr(), bd.data_ptr(), L.ptr(rd), v.data_ptr(), sp.data_ptr(),
                                v.data_ptr(), T, B, 36, H, H, cout, 1, 1, 1, 0, 1, L.F32, L.F32, L.F32, 1.0, 0.0, 2.0, L.PATH_AUTO,
                                None), "conv")
    check_parity(sp.permute(0, 1, 4, 2, 3), v.permute(0, 3, 1, 2), rs, rv, torch.float32, what=str(tile))
