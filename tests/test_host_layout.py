"""The backends' layout checks on the host against the general tensor operations (CPU only)."""
import itertools

import pytest
import torch

from triton_snn_fusion_b200.runtime import _common as cm
from triton_snn_fusion_b200.runtime import triton_convlif_backend as be
from triton_snn_fusion_b200.runtime import triton_temporal_lif_backend as lf


def _dense(t):
    d = t.dim()
    return t.permute(list(range(d - 3)) + [d - 2, d - 1, d - 3]).is_contiguous()


@pytest.mark.parametrize("shape", [(2, 3, 4, 5), (1, 3, 1, 5), (2, 1, 4, 1), (4, 2, 3, 4, 5), (1, 1, 1, 1), (3, 0, 2, 2),
                                   (2, 1, 3, 1, 4)])
def test_channels_last_check_agrees_with_contiguity(shape):
    lead = len(shape) - 3
    for perm in itertools.permutations(range(len(shape))):
        t = torch.empty([shape[i] for i in perm]).permute([perm.index(i) for i in range(len(shape))])
        assert t.shape == torch.Size(shape) and cm.is_nhwc_dense(t) == _dense(t)
        wide = torch.empty([2 * n for n in t.shape])[tuple(slice(0, n) for n in t.shape)]
        assert cm.is_nhwc_dense(wide) == _dense(wide)
    e = cm.empty_nhwc(shape, torch.float32, "cpu")
    assert e.shape == torch.Size(shape) and (0 in shape or e.permute(list(range(lead)) + [lead + 1, lead + 2, lead]).is_contiguous())


def test_frames_are_used_in_place_only_where_they_are_equally_spaced_and_dense():
    stack = torch.arange(5 * 2 * 4 * 4 * 8.0).reshape(5, 2, 4, 4, 8).movedim(-1, -3)
    fr = list(stack)
    assert cm.stack_frames(fr)[1:] == (stack.stride(0), False)
    assert cm.stack_frames(fr[::2])[1:] == (2 * stack.stride(0), False)
    assert cm.stack_frames([fr[1]] * 3)[1:] == (0, False) and cm.stack_frames(fr[:1])[1:] == (0, False)
    nchw = [f.contiguous() for f in fr]
    for xs in (fr[::-1], [fr[0], fr[1], fr[3]], nchw, [fr[0], nchw[1]], [f[:, :, :2] for f in fr]):
        base, step, copied = cm.stack_frames(xs)
        assert copied and step == base.numel()
        for t, x in enumerate(xs):
            assert torch.equal(torch.as_strided(base, base.shape, base.stride(), base.storage_offset() + t * step), x)
    base, step, copied = cm.stack_frames([nchw[0]] * 2)
    assert copied and step == 0 and torch.equal(base, nchw[0])


def test_scan_layout_check():
    x = torch.zeros(3, 2, 4, 5, 6)
    ok = lf._same_dense_layout
    assert ok(x, None) and ok(x, x[0]) and ok(x.movedim(-1, -3), x.movedim(-1, -3)[0])
    assert not ok(x, x.movedim(-1, -3)[0].reshape(2, 4, 5, 6).clone(memory_format=torch.channels_last))
    assert not ok(x[:, :1], None) and not ok(x.transpose(0, 1), None) and not ok(x[..., :3], None)


def test_kept_plans_do_not_let_an_unsupported_call_through(monkeypatch):
    monkeypatch.setattr(cm.Gate, "lead_is", lambda self, rank: None)   # CPU tensors stand in for GPU ones
    x, w, b, v = torch.zeros(1, 4, 8, 8), torch.zeros(8, 4, 3, 3), torch.zeros(8), torch.tensor(0.0)
    call = lambda **k: be._plan(*[k.get(n, d) for n, d in (("x", x), ("w", w), ("b", b), ("v", v), ("s", [1, 1]), ("p", 1),
                                                           ("d", 1), ("g", 1))], 1.0, 0.0, k.get("tau", 2.0), True, False, False)
    try:
        assert call() == call() == ("k3_s1_p1", (1, 8, 8, 8)) and call(s=2) == ("k3_s2_p1", (1, 8, 4, 4))
        for bad in (dict(tau=0.0), dict(b=None), dict(b=b.half()), dict(v=torch.zeros(1, 8, 8, 7)), dict(w=w[:, :2]), dict(d=2),
                    dict(s=3), dict(p=0), dict(g=2), dict(v=torch.tensor(0.0).half().reshape(1))):
            with pytest.raises(RuntimeError):
                call(**bad)
    finally:
        be._PLANS.clear()   # plans of CPU tensors must not outlive the patch
