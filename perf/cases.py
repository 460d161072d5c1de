"""Workloads of the fused spiking ops and networks, each through the public entry point a program calls.

A case is a dict of plain values; ``kind`` names the entry point:

  lif      the standalone LIF scan over a pre-activation sequence
  conv     dense conv + folded BatchNorm (+ residual) + LIF over T steps; with ``sc_cin`` the residual is the strided
           1x1 shortcut conv of a down-sampling block, run by its own call in front
  dw       3x3 depthwise conv + LIF
  linear   linear + LIF over packed tokens
  tail     LIF -> global average pool -> linear
  net      one forward pass of a compiled network (CUDA graph, batch already on the GPU)

Inputs of conv / dw / linear layers are spikes (0 / 1, about one in five set), what such a layer meets behind another
LIF layer. Weights are scaled so that the currents have a standard deviation near 3, as the conv weights x4 under which
every stage of the benchmark networks keeps firing; about a third of the neurons spike per step.

Spikes are returned as the integers that their bits spell, because they are whole values: an implementation that sums
in another order may flip the few neurons whose charge lies within a rounding of the threshold and must agree in all
others. Such a flip moves that neuron's membrane by about the threshold, so an fp32 membrane behind a convolution has no
meaningful distance to a 64-bit evaluation (it is 1e-7 without a flip and 1e-3 with one); the fp32 case returns its
shortcut conv, which has no threshold, and that is compared.
"""
import math

import torch
import torch.nn.functional as F

from triton_snn_fusion_b200 import nets
from triton_snn_fusion_b200.runtime import triton_convlif_backend as conv
from triton_snn_fusion_b200.runtime import triton_temporal_lif_avgpool_linear_backend as tail
from triton_snn_fusion_b200.runtime import triton_temporal_lif_backend as lif
from triton_snn_fusion_b200.runtime import triton_temporal_linear_lif_backend as linear

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
SIZE = {"fp32": 4, "bf16": 2, "fp16": 2}
V_TH, V_RESET, TAU = 1.0, 0.0, 2.0
RATE = 0.2          # share of set inputs
SIGMA = 3.0         # standard deviation of the currents


def listed():
    return [
        # the smallest call: one CIFAR-sized activation map, where the launch is what counts
        dict(name="lif_small_fp32", kind="lif", dtype="fp32", T=4, B=2, C=64, H=32, W=32, carry=False),
        # a standalone LIF behind an un-fused op at the width of a ResNet's first stage
        dict(name="lif_large_bf16", kind="lif", dtype="bf16", T=4, B=64, C=64, H=112, W=112, carry=False),
        # the second conv of a ResNet block at serving batch: identity shortcut added before the LIF
        dict(name="conv_residual_bf16", kind="conv", dtype="bf16", T=4, B=64, cin=128, cout=128, H=28, W=28, k=3, s=1,
             residual=True, sc_cin=0, carry=False),
        # the same layer of the last stage for one image: latency of a long reduction with few output tiles
        dict(name="conv_one_image_bf16", kind="conv", dtype="bf16", T=4, B=1, cin=512, cout=512, H=7, W=7, k=3, s=1,
             residual=True, sc_cin=0, carry=False),
        # a strided stage transition on an odd map, fp16
        dict(name="conv_stride2_fp16", kind="conv", dtype="fp16", T=4, B=16, cin=128, cout=256, H=29, W=29, k=3, s=2,
             residual=False, sc_cin=0, carry=False),
        # a down-sampling block's end in fp32, the default type of the reference's models, on CIFAR-sized maps
        dict(name="conv_shortcut_fp32", kind="conv", dtype="fp32", T=4, B=16, cin=128, cout=128, H=16, W=16, k=3, s=1,
             residual=False, sc_cin=64, carry=False),
        # pointwise and depthwise layers of MobileNetV1
        dict(name="pointwise_bf16", kind="conv", dtype="bf16", T=4, B=32, cin=256, cout=256, H=28, W=28, k=1, s=1,
             residual=False, sc_cin=0, carry=False),
        dict(name="depthwise_bf16", kind="dw", dtype="bf16", T=4, B=32, C=128, H=56, W=56, s=1, carry=False),
        # the feed-forward expansion of a spiking transformer (config 1)
        dict(name="linear_bf16", kind="linear", dtype="bf16", T=4, M=4096, K=768, N=3072, carry=False),
        # classifier tail of MobileNetV1
        dict(name="tail_bf16", kind="tail", dtype="bf16", T=4, B=64, C=1024, H=7, W=7, classes=1000, carry=False),
        # whole networks: a request of two images, and a serving batch
        dict(name="resnet18_two_images", kind="net", net="resnet18", dtype="bf16", T=4, B=2, hw=224),
        dict(name="mobilenet_v1_batch64", kind="net", net="mobilenet_v1", dtype="bf16", T=4, B=64, hw=224),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: the same ops over their ranges; the batch is what is left of a work budget drawn log-uniformly."""
    kind = rng.choice(["lif", "conv", "conv", "conv", "conv", "dw", "linear", "tail", "net"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    T = rng.choice([4, 4, 4, 2, 8, 1, 6, 3])
    carry = rng.random() < 0.25     # the state of the previous window goes in
    if kind == "net":
        net = rng.choice(["resnet18", "mobilenet_v1"])
        return dict(kind="net", net=net, dtype=rng.choice(["bf16", "fp16"]), T=rng.choice([4, 4, 2]),
                    B=_log_int(rng, 1, 32 if net == "resnet18" else 48), hw=rng.choice([224, 224, 192, 160]))
    if kind == "linear":
        K, N = rng.choice([(768, 3072), (3072, 768), (512, 512), (384, 1536), (512, 100), (1024, 4096)])
        flops = math.exp(rng.uniform(math.log(1e8), math.log(8e9 if dtype == "fp32" else 1.2e11)))
        M = max(1, int(flops / (2 * T * K * N)))
        M = M if rng.random() < 0.3 else max(8, M // 8 * 8)
        return dict(kind="linear", dtype=dtype, T=T, M=M, K=K, N=N, carry=carry)
    hw = rng.choice([7, 8, 14, 16, 28, 32, 56, rng.randint(7, 56)])
    if kind == "lif":
        C = rng.choice([32, 64, 128, 256, 100, 48])
        B = max(1, int(math.exp(rng.uniform(math.log(1e4), math.log(3e7))) / (C * hw * hw)))
        return dict(kind="lif", dtype=dtype, T=T, B=B, C=C, H=hw, W=hw, carry=carry)
    if kind == "dw":
        C = rng.choice([32, 64, 128, 256, 512, 1024, 96])
        B = max(1, int(math.exp(rng.uniform(math.log(1e5), math.log(3e7))) / (C * hw * hw * T)))
        return dict(kind="dw", dtype=dtype, T=T, B=B, C=C, H=hw, W=hw, s=rng.choice([1, 1, 2]), carry=carry)
    if kind == "tail":
        C, hw = rng.choice([256, 512, 1024, 100]), rng.choice([4, 7, 7, 8])
        return dict(kind="tail", dtype=dtype, T=T, B=_log_int(rng, 1, 512), C=C, H=hw, W=hw,
                    classes=rng.choice([10, 100, 1000]), carry=carry)
    k = rng.choice([3, 3, 3, 1])
    s = rng.choice([1, 1, 2]) if k == 3 else 1
    cin, cout = rng.choice([(64, 64), (64, 128), (128, 128), (128, 256), (256, 256), (256, 512), (512, 512), (512, 1024),
                            (192, 96)])
    if cout >= 512:
        hw = min(hw, 28)
    extra = rng.random()
    flops = math.exp(rng.uniform(math.log(2e8), math.log(8e9 if dtype == "fp32" else 1.5e11)))
    ho = (hw - 1) // s + 1
    B = max(1, int(flops / (2 * T * ho * ho * cin * cout * k * k)))
    return dict(kind="conv", dtype=dtype, T=T, B=B, cin=cin, cout=cout, H=hw, W=hw, k=k, s=s,
                residual=extra < 0.35, sc_cin=cin // 2 if extra > 0.85 and s == 1 and k == 3 and cin % 128 == 0 else 0,
                carry=carry)


# ------------------------------------------------------------------------------------------------- sizes ----
def _out_hw(c):
    s = c.get("s", 1)
    return (c["H"] - 1) // s + 1, (c["W"] - 1) // s + 1


def _layer_work(L, T, B, h, w, ho, wo, sz):
    """bytes and flops of one layer of a network spec; spikes in and out once, weights once."""
    if L["op"] == "conv":
        steps = 1 if L["src"] == "input" else T
        return (steps * B * h * w * L["cin"] * sz * (L["src"] == "input"),
                2 * steps * B * ho * wo * L["cout"] * (L["cin"] // L["groups"]) * L["k"] ** 2,
                L["cout"] * (L["cin"] // L["groups"]) * L["k"] ** 2 * sz)
    if L["op"] in ("tail", "head"):
        return B * L["classes"] * 4, 2 * B * L["cin"] * L["classes"], L["cin"] * L["classes"] * sz
    return 0, 0, 0


def work(c):
    sz, T = SIZE[c["dtype"]], c["T"]
    if c["kind"] == "net":
        # input, weights and logits; each layer's spikes written and read once
        spec = nets.NETS[c["net"]](1000)
        shape, nbytes, flops = {"input": (c["hw"], c["hw"], 3)}, 0, 0
        for L in spec:
            h, w, ch = shape[L["src"]]
            ho, wo = h, w
            if L["op"] == "conv":
                ho, wo = (h + 2 * L["p"] - L["k"]) // L["s"] + 1, (w + 2 * L["p"] - L["k"]) // L["s"] + 1
                shape[L["dst"]] = (ho, wo, L["cout"])
                nbytes += 2 * T * c["B"] * ho * wo * L["cout"] * sz
            elif L["op"] == "maxpool":
                ho, wo = (h - 1) // 2 + 1, (w - 1) // 2 + 1
                shape[L["dst"]] = (ho, wo, ch)
                nbytes += 2 * T * c["B"] * ho * wo * ch * sz
            a, f, wb = _layer_work(L, T, c["B"], h, w, ho, wo, sz)
            nbytes, flops = nbytes + a + wb, flops + f
        return {"bytes": nbytes, "flops": flops}
    states = 2 if c["carry"] else 1
    if c["kind"] == "linear":
        M, K, N = c["M"], c["K"], c["N"]
        return {"bytes": sz * (T * M * K + N * K + N + T * M * N + states * M * N), "flops": 2 * T * M * K * N}
    B, pix = c["B"], c["H"] * c["W"]
    if c["kind"] == "lif":
        n = B * c["C"] * pix
        return {"bytes": sz * n * (2 * T + states), "flops": 5 * T * n}
    if c["kind"] == "tail":
        n = B * c["C"] * pix
        return {"bytes": sz * (n * (T + states) + (c["C"] + 1 + B) * c["classes"]),
                "flops": 5 * T * n + 2 * B * c["C"] * c["classes"]}
    ho, wo = _out_hw(c)
    if c["kind"] == "dw":
        n_in, n_out = B * c["C"] * pix, B * c["C"] * ho * wo
        return {"bytes": sz * (T * (n_in + n_out) + states * n_out + 10 * c["C"]), "flops": 18 * T * n_out}
    n_in, n_out, K = B * c["cin"] * pix, B * c["cout"] * ho * wo, c["cin"] * c["k"] ** 2
    nbytes = T * (n_in + n_out * (2 if c["residual"] else 1)) + states * n_out + c["cout"] * (K + 1)
    flops = 2 * T * n_out * K
    if c["sc_cin"]:   # the shortcut conv is a result of its own; of its input every second pixel is read
        nbytes += T * n_out * 2 + T * B * ho * wo * c["sc_cin"] + c["cout"] * (c["sc_cin"] + 1)
        flops += 2 * T * n_out * c["sc_cin"]
    return {"bytes": sz * nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------------ inputs ----
def _spikes(g, shape, dt):
    """0 / 1 values, channels innermost in memory; logical [..., C, H, W] for shape [..., H, W, C]."""
    x = (torch.rand(shape, device="cuda", generator=g) < RATE).to(dt)
    return x.movedim(-1, -3)


def _weights(g, cout, cin, k, dt):
    w = torch.randn(cout, k, k, cin, device="cuda", generator=g) * (SIGMA / math.sqrt(RATE * cin * k * k))
    b = torch.randn(cout, device="cuda", generator=g) * 0.3
    return w.to(dt).permute(0, 3, 1, 2), b.to(dt)


def _state(g, c, shape, dt):
    """The membrane of the previous window, or the 0-dim tensor that stands for a start from rest."""
    if not c["carry"]:
        return torch.zeros((), device="cuda", dtype=dt)
    v = torch.randn(shape, device="cuda", generator=g) - 0.5
    return torch.where(v < V_TH, v, torch.zeros_like(v)).to(dt).movedim(-1, -3)


def prepare(c, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dt, T = DTYPES[c["dtype"]], c["T"]
    if c["kind"] == "net":
        spec = nets.NETS[c["net"]](1000)
        net = nets.CompiledNet(spec, nets.make_params(spec, seed=int(seed), gain=4.0), c["B"], T, (c["hw"], c["hw"]), dt)
        x = torch.randn(c["B"], c["hw"], c["hw"], 3, device="cuda", generator=g).to(dt)
        net.forward(x)
        net.capture()
        return dict(kind="net", net=net, x=x)
    if c["kind"] == "linear":
        x = (torch.rand(T, c["M"], c["K"], device="cuda", generator=g) < RATE).to(dt)
        w = torch.randn(c["N"], c["K"], device="cuda", generator=g) * (SIGMA / math.sqrt(RATE * c["K"]))
        b = torch.randn(c["N"], device="cuda", generator=g) * 0.3
        v = torch.zeros((), device="cuda", dtype=dt)
        if c["carry"]:
            v = torch.randn(c["M"], c["N"], device="cuda", generator=g) - 0.5
            v = torch.where(v < V_TH, v, torch.zeros_like(v)).to(dt)
        return dict(kind="linear", x=x, w=w.to(dt), b=b.to(dt), v=v)
    B, H, W = c["B"], c["H"], c["W"]
    if c["kind"] in ("lif", "tail"):
        C = c["C"]
        x = (torch.randn(T, B, H, W, C, device="cuda", generator=g) * 0.8 + 0.6).to(dt).movedim(-1, -3)
        s = dict(kind=c["kind"], x=x, v=_state(g, c, (B, H, W, C), dt))
        if c["kind"] == "tail":
            s["w"] = (torch.randn(c["classes"], C, device="cuda", generator=g) * math.sqrt(2.0 / C)).to(dt)
            s["b"] = (torch.randn(c["classes"], device="cuda", generator=g) * 0.01).to(dt)
        return s
    ho, wo = _out_hw(c)
    if c["kind"] == "dw":
        C = c["C"]
        x = _spikes(g, (T, B, H, W, C), dt)
        w, b = _weights(g, C, 1, 3, dt)
        return dict(kind="dw", x=list(x), w=w.contiguous(), b=b, v=_state(g, c, (B, ho, wo, C), dt), s=c["s"], C=C)
    x = _spikes(g, (T, B, H, W, c["cin"]), dt)
    w, b = _weights(g, c["cout"], c["cin"], c["k"], dt)
    st = dict(kind="conv", x=list(x), w=w, b=b, v=_state(g, c, (B, ho, wo, c["cout"]), dt), s=c["s"], k=c["k"], res=None,
              sc_x=None)
    if c["residual"]:
        st["res"] = list(_spikes(g, (T, B, ho, wo, c["cout"]), dt))
    if c["sc_cin"]:   # the block's input, at twice the resolution
        st["sc_x"] = list(_spikes(g, (T, B, 2 * H, 2 * W, c["sc_cin"]), dt))
        st["sc_w"], st["sc_b"] = _weights(g, c["cout"], c["sc_cin"], 1, dt)
    return st


# --------------------------------------------------------------------------------------------- the calls ----
def _bits(spikes):
    return spikes.view(torch.int32 if spikes.dtype == torch.float32 else torch.int16)


def run(s):
    kind = s["kind"]
    if kind == "net":
        return s["net"].forward(s["x"])
    if kind == "lif":
        r = lif.run_triton_fused_temporal_lif_state(s["x"], s["v"], V_TH, V_RESET, TAU, True)
        return {"spikes": _bits(r.spikes), "v": r.v_next}
    if kind == "linear":
        r = linear.run_triton_fused_temporal_linear_lif_state_packed(s["x"], s["w"], s["b"], s["v"], V_TH, V_RESET, TAU, True)
        return {"spikes": _bits(r.spikes), "v": r.v_next}
    if kind == "tail":
        r = tail.run_triton_fused_temporal_lif_avgpool_linear(s["x"], s["v"], s["w"], s["b"], V_TH, V_RESET, TAU, True)
        return {"out": r.out_sum, "v": r.v_next}
    if kind == "dw":
        r = conv.run_triton_fused_temporal_depthwise_conv_lif_state(
            s["x"], s["w"], s["b"], s["v"], s["s"], 1, 1, s["C"], V_TH, V_RESET, TAU, True)
        return {"spikes": _bits(r.spikes), "v": r.v_next}
    args = (s["w"], s["b"], s["v"], s["s"], s["k"] // 2, 1, 1, V_TH, V_RESET, TAU, True)
    if s["sc_x"] is not None:
        sc = conv.conv_bias_only(s["sc_x"], s["sc_w"], s["sc_b"], 2, 0)
        r = conv.run_triton_fused_temporal_conv_add_lif_state(s["x"], list(sc), *args)
        return {"spikes": _bits(r.spikes), "v": r.v_next, "shortcut": sc}
    if s["res"] is not None:
        r = conv.run_triton_fused_temporal_conv_add_lif_state(s["x"], s["res"], *args)
    elif s["k"] == 1:
        r = conv.run_triton_fused_temporal_pointwise_conv_lif_state(s["x"], *args)
    else:
        r = conv.run_triton_fused_temporal_conv_lif_state(s["x"], *args)
    return {"spikes": _bits(r.spikes), "v": r.v_next}


# -------------------------------------------------------------------------------------------- comparison ----
def tolerance(c):
    if c["kind"] == "lif":
        return "exact"    # one defined order of operations per neuron
    if c["kind"] == "net":
        # With 16-bit weights and whole inputs nearly all partial sums are exact in fp32: logits of the same network on
        # kernels with another order of summation were the same. One flipped spike travels through all later layers,
        # so a neuron or two on the threshold have to be allowed for.
        return {"rel": 0.02, "max": 0.2}
    if c["kind"] == "tail":
        # counts are whole; the class sums are rounded to the activation type (fp32: 512-term sums)
        return {"rel": 1e-5 if c["dtype"] == "fp32" else 1e-2, "max": 1e-3 if c["dtype"] == "fp32" else 0.05}
    # a neuron whose charge lies within a rounding of the threshold may fire on one side only, which moves its
    # membrane by the threshold (about 0.7 of its root mean square)
    return {"rel": 1e-2, "max": 0.99, "differ": 1e-4}


def _lif64(xs, v):
    spikes = []
    for x in xs:
        h = v + (x - v) / TAU
        s = h >= V_TH
        v = torch.where(s, torch.full_like(h, V_RESET), h)
        spikes.append(s)
    return spikes, v


def exact(c, seed):
    if c["kind"] == "net":
        return None       # a flip in one layer moves all later ones: no 64-bit value to hold a 16-bit network against
    s = prepare(c, seed)
    v = s["v"].double()
    if c["kind"] in ("lif", "tail"):
        spikes, v = _lif64([x.double() for x in s["x"]], v.expand(s["x"].shape[1:]))
        if c["kind"] == "lif":
            return {"spikes": None, "v": v}
        count = sum(z.double().mean(dim=(2, 3)) for z in spikes)
        return {"out": count @ s["w"].double().t() + c["T"] * s["b"].double(), "v": v}
    if c["kind"] == "linear":
        ys = [x.double() @ s["w"].double().t() + s["b"].double() for x in s["x"]]
    else:
        w, b = s["w"].double(), s["b"].double()
        groups = c["C"] if c["kind"] == "dw" else 1
        ys = [F.conv2d(x.double().contiguous(), w, b, stride=s["s"], padding=w.shape[-1] // 2, groups=groups) for x in s["x"]]
    out = {}
    if c["kind"] == "conv" and s["sc_x"] is not None:
        sc = [F.conv2d(x.double().contiguous(), s["sc_w"].double(), s["sc_b"].double(), stride=2) for x in s["sc_x"]]
        out["shortcut"] = torch.stack(sc)
        ys = [y + r.to(DTYPES[c["dtype"]]).double() for y, r in zip(ys, sc)]
    if c["kind"] == "conv" and s["res"] is not None:
        ys = [y + r.double() for y, r in zip(ys, s["res"])]
    _, v = _lif64(ys, v.expand(ys[0].shape))
    if c["dtype"] == "fp32":
        return {"spikes": None, "v": None, **out} if out else None
    return {"spikes": None, "v": v, **out}
