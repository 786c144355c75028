"""The work a user of this library has it do, as cases that can be timed.

A case is a dict of plain values.  `kind` names the piece of a training or inference program it is:

  conv     one Conv3D unit's training step: forward (with bias), deltaX, deltaW and deltaB
  act      inference through one Conv3D unit with its LeakyReLU fused, batch as given
  deconv   one Deconv3D unit's training step (a generator layer): dconv3D and its two gradients
  resnet   the 20 convolutions of the CIFAR-10 ResNet-18, forward, deltaX and deltaW of each
  sweep    3x3 layers of the benchmark's sweep, forward, deltaX and deltaW of each
  dcgan    the four transposed convolutions of the DCGAN generator with their gradients
  large    the large-image layers: 3x3 and 5x5 at 112 x 112, 1x1 with 1024 channels
  fc       one FullConnect unit's training step: matMul_biased, matMulT2, matMulT1, the bias gradient
  bmm      attention-like batched products: batchMatMul, batchMatMulT1, batchMatMulT2
  pool     indexed max pooling and average pooling with their gradients

Everything runs through Engine, eagerly and on the current stream, as a program without CUDA graphs calls it.
Activations are NHWC float32: ReLU(N(0,1)) inputs, He-normal weights, N(0,1) output gradients; images are uniform [0,1).
"""
import math

import torch

from __graft_entry__ import submodule


def _case(name, kind, **values):
    return dict(name=name, kind=kind, **values)


def listed():
    return [
        # the smallest calls: the single-layer configuration of the tests (launch count and host path decide)
        _case("conv_small", "conv", N=4, IH=32, IW=32, IC=16, OC=32, F=3, s=1, p=1, math="3xtf32"),
        # CIFAR-10 ResNet-18 at the batch one of eight data-parallel ranks sees
        _case("resnet18_b64", "resnet", N=64, math="3xtf32"),
        # the same network at the benchmark's batch
        _case("resnet18_b512", "resnet", N=512, math="3xtf32"),
        # the benchmark's own step: four layers, batch 256
        _case("sweep_b256", "sweep", N=256, math="3xtf32"),
        # large images and wide filters in the opt-in plain TF32 mode (the largest case)
        _case("large_tf32", "large", N=128, math="tf32"),
        # DCGAN generator: transposed 4x4 stride-2 layers, training
        _case("dcgan_b256", "dcgan", N=256, math="3xtf32"),
        # a down-sampling layer on a large image
        _case("down_112", "conv", N=128, IH=112, IW=112, IC=128, OC=64, F=3, s=2, p=1, math="3xtf32"),
        # channel counts and image sizes that are multiples of nothing (36 -> 100 channels on 35 x 29)
        _case("ragged_conv", "conv", N=50, IH=35, IW=29, IC=36, OC=100, F=3, s=1, p=1, math="3xtf32"),
        # inference: a 7x7 stride-2 stem on 3 colour planes with its activation
        _case("stem_224", "act", N=32, IH=224, IW=224, IC=3, OC=64, F=7, s=2, p=3),
        # a classifier's FullConnect layer, training
        _case("fc_1000", "fc", N=512, K=4096, M=1000, math="3xtf32"),
        # batched products at the shape of the reference's own table
        _case("bmm_128", "bmm", B=256, N=128, M=128, K=256, math="3xtf32"),
        # pooling after a stem, forward and backward
        _case("pool_112", "pool", N=256, IH=112, IW=112, IC=64, F=3, s=2, p=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _conv_flops(c):
    OH, OW = _out(c["IH"], c), _out(c["IW"], c)
    return 2.0 * c["N"] * OH * OW * c["OC"] * c["F"] ** 2 * c["IC"]


def draw(rng):
    kind = rng.choice(("conv", "conv", "conv", "conv", "act", "deconv", "resnet", "sweep", "fc", "bmm", "pool"))
    mode = rng.choice(("3xtf32", "3xtf32", "tf32"))
    if kind in ("conv", "act", "deconv"):
        while True:
            F, s, p = rng.choice(((3, 1, 1), (3, 1, 1), (3, 2, 1), (1, 1, 0), (1, 2, 0), (4, 2, 1), (5, 1, 2), (7, 2, 3)))
            if kind == "deconv":
                F, s, p = rng.choice(((4, 2, 1), (4, 2, 1), (3, 1, 1), (2, 2, 0)))
            # half of the channel counts are the usual multiples of 32, half are whatever the log scale gives
            ch = [_log(rng, 3, 768) if rng.random() < 0.5 else 32 * _log(rng, 1, 20) for _ in range(2)]
            IH = _log(rng, 4, 130)
            IW = IH if rng.random() < 0.6 else _log(rng, 4, 130)
            c = dict(kind=kind, N=_log(rng, 1, 512), IH=IH, IW=IW, IC=ch[0], OC=ch[1], F=F, s=s, p=p)
            # the reference's deltaX wants windows that cover the padded image exactly up to the stride
            c["IH"] += (F - IH - 2 * p) % s if s > 1 and F % 2 == 0 else 0
            c["IW"] += (F - IW - 2 * p) % s if s > 1 and F % 2 == 0 else 0
            size = c["N"] * (c["IH"] * c["IW"] * max(c["IC"], 4) + _out(c["IH"], c) * _out(c["IW"], c) * max(c["OC"], 4))
            if 1e7 <= _conv_flops(c) <= 1.2e11 and size <= 2.5e8:
                break
        return c if kind == "act" else dict(c, math=mode)
    if kind == "resnet":
        return dict(kind=kind, N=_log(rng, 8, 640), math=mode)
    if kind == "sweep":
        return dict(kind=kind, N=_log(rng, 16, 256), math=mode)
    if kind == "fc":
        return dict(kind=kind, N=_log(rng, 16, 2048), K=_log(rng, 64, 8192), M=_log(rng, 10, 8192), math=mode)
    if kind == "bmm":
        while True:
            c = dict(kind=kind, B=_log(rng, 4, 512), N=_log(rng, 20, 512), M=_log(rng, 20, 512), K=_log(rng, 20, 512), math=mode)
            if c["B"] * c["N"] * c["M"] * c["K"] <= 2e10:
                return c
    F, s, p = rng.choice(((3, 2, 1), (2, 2, 0), (3, 1, 1)))
    while True:
        IH = _log(rng, 4, 130)
        c = dict(kind="pool", N=_log(rng, 1, 512), IH=IH, IW=IH if rng.random() < 0.6 else _log(rng, 4, 130), IC=_log(rng, 3, 512), F=F, s=s, p=p)
        if c["N"] * c["IH"] * c["IW"] * c["IC"] <= 2.1e8:
            return c


def _out(size, c):
    return (size + 2 * c["p"] - c["F"]) // c["s"] + 1


# ---- the layers of the stacks, as (IH, IW, IC, OC, F, s, p) of the convolution -------------------------------

def _layers(c):
    synth = submodule("synth")
    if c["kind"] == "resnet":
        return [(ih, ih, ic, oc, F, s, p) for ih, ic, oc, F, s, p in synth.RESNET18_CONVS]
    if c["kind"] == "sweep":
        return [(hw, hw, ch, ch, 3, 1, 1) for hw, ch in synth.SWEEP_LAYERS]
    if c["kind"] == "large":
        return [(112, 112, 64, 64, 3, 1, 1), (112, 112, 64, 128, 5, 1, 2), (14, 14, 1024, 1024, 1, 1, 0)]
    if c["kind"] == "dcgan":   # a generator layer grows h to 2h: as a convolution its image is the output
        return [(2 * h, 2 * h, cout, cin, 4, 2, 1) for h, cin, cout in synth.DCGAN_DECONVS]
    return [(c["IH"], c["IW"], c["IC"], c["OC"], c["F"], c["s"], c["p"])]


_STACKS = ("resnet", "sweep", "large", "dcgan", "deconv", "conv", "act")


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    engine = submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=case.get("math")))
    st = dict(case=case, eng=eng)

    def normal(*shape, scale=1.0):
        return torch.randn(shape, device=dev, generator=g).mul_(scale)

    kind, N = case["kind"], case["N"]
    if kind in _STACKS:
        st["layers"] = []
        for IH, IW, IC, OC, F, s, p in _layers(case):
            OH, OW = (IH + 2 * p - F) // s + 1, (IW + 2 * p - F) // s + 1
            L = dict(IH=IH, IW=IW, F=F, s=s, p=p)
            if kind in ("dcgan", "deconv"):
                L["Z"] = normal(N, OH, OW, OC).relu_()          # the unit's input
                L["dX"] = normal(N, IH, IW, IC)                 # gradient at the unit's output
                L["W"] = normal(OC, F, F, IC, scale=0.02)
            else:
                if IC <= 4:
                    L["X"] = torch.rand((N, IH, IW, IC), device=dev, generator=g)
                    if IC == 4:
                        L["X"][..., 3] = 0                      # three colour planes padded to four
                else:
                    L["X"] = normal(N, IH, IW, IC).relu_()
                L["W"] = normal(OC, F, F, IC, scale=math.sqrt(2.0 / (F * F * IC)))
                if kind != "act":
                    L["dY"] = normal(N, OH, OW, OC)
                L["B"] = torch.rand((OC,), device=dev, generator=g).sub_(0.5).mul_(0.2)
            st["layers"].append(L)
    elif kind == "fc":
        K, M = case["K"], case["M"]
        st.update(X=normal(N, K).relu_(), W=normal(K, M, scale=math.sqrt(2.0 / K)), dY=normal(N, M, scale=1.0),
                  B=torch.rand((M,), device=dev, generator=g).sub_(0.5).mul_(0.2))
    elif kind == "bmm":
        B, M, K = case["B"], case["M"], case["K"]
        st.update(A=normal(B, N, K), V=normal(B, K, M), dC=normal(B, N, M))
    else:
        shape = (N, case["IH"], case["IW"], case["IC"])
        out = (N, _out(case["IH"], case), _out(case["IW"], case), case["IC"])
        st.update(X=normal(*shape).relu_(), dY=normal(*out))
    return st


def run(state):
    c, eng = state["case"], state["eng"]
    kind = c["kind"]
    if kind == "act":
        L = state["layers"][0]
        return eng.conv3D_leakyRelu(L["X"], L["W"], L["B"], 0.2, L["s"], L["s"], L["p"], L["p"])
    if kind in ("dcgan", "deconv"):
        out = []
        for L in state["layers"]:
            F, s, p = L["F"], L["s"], L["p"]
            X = eng.dconv3D_deltaX(L["Z"], L["W"], L["IH"], L["IW"], s, s, p, p)   # Deconv3D forward
            dZ = eng.conv3D(L["dX"], L["W"], s, s, p, p)
            dW = eng.dconv3D_deltaW(L["dX"], L["Z"], F, F, s, s, p, p)
            out += [X, dZ, dW]
        return out
    if kind in _STACKS:
        out = []
        for L in state["layers"]:
            s, p, F = L["s"], L["p"], L["F"]
            Y = eng.conv3D(L["X"], L["W"], s, s, p, p, Bias=L["B"] if kind == "conv" else None)
            dX = eng.dconv3D_deltaX(L["dY"], L["W"], L["IH"], L["IW"], s, s, p, p)
            dW = eng.dconv3D_deltaW(L["X"], L["dY"], F, F, s, s, p, p)
            out += [Y, dX, dW]
            if kind == "conv":
                out.append(eng.field_sum(L["dY"]))
        return out
    if kind == "fc":
        Y = eng.matMul(state["X"], state["W"], Bias=state["B"])
        dX = eng.matMulT2(state["dY"], state["W"])
        dW = eng.matMulT1(state["X"], state["dY"])
        return Y, dX, dW, eng.field_sum(state["dY"])
    if kind == "bmm":
        C = eng.batchMatMul(state["A"], state["V"])                  # C = A V
        dV = eng.batchMatMulT1(state["A"], state["dC"])              # A^T dC
        dA = eng.batchMatMulT2(state["dC"], state["V"])              # dC V^T
        return C, dV, dA
    F, s, p, X, dY = c["F"], c["s"], c["p"], state["X"], state["dY"]
    Y, index = eng.pool2D_max(X, F, F, s, s, p, p, indexed=True)
    dX = eng.upool2D_max_indexed(dY, index, c["IH"], c["IW"], F, F, s, s, p, p)
    A = eng.pool2D_avg(X, F, F, s, s, p, p)
    dA = eng.upool2D_avg(dY, c["IH"], c["IW"], F, F, s, s, p, p)
    return Y, index, dX, A, dA


def work(case):
    kind, N = case["kind"], case["N"]
    if kind in _STACKS:
        b = f = 0.0
        for IH, IW, IC, OC, F, s, p in _layers(case):
            OH, OW = (IH + 2 * p - F) // s + 1, (IW + 2 * p - F) // s + 1
            x, y, w = N * IH * IW * IC, N * OH * OW * OC, OC * F * F * IC
            ops = 1 if kind == "act" else 3
            # a training step reads X, deltaY and W once and writes Y, deltaX and deltaW once
            b += 4.0 * ((x + w + y) if kind == "act" else 2 * (x + w + y))
            f += ops * 2.0 * N * OH * OW * OC * F * F * IC
        return {"bytes": b, "flops": f}
    if kind == "fc":
        K, M = case["K"], case["M"]
        return {"bytes": 8.0 * (N * K + K * M + N * M), "flops": 6.0 * N * K * M}
    if kind == "bmm":
        B, M, K = case["B"], case["M"], case["K"]
        return {"bytes": 8.0 * B * (N * K + K * M + N * M), "flops": 6.0 * B * N * K * M}
    x = N * case["IH"] * case["IW"] * case["IC"]
    y = N * _out(case["IH"], case) * _out(case["IW"], case) * case["IC"]
    # X, deltaY in; Y, index, deltaX, average, its gradient out
    return {"bytes": 4.0 * (3 * x + 4 * y), "flops": 0.0}


# Largest relative error (2-norm of the difference over 2-norm of the result) of an output against float64 sums, over the
# listed cases at their full sizes and 30 drawn ones; about four times as much is stated.  The tensor core truncates when it
# accumulates, so the error of 3xTF32 grows with the length of a sum: 1e-6 for bmm, 7e-6 for fc, 1.3e-5 for resnet and
# dcgan, 3.8e-5 for the deltaW of sweep, 7.4e-5 (2.3e-4 once, 7x7 on 288 channels) for drawn layers; their bound stays
# under half of what plain TF32 operands show (7.8e-4 to 8.3e-4 everywhere).
_REL_3XTF32 = {"bmm": 1e-5, "fc": 3e-5, "resnet": 6e-5, "dcgan": 6e-5, "sweep": 1.5e-4, "conv": 3e-4, "act": 3e-4, "deconv": 3e-4}


def tolerance(case):
    if case["kind"] == "pool":
        return {"rel": 1e-6}      # maxima, indices and their gradient are exact; an average rounds once per addend (5e-8)
    rel = 3e-3 if case.get("math") == "tf32" else _REL_3XTF32[case["kind"]]
    return {"rel": rel, "max": 15 * rel}
