"""Layers gathered straight from their tensors by the bf16-plane kernel: against 64-bit sums at the edges of tiles, stages, taps and
parts, which layers take that route, and that it gives the same bits under every option that must not change a result.

Bound of a sum of K products: that of test_gpu_planes, and one rounded addition of 2^-24 for each of up to 16 parts (the more parts of a deltaW are added with compensation)."""
import numpy as np
import pytest

from helpers import gen, out_hw

pytestmark = pytest.mark.gpu


def bound(K):
    return 2.0 ** -24 + 2.0 ** -34 + 4 * 2.0 ** -23 + (K / 64 + 3 + 16) * 2.0 ** -24


@pytest.fixture
def gather(pkg):
    lib = pkg.submodule("lib")
    lib.set_math_mode("3xtf32")
    set_option = lambda v: lib.check(lib.load().alpha_conv_set_option(b"GATHER", v))
    set_option(2)
    yield set_option
    set_option(1)


# N, IH, IW, IC, OC, F, s, p: both column tiles and remainders of each, one product, one stage and its remainders, split reductions and W split
# beforehand or in the kernel, taps outside the picture on every side, phases without a tap
SHAPES = [(1, 1, 1, 4, 4, 1, 1, 0), (1, 9, 9, 4, 12, 3, 1, 1), (2, 35, 29, 36, 100, 3, 1, 1), (3, 16, 16, 132, 20, 3, 2, 1), (2, 15, 17, 64, 68, 1, 2, 0),
          (2, 9, 11, 40, 44, 2, 3, 0), (1, 6, 6, 260, 36, 4, 2, 1), (130, 1, 1, 196, 180, 1, 1, 0), (5, 1, 1, 2764, 52, 1, 1, 0), (1, 7, 5, 8, 4, 7, 2, 3),
          (16, 8, 8, 128, 128, 3, 1, 1), (64, 4, 4, 64, 256, 3, 2, 1), (2, 20, 20, 128, 36, 5, 1, 2), (300, 28, 28, 24, 72, 3, 1, 1), (37, 31, 29, 36, 100, 3, 1, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_operators(pkg, oracle_mod, gather, shape):
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    rng = np.random.default_rng(IC * 1000 + OC)
    X, W, dY = gen((N, IH, IW, IC), "n01", rng), gen((OC, F, F, IC), "n01", rng), gen((N, OH, OW, OC), "n01", rng)
    bias = gen((OC,), "n01", rng)
    Xd, Wd, Yd, bd = (torch.from_numpy(t).cuda() for t in (X, W, dY, bias))
    ref, mag = oracle_mod.conv3D_f64(X, W, s, s, p, p, threads=8)
    got = eng.conv3D(Xd, Wd, s, s, p, p)
    assert lib.last_plan().startswith("gather")
    assert (np.abs(got.cpu().numpy() - ref) <= bound(F * F * IC) * mag).all()
    act = eng.conv3D_leakyRelu(Xd, Wd, bd, 0.25, s, s, p, p).cpu().numpy()
    ref, mag = ref + bias, mag + np.abs(bias)
    assert (np.abs(act - np.where(ref > 0, ref, 0.25 * ref)) <= bound(F * F * IC) * mag).all()
    got = eng.dconv3D_deltaX(Yd, Wd, IH, IW, s, s, p, p)
    if OC % (8 if s == 1 else 32) == 0:
        assert lib.last_plan().startswith("gather")
    if (IH + 2 * p - F) % s == 0 and (IW + 2 * p - F) % s == 0:
        ref, mag = oracle_mod.deconv3D_deltaX_f64(dY, W, IH, IW, s, s, p, p, threads=8)
    else:                                                          # rows and columns past the last window, which the oracle does not have: zeros
        grad = lambda w, y: torch.nn.grad.conv2d_input((N, IC, IH, IW), torch.from_numpy(w).double().permute(0, 3, 1, 2), torch.from_numpy(y).double().permute(0, 3, 1, 2),
                                                       stride=s, padding=p).permute(0, 2, 3, 1).numpy()
        ref, mag = grad(W, dY), grad(np.abs(W), np.abs(dY))
    assert (np.abs(got.cpu().numpy() - ref) <= bound(F * F * OC) * mag).all()
    got = eng.dconv3D_deltaW(Xd, Yd, F, F, s, s, p, p)
    assert lib.last_plan().startswith("gather")
    ref, mag = oracle_mod.deconv3D_deltaW_f64(X, dY, F, F, s, s, p, p, threads=8)
    assert (np.abs(got.cpu().numpy() - ref) <= bound(N * OH * OW) * mag).all()
    both, dB = eng.dconv3D_deltaW_bias(Xd, Yd, F, F, s, s, p, p)
    assert torch.equal(both, got)
    assert torch.allclose(dB.double(), Yd.double().sum((0, 1, 2)), rtol=1e-5, atol=1e-5 * Yd.abs().sum((0, 1, 2)).max().item())
    assert lib.load().alpha_conv_device_status() == 0


@pytest.mark.parametrize("op", ["forward", "deltaW"])
@pytest.mark.parametrize("what", ["inf", "nan", "largest", "tiny"])
def test_operands_outside_the_planes(pkg, gather, op, what):
    """Tiles with such operands are formed by FMAs: Infs and NaNs where the sums have them, and no others."""
    import torch
    eng = pkg.submodule("engine").Engine()
    N, H, IC, OC = 2, 17, 40, 100
    g = torch.Generator(device="cuda").manual_seed(3)
    X, W, dY = (torch.randn(s, device="cuda", generator=g) for s in ((N, H, H, IC), (OC, 3, 3, IC), (N, H, H, OC)))
    if what == "tiny":
        X *= 1e-34
    elif what == "largest":
        X[0, 8, 8, :] = -torch.finfo(torch.float32).max
        W *= 1e-3
        dY *= 1e-3
    else:
        X[1, 3, 4, 9] = float(what)
    conv = lambda x, w: torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
    grad = lambda x, y: torch.nn.grad.conv2d_weight(x.permute(0, 3, 1, 2), (OC, IC, 3, 3), y.permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
    if op == "forward":
        got, ref, mag = eng.conv3D(X, W, 1, 1, 1, 1), conv(X.double(), W.double()), conv(X.double().abs().nan_to_num(0, 0, 0), W.double().abs())
    else:
        got, ref, mag = eng.dconv3D_deltaW(X, dY, 3, 3, 1, 1, 1, 1), grad(X.double(), dY.double()), grad(X.double().abs().nan_to_num(0, 0, 0), dY.double().abs())
    assert pkg.submodule("lib").last_plan().startswith("gather")
    finite = ref.isfinite()
    if what in ("inf", "nan"):
        assert bool((got.isfinite() == finite).all())
    K = 360 if op == "forward" else N * H * H
    assert bool(((got.double() - ref).abs()[finite] <= (K * 2.0 ** -24 * mag + K * 2.0 ** -149)[finite]).all())


@pytest.mark.parametrize("small,large", [(1e-36, 1e10), (1e-37, 1e11)], ids=str)
@pytest.mark.parametrize("side", ["X", "W"])
def test_tiny_operands_with_large_partners(pkg, gather, small, large, side):
    """Operands whose last bits no bf16 word holds, in sums that do not show it: forward (W split beforehand and not), deltaX, deltaW."""
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    g = torch.Generator(device="cuda").manual_seed(8)
    sx, sw = (small, large) if side == "X" else (large, small)
    rand = lambda *q: torch.rand(q, device="cuda", generator=g) + 0.5
    plans = []
    for N, H, IC, OC in ((1, 9, 36, 40), (256, 14, 64, 128)):
        X, W = rand(N, H, H, IC) * sx, rand(OC, 3, 3, IC) * sw
        y = eng.conv3D(X, W, 1, 1, 1, 1).double()
        plans.append(lib.last_plan())
        ref = torch.nn.functional.conv2d(X.double().permute(0, 3, 1, 2), W.double().permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
        assert bool(((y - ref).abs() <= 9 * IC * 2.0 ** -24 * ref).all()), plans[-1]
        dY, V = rand(N, H, H, IC) * sx, rand(IC, 3, 3, OC) * sw
        y = eng.dconv3D_deltaX(dY, V, H, H, 1, 1, 1, 1).double()
        ref = torch.nn.functional.conv_transpose2d(dY.double().permute(0, 3, 1, 2), V.double().permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
        assert bool(((y - ref).abs() <= 9 * IC * 2.0 ** -24 * ref).all()), lib.last_plan()
    assert all(q.startswith("gather") for q in plans) and "copy" not in plans[0] and "copy" in plans[1], plans
    dY = rand(2, 9, 9, 40) * sw
    X = rand(2, 9, 9, 36) * sx
    y = eng.dconv3D_deltaW(X, dY, 3, 3, 1, 1, 1, 1).double()
    ref = torch.nn.grad.conv2d_weight(X.double().permute(0, 3, 1, 2), (40, 36, 3, 3), dY.double().permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
    assert lib.last_plan().startswith("gather") and bool(((y - ref).abs() <= 162 * 2.0 ** -24 * ref).all())


# the smallest fill, channel count and time at which a layer leaves the other kernels, and its neighbours
ROUTES = [("forward", (512, 8, 8, 128, 128, 3, 1, 1), True), ("forward", (512, 14, 14, 128, 128, 3, 1, 1), False), ("forward", (8, 8, 8, 32, 64, 3, 1, 1), False),
          ("forward", (64, 28, 28, 12, 64, 3, 1, 1), False), ("forward", (512, 8, 8, 256, 512, 3, 2, 1), True), ("forward", (512, 16, 16, 64, 128, 3, 2, 1), False),
          ("forward", (64, 15, 13, 36, 100, 3, 1, 1), True), ("forward", (2, 5, 5, 36, 100, 3, 1, 1), False), ("forward", (250, 1, 1, 1024, 1024, 1, 1, 0), True),
          ("forward", (256, 16, 16, 128, 256, 4, 2, 1), True), ("forward", (64, 7, 7, 512, 512, 3, 1, 1), True), ("forward", (256, 7, 7, 512, 512, 3, 1, 1), False),
          ("deltaX", (256, 16, 16, 128, 256, 4, 2, 1), True), ("deltaX", (256, 16, 16, 32, 256, 4, 2, 1), False), ("deltaX", (512, 8, 8, 128, 128, 3, 1, 1), True), ("deltaX", (512, 14, 14, 128, 128, 3, 1, 1), False), ("deltaX", (512, 4, 4, 256, 512, 3, 2, 1), False),
          ("deltaX", (250, 1, 1, 1024, 1024, 1, 1, 0), True), ("deltaW", (512, 4, 4, 256, 256, 3, 1, 1), True), ("deltaW", (512, 8, 8, 128, 128, 3, 1, 1), False), ("deltaW", (33, 21, 21, 128, 192, 7, 2, 3), True),
          ("deltaW", (256, 16, 16, 128, 256, 4, 2, 1), False),
          ("deltaW", (7, 28, 28, 28, 88, 3, 1, 1), True), ("deltaW", (50, 35, 29, 36, 100, 3, 1, 1), True), ("deltaW", (250, 1, 1, 1024, 1024, 1, 1, 0), True), ("deltaW", (64, 1, 1, 4096, 1024, 1, 1, 0), False)]


@pytest.mark.parametrize("op,shape,taken", ROUTES, ids=str)
def test_route(pkg, gather, op, shape, taken):
    """In 3xTF32 by the layer alone: prepared weights, the weight cache, a limit on SMs and a capture keep the route or, where scratch
    is refused, the result to rounding; in TF32 and with the option off the layer stays."""
    import ctypes as C
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    L = lib.load()
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(7)
    X, W, dY = (torch.randn(q, device="cuda", generator=g) for q in ((N, IH, IW, IC), (OC, F, F, IC), (N, OH, OW, OC)))
    base = engine.CudaFloat32EngineBase(math="3xtf32")

    def call(math="3xtf32"):
        eng = engine.Engine(base if math == "3xtf32" else engine.CudaFloat32EngineBase(math=math))
        if op == "forward":
            return eng.conv3D(X, W, s, s, p, p)
        return eng.dconv3D_deltaX(dY, W, IH, IW, s, s, p, p) if op == "deltaX" else eng.dconv3D_deltaW(X, dY, F, F, s, s, p, p)

    gather(0)
    other = call()
    assert lib.last_algo() != "gather"
    gather(1)
    got = call()
    assert (lib.last_algo() == "gather") == taken
    # (either side errs by no more than 2e-5 of the largest of the result: 3xTF32 chains of up to 4096 products)
    assert float((got - other).abs().max()) <= 4e-5 * float(other.abs().max())
    call("tf32")
    assert lib.last_algo() != "gather"
    if not taken:
        return
    old = lib.set_option("SM_BUDGET", 74)
    try:
        assert torch.equal(call(), got)
    finally:
        lib.set_option("SM_BUDGET", old)
    lib.check(L.alpha_conv_weight_cache(1))
    try:
        assert torch.equal(call(), got)
    finally:
        lib.check(L.alpha_conv_weight_cache(0))
    if op != "deltaW":
        assert base.prepare_weights(op, W, F, F, N, IH, IW, OH, OW, IC, OC, s, s, p, p) is None
    ran = []
    for option in (0, 1):                                          # a fresh stream: no block to take scratch from
        gather(option)
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            try:
                again = call()
                ran.append(True)
            except lib.AlphaConvError:
                ran.append(False)
    assert ran[1] or not ran[0]
    if ran[1]:
        graph.replay()
        torch.cuda.synchronize()
        assert float((again - other).abs().max()) <= 4e-5 * float(other.abs().max())
    assert L.alpha_conv_device_status() == 0


# split reductions and W split beforehand, whose scratch a capture on a new stream refuses; the other routes need scratch for the transform of W alone
PREPARED = [("forward", (512, 8, 8, 128, 128, 3, 1, 1)), ("forward", (64, 15, 13, 36, 100, 3, 1, 1)), ("forward", (16, 8, 8, 256, 256, 3, 1, 1)),
            ("deltaX", (512, 8, 8, 128, 128, 3, 1, 1)), ("deltaX", (250, 1, 1, 1024, 1024, 1, 1, 0)), ("deltaX", (16, 8, 8, 256, 256, 3, 1, 1))]


@pytest.mark.parametrize("op,shape", PREPARED, ids=str)
def test_prepared_layers_are_captured_on_a_new_stream(pkg, gather, op, shape):
    """With weights prepared for them such layers needed no scratch on the other kernels; gathered, they have no prepared weights, and run without."""
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(9)
    X, W, dY = (torch.randn(q, device="cuda", generator=g) for q in ((N, IH, IW, IC), (OC, F, F, IC), (N, OH, OW, OC)))
    base = engine.CudaFloat32EngineBase(math="3xtf32")
    got = {}
    for option in (0, 1):
        gather(option)
        block = base.prepare_weights(op, W, F, F, N, IH, IW, OH, OW, IC, OC, s, s, p, p)

        def call():
            out = torch.empty_like(dY if op == "forward" else X)
            if op == "forward":
                base.conv3D_prepared(out, OH, OW, X, IH, IW, W, F, F, N, IC, OC, s, s, p, p, block)
            else:
                base.dconv3D_deltaX_prepared(out, IH, IW, dY, OH, OW, W, F, F, N, IC, OC, s, s, p, p, block)
            return out

        eager = call()
        assert (lib.last_algo() == "gather") == (option == 1)
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            got[option] = call()
        if option:
            assert lib.last_plan().startswith("gather")
        graph.replay()
        torch.cuda.synchronize()
        if op == "deltaX" and option:
            assert torch.equal(got[option], eager)               # (forwards, of both sides, add their products up in fewer parts)
    assert float((got[1] - got[0]).abs().max()) <= 4e-5 * float(got[0].abs().max())
    assert lib.device_status() == 0


def test_blocks_that_are_not_the_layers_are_refused(pkg, gather):
    """A block serves every batch of its layer, those that are gathered (512) and need none among them; made for another operator, tensor or math
    mode, or cut short, it is refused whatever the batch."""
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    base = engine.CudaFloat32EngineBase()
    C, H = 128, 8
    g = torch.Generator(device="cuda").manual_seed(11)
    W, V = (torch.randn((C, 3, 3, C), device="cuda", generator=g) for _ in range(2))
    gather(1)

    def call(op, n, block, w=W):
        x, out = torch.ones((n, H, H, C), device="cuda"), torch.empty((n, H, H, C), device="cuda")
        (base.conv3D_prepared if op == "forward" else base.dconv3D_deltaX_prepared)(out, H, H, x, H, H, w, 3, 3, n, C, C, 1, 1, 1, 1, block)
        return out

    make = lambda op, n, w=W: base.prepare_weights(op, w, 3, 3, n, H, H, H, H, C, C, 1, 1, 1, 1)
    blocks = {op: make(op, 8) for op in ("forward", "deltaX")}
    others = {op: make(op, 8, V) for op in blocks}
    lib.set_math_mode("tf32")
    plain = make("deltaX", 8)
    lib.set_math_mode("3xtf32")
    for op in blocks:
        for n in (8, 512):
            want = call(op, n, None)
            assert (lib.last_algo() == "gather") == (n == 512)
            assert torch.equal(call(op, n, blocks[op]), want)
            for bad in (blocks["deltaX" if op == "forward" else "forward"], others[op], blocks[op][:256]) + ((plain,) if op == "deltaX" else ()):
                with pytest.raises(lib.AlphaConvError):
                    call(op, n, bad)
    # a layer without a transform, prepared into memory that held another's
    L = lib.load()
    import ctypes
    shape = lib.AlphaConvShape(512, H, H, C, C, 3, 3, H, H, 1, 1, 1, 1)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    old = others["forward"]
    assert lib.prepared_weights_bytes(shape, "forward") == 0
    lib.check(L.alpha_conv_prepare_weights(ctypes.byref(shape), lib.OPS["forward"], p(W), p(old), old.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(call("forward", 512, old), call("forward", 512, None))
