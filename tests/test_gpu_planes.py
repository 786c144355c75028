"""fp32 products as three bf16 planes on the tensor cores: against 64-bit sums at the edges of tiles, stages, taps and parts, and
against the FMA kernel where planes do not represent the operands.

Bound of a sum of K products: what is dropped of a product (two terms below 2^-25 of it, one below 2^-34), four truncated additions of
2^-23 for every 64 of them, and one rounded addition of 2^-24 for each such window and the small products."""
import numpy as np
import pytest

from helpers import gen, out_hw

pytestmark = pytest.mark.gpu


def bound(K):
    return 2.0 ** -24 + 2.0 ** -34 + 4 * 2.0 ** -23 + (K / 64 + 3) * 2.0 ** -24


@pytest.fixture
def planes(pkg):
    lib = pkg.submodule("lib")
    L = lib.load()
    lib.check(L.alpha_conv_set_option(b"F32_PLANES", 2))
    yield lambda v: lib.check(L.alpha_conv_set_option(b"F32_PLANES", v))
    lib.check(L.alpha_conv_set_option(b"F32_PLANES", 1))


# N, IH, IW, IC, OC, F, s, p: both column tiles and a remainder of each, one stage, half stages, odd and even windows, phases without
# a tap, rows past the last one, split reductions
DX = [(2, 35, 29, 36, 100, 3, 1, 1), (1, 9, 9, 4, 12, 3, 1, 1), (3, 16, 16, 132, 20, 3, 2, 1), (2, 15, 17, 64, 68, 1, 2, 0), (2, 9, 11, 40, 44, 2, 3, 0),
      (1, 6, 6, 260, 36, 4, 2, 1), (5, 1, 4, 52, 2764, 1, 1, 0), (1, 7, 5, 8, 4, 7, 2, 3), (2, 20, 20, 128, 36, 5, 1, 2), (1, 1, 1, 4, 4, 1, 1, 0),
      (130, 1, 1, 196, 180, 1, 1, 0)]


@pytest.mark.parametrize("shape", DX, ids=str)
def test_deltaX(pkg, oracle_mod, planes, shape):
    import torch
    eng = pkg.submodule("engine").Engine()
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    IH, IW = (OH - 1) * s + F - 2 * p, (OW - 1) * s + F - 2 * p
    rng = np.random.default_rng(IC * 1000 + OC)
    W, dY = gen((OC, F, F, IC), "n01", rng), gen((N, OH, OW, OC), "n01", rng)
    got = eng.dconv3D_deltaX(torch.from_numpy(dY).cuda(), torch.from_numpy(W).cuda(), IH, IW, s, s, p, p).cpu().numpy()
    ref, mag = oracle_mod.deconv3D_deltaX_f64(dY, W, IH, IW, s, s, p, p, threads=8)
    assert pkg.submodule("lib").last_plan().startswith("gemm_f32 planes")
    assert (np.abs(got - ref) <= bound(F * F * OC) * mag).all()


@pytest.mark.parametrize("dims", [(2, 1, 1, 1), (3, 20, 20, 20), (2, 65, 33, 17), (2, 130, 129, 50), (1, 264, 425, 220), (5, 88, 79, 24), (2, 64, 65, 36), (3, 128, 128, 97)], ids=str)
def test_batched_products(pkg, planes, dims):
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    Bt, N, M, K = dims
    g = torch.Generator().manual_seed(Bt + N + M + K)
    A, B = torch.randn((Bt, N, K), generator=g), torch.randn((Bt, K, M), generator=g)
    ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    for op, a, b in (("batchMatMul", A, B), ("batchMatMulT1", A.transpose(1, 2).contiguous(), B), ("batchMatMulT2", A, B.transpose(1, 2).contiguous())):
        y = getattr(eng, op)(a.cuda(), b.cuda()).cpu().double()
        assert lib.last_plan().startswith("gemm_f32 planes")
        assert bool(((y - ref).abs() <= bound(K) * mag).all()), op


def test_one_product(pkg, planes):
    """What is dropped of a single product (2^-24), and the two rounded additions of its small terms: less than 2^-22 in all.  Words cut
    instead of rounded lose 2^-21, 4.7e-7 of 1.0078124 squared."""
    import torch
    eng = pkg.submodule("engine").Engine()
    g = torch.Generator().manual_seed(4)
    A, B = torch.rand((3, 130, 1), generator=g) + 1, torch.rand((3, 1, 68), generator=g) + 1
    A[:, 0] = B[:, :, 0] = 1.0078124
    C = eng.batchMatMul(A.cuda(), B.cuda()).cpu().double()
    assert pkg.submodule("lib").last_plan().startswith("gemm_f32 planes")
    ref = A.double() * B.double()
    assert bool(((C - ref).abs() <= 2.0 ** -22 * ref).all())


@pytest.mark.parametrize("low", [0.0, 1.0])
def test_long_sums_of_one_sign(pkg, planes, low):
    """The four truncated additions of a window cost 2^-22 of it at most; those of the windows are rounded, to either side, and so are the
    small products: they grow with the square root of their number.  (Words cut instead of rounded: 1.2e-6 and 1.3e-6.)"""
    import torch
    eng = pkg.submodule("engine").Engine()
    K = 20001
    g = torch.Generator(device="cuda").manual_seed(5)
    A, B = torch.rand((2, 129, K), device="cuda", generator=g) + low, torch.rand((2, K, 65), device="cuda", generator=g) + low
    C = eng.batchMatMul(A, B).double()
    assert pkg.submodule("lib").last_plan().startswith("gemm_f32 planes")
    ref = A.double() @ B.double()
    assert float((C - ref).norm() / ref.norm()) <= 2.0 ** -22 + (K / 64) ** 0.5 * 2.0 ** -25


# (operands below 2^-110, whose last bits no bf16 word holds, times partners that make the sum an ordinary number)
TINY = [(1e-34, 1e8), (1e-36, 1e10), (1e-37, 1e11), (1e-39, 1e20)]


@pytest.mark.parametrize("small,large", TINY, ids=str)
@pytest.mark.parametrize("side", ["A", "B"])
def test_tiny_operands_with_large_partners(pkg, planes, small, large, side):
    """Batched products in each layout and fp32 deltaX with W split beforehand and not: within the bound of an fp32 sum."""
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    g = torch.Generator(device="cuda").manual_seed(6)
    sa, sb = (small, large) if side == "A" else (large, small)
    K = 97
    A, B = (torch.rand((2, 130, K), device="cuda", generator=g) + 0.5) * sa, (torch.rand((2, K, 68), device="cuda", generator=g) + 0.5) * sb
    ref = A.double() @ B.double()
    for op, a, b in (("batchMatMul", A, B), ("batchMatMulT1", A.transpose(1, 2).contiguous(), B), ("batchMatMulT2", A, B.transpose(1, 2).contiguous())):
        y = getattr(eng, op)(a, b).double()
        assert lib.last_plan().startswith("gemm_f32 planes")
        assert bool(((y - ref).abs() <= K * 2.0 ** -24 * ref).all()), op
    plans = []
    for N, OH, IC, OC in ((1, 9, 40, 44), (64, 14, 132, 36)):
        dY, W = (torch.rand((N, OH, OH, OC), device="cuda", generator=g) + 0.5) * sa, (torch.rand((OC, 3, 3, IC), device="cuda", generator=g) + 0.5) * sb
        y = eng.dconv3D_deltaX(dY, W, OH, OH, 1, 1, 1, 1).double()
        plans.append(lib.last_plan())
        assert plans[-1].startswith("gemm_f32 planes")
        ref = torch.nn.functional.conv_transpose2d(dY.double().permute(0, 3, 1, 2), W.double().permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
        assert bool(((y - ref).abs() <= 9 * OC * 2.0 ** -24 * ref).all()), plans[-1]
    assert "copy" not in plans[0] and "copy" in plans[1], plans


@pytest.mark.parametrize("what", ["inf weight", "nan gradient", "largest", "tiny", "overflow"])
def test_operands_outside_the_planes(pkg, planes, what):
    """Tiles with such operands are formed by FMAs: the values, Infs and NaNs of the FMA kernel, and border pixels untouched by taps
    that miss the output."""
    import torch
    eng = pkg.submodule("engine").Engine()
    N, H, IC, OC = 2, 17, 40, 100
    g = torch.Generator(device="cuda").manual_seed(3)
    W, dY = torch.randn((OC, 3, 3, IC), device="cuda", generator=g), torch.randn((N, H, H, OC), device="cuda", generator=g)
    big = torch.finfo(torch.float32).max
    if what == "inf weight":
        W[5, 2, 1, 7] = float("inf")
    elif what == "nan gradient":
        dY[1, 3, 4, 9] = float("nan")
    elif what == "largest":
        dY[0, 8, 8, :] = -big
        W *= 1e-3
    elif what == "tiny":
        dY *= 1e-34
    else:
        dY[0, 8, 8, :] = big
        W.abs_()
    out = []
    for mode in (0, 2):
        planes(mode)
        out.append(eng.dconv3D_deltaX(dY, W, H, H, 1, 1, 1, 1))
        assert pkg.submodule("lib").last_plan().startswith("gemm_f32 planes" if mode else "gemm_f32")
    a, b = out
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    ok = a.isfinite()
    scale = a[ok].abs().max().double() if what == "largest" else torch.nn.functional.conv_transpose2d(
        dY.double().abs().nan_to_num(0, 0, 0).permute(0, 3, 1, 2), W.double().abs().nan_to_num(0, 0, 0).permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)[ok]
    assert bool(((a[ok].double() - b[ok].double()).abs() <= 2 * 900 * 2.0 ** -24 * scale).all())
    if what == "inf weight":
        assert bool(b[:, 0].isfinite().all()) and bool(b[..., :7].isfinite().all())


# N, OH, IC, OC, F: a split reduction, W split beforehand, both, and a split reduction under a stride
@pytest.mark.parametrize("shape,words", [((130, 1, 132, 2764, 1, 1), {"ksplit"}), ((64, 14, 132, 36, 3, 1), {"copy"}), ((26, 14, 132, 1004, 3, 1), {"copy", "ksplit"}), ((4, 9, 20, 1036, 3, 2), {"ksplit"})],
                         ids=str)
def test_parts_give_the_same_bits_with_and_without_scratch(pkg, planes, shape, words):
    """A block of 256 bytes refuses all scratch: the parts then run in turns and add up in deltaX, and the kernel splits W itself."""
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    N, OH, IC, OC, F, s = shape
    p = F // 2
    IH = (OH - 1) * s + F - 2 * p
    g = torch.Generator(device="cuda").manual_seed(12)
    dY, W = torch.randn((N, OH, OH, OC), device="cuda", generator=g), torch.randn((OC, F, F, IC), device="cuda", generator=g)
    want = eng.dconv3D_deltaX(dY, W, IH, IH, s, s, p, p)
    plan = lib.last_plan()
    assert plan.startswith("gemm_f32 planes") and "in turns" not in plan, plan
    assert {word for word, used in (("copy", " copy" in plan), ("ksplit", "ksplit=1" not in plan.split())) if used} == words, plan
    stream, block = torch.cuda.Stream(), torch.empty(256, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    lib.set_workspace(stream.cuda_stream, block.data_ptr(), 256)
    try:
        with torch.cuda.stream(stream):
            got = eng.dconv3D_deltaX(dY, W, IH, IH, s, s, p, p)
        plan = lib.last_plan()
        stream.synchronize()
    finally:
        lib.set_workspace(stream.cuda_stream, 0, 0)
    assert plan.startswith("gemm_f32 planes") and "copy" not in plan and ("in turns" in plan) == ("ksplit" in words), plan
    assert torch.equal(got, want)


@pytest.mark.parametrize("op", ["batchMatMul", "batchMatMulT1", "batchMatMulT2"])
def test_tiny_rows_beside_ordinary_ones(pkg, planes, op):
    """Sums that stand although an operand lost bits, sums that do not, and zero rows and columns: what an fp32 sum gives."""
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    g = torch.Generator(device="cuda").manual_seed(11)
    N, M, K = 150, 70, 97
    for tails in (False, True):
        A, B = torch.randn((2, N, K), device="cuda", generator=g), torch.randn((2, K, M), device="cuda", generator=g)
        A[:, :, 5] = 3.3e-37
        A[:, 7], B[:, :, 9] = 0.0, 0.0
        if tails:
            A[0, 3] *= 1e-41
            A[1, 140] *= 1e-35
            B[1, :, 68] *= 1e-39
        ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
        a, b = A.transpose(1, 2).contiguous() if op == "batchMatMulT1" else A, B.transpose(1, 2).contiguous() if op == "batchMatMulT2" else B
        y = getattr(eng, op)(a, b).double()
        assert lib.last_plan().startswith("gemm_f32 planes")
        assert bool(((y - ref).abs() <= K * 2.0 ** -24 * mag + K * 2.0 ** -149).all())


def time_of(call):
    import torch
    for _ in range(3):
        call()
    best = float("inf")
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("what", ["inf", "1e-25", "1e-35", "tails"])
def test_time_of_tiles_formed_again(pkg, planes, what):
    """Tiles that the planes cannot form take some four to eight times as long (a form that read its operands anew for every step took 58 to
    280 times), gradients of 1e-25 and tails of a softmax none of that."""
    import torch
    eng = pkg.submodule("engine").Engine()
    g = torch.Generator(device="cuda").manual_seed(9)
    X, W = torch.randn((512, 8, 8, 128), device="cuda", generator=g), torch.randn((128, 3, 3, 128), device="cuda", generator=g) * 0.05
    A, B = torch.softmax(torch.randn((64, 250, 250), device="cuda", generator=g), -1), torch.randn((64, 250, 130), device="cuda", generator=g)
    usual = time_of(lambda: eng.batchMatMul(A, B)) if what == "tails" else time_of(lambda: eng.conv3D(X, W, 1, 1, 1, 1))
    assert pkg.submodule("lib").last_plan().startswith("gemm_f32 planes" if what == "tails" else "gather")
    if what == "tails":
        A[:, :, ::7] = 3.3e-37
        time = time_of(lambda: eng.batchMatMul(A, B))
    else:
        if what == "inf":
            X[:, 3, 4, 5] = float("inf")
        else:
            X *= float(what)
        time = time_of(lambda: eng.conv3D(X, W, 1, 1, 1, 1))
    assert time <= (1.1 if what == "1e-25" else 3 if what == "tails" else 16) * usual, (time, usual)


@pytest.mark.parametrize("op", ["batchMatMul", "batchMatMulT1"])
def test_what_lies_between_matrix_and_pitch(pkg, planes, op):
    """NaN in the columns between A and its pitch reaches neither the sums nor the time."""
    import ctypes as C
    import torch
    lib = pkg.submodule("lib")
    call = getattr(lib.load(), "alpha_engine_" + op)
    Bt, N, M, K = 40, 250, 132, 198
    p, stream = lambda t: C.c_void_p(t.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = []
    for pad in (0.0, float("nan")):
        g = torch.Generator(device="cuda").manual_seed(10)
        B, Y = torch.randn((Bt, K, M), device="cuda", generator=g), torch.zeros((Bt, N, M), device="cuda")
        A = torch.full((Bt, N, 200) if op == "batchMatMul" else (Bt, K, 252), pad, device="cuda")
        used = A[..., :K] if op == "batchMatMul" else A[..., :N]
        used.copy_(torch.randn(used.shape, device="cuda", generator=g))
        args = (Bt, N, M, K, 200) if op == "batchMatMul" else (Bt, N, 252, M, K)
        time = time_of(lambda: lib.check(call(p(Y), p(A), p(B), *args, stream)))
        assert lib.last_plan().startswith("gemm_f32 planes")
        want = (used if op == "batchMatMul" else used.transpose(1, 2)).double() @ B.double()
        assert float((Y.double() - want).norm() / want.norm()) <= 3e-7
        out.append((time, Y))
    assert torch.equal(out[0][1], out[1][1])
    assert out[1][0] <= 1.5 * out[0][0], (out[1][0], out[0][0])


# N, H, IC, OC, F, s, p: deltaW of odd channel counts whose rows are too long for a patch product, 1 to 8664 pixels
@pytest.mark.parametrize("shape", [(1, 2, 4100, 8, 2, 1, 0), (1, 6, 460, 8, 6, 1, 2), (2, 30, 700, 160, 7, 2, 3), (15, 8, 760, 160, 5, 1, 2), (24, 37, 508, 20, 7, 2, 3)], ids=str)
@pytest.mark.parametrize("data", ["relu", "n01"])
def test_long_deltaW_errs_no_more_than_the_fma_kernel(pkg, shape, data):
    """That one adds 128 lanes of K / 128 products in a tree: 7e-8 to 1.2e-7 against 64 bits, so that windows in one chain would not do."""
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    L = lib.load()
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    N, H, IC, OC, F, s, p = shape
    OH, OW = out_hw(H, H, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(H)
    X, dY = torch.randn((N, H, H, IC), device="cuda", generator=g), torch.randn((N, OH, OW, OC), device="cuda", generator=g)
    if data == "relu":
        X.relu_()
    ref = torch.nn.grad.conv2d_weight(X.double().permute(0, 3, 1, 2), (OC, IC, F, F), dY.double().permute(0, 3, 1, 2), stride=s, padding=p).permute(0, 2, 3, 1)
    err = {}
    for option in (0, 1):
        lib.check(L.alpha_conv_set_option(b"F32_PLANES", option))
        try:
            err[option] = float((eng.dconv3D_deltaW(X, dY, F, F, s, s, p, p).double() - ref).norm() / ref.norm())
        finally:
            lib.check(L.alpha_conv_set_option(b"F32_PLANES", 1))
        assert lib.last_algo() == "simt"
    assert N * OH * OW < 4 or lib.last_plan().startswith("gemm_f32 planes")
    assert err[1] <= err[0], err
