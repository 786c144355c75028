"""The register-tiled fp32 kernel: deltaX of channel counts the tensor-core paths do not take and batched products of ragged
sizes, within the bound of an fp32 sum of K products in any order, K * 2^-24 * sum |product|."""
import numpy as np
import pytest

from helpers import gen, out_hw

pytestmark = pytest.mark.gpu

# N, IH, IW, IC, OC, F, s, p: column tiles of 32, 64 and 128, row remainders, phases without a tap, split reductions
SHAPES = [
    (2, 35, 29, 36, 100, 3, 1, 1), (1, 9, 9, 4, 12, 3, 1, 1), (3, 16, 16, 132, 20, 3, 2, 1), (2, 15, 17, 64, 68, 1, 2, 0), (2, 9, 11, 40, 44, 2, 3, 0),
    (1, 6, 6, 260, 36, 4, 2, 1), (5, 1, 4, 52, 2764, 1, 1, 0), (1, 7, 5, 8, 4, 7, 2, 3), (2, 20, 20, 128, 36, 5, 1, 2), (40, 30, 30, 128, 44, 3, 2, 1),
]


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_fp32_deltaX(pkg, oracle_mod, shape, mode):
    import torch
    engine = pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    IH, IW = (OH - 1) * s + F - 2 * p, (OW - 1) * s + F - 2 * p
    rng = np.random.default_rng(IC * 1000 + OC)
    W, dY = gen((OC, F, F, IC), "u11", rng), gen((N, OH, OW, OC), "n01", rng)
    got = eng.dconv3D_deltaX(torch.from_numpy(dY).cuda(), torch.from_numpy(W).cuda(), IH, IW, s, s, p, p).cpu().numpy()
    ref, mag = oracle_mod.deconv3D_deltaX_f64(dY, W, IH, IW, s, s, p, p, threads=8)
    if OC % 32 and (s > 1 or OC % 8):
        assert pkg.submodule("lib").last_algo() == "simt" and pkg.submodule("lib").last_plan().startswith("gemm_f32")
        assert (np.abs(got - ref) <= F * F * OC * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("dims", [(2, 1, 1, 1), (3, 20, 20, 20), (2, 65, 33, 17), (2, 130, 129, 50), (1, 264, 425, 220), (5, 88, 79, 24), (2, 64, 128, 36)], ids=str)
def test_fp32_batched_products(pkg, dims):
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="tf32"))
    Bt, N, M, K = dims
    g = torch.Generator().manual_seed(Bt + N + M + K)
    A, B = torch.randn((Bt, N, K), generator=g), torch.randn((Bt, K, M), generator=g)
    ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    for op, a, b in (("batchMatMul", A, B), ("batchMatMulT1", A.transpose(1, 2).contiguous(), B), ("batchMatMulT2", A, B.transpose(1, 2).contiguous())):
        y = getattr(eng, op)(a.cuda(), b.cuda()).cpu().double()
        assert lib.last_algo() == "bmm_simt" and lib.last_plan().startswith("gemm_f32")
        assert bool(((y - ref).abs() <= K * 2.0 ** -24 * mag).all()), op


def test_padding_columns_and_neighbours_do_not_leak(pkg):
    """Row padding of A full of NaN, batch entries beside each other: only the first K columns count, only N x M is written."""
    import ctypes as C
    import torch
    lib = pkg.submodule("lib")
    L = lib.load()
    Bt, N, M, K, AK = 3, 21, 36, 18, 20
    A = torch.full((Bt, N, AK), float("nan"), device="cuda")
    A[..., :K] = torch.randn((Bt, N, K), device="cuda")
    B = torch.randn((Bt, K, M), device="cuda")
    out = torch.full((Bt * N * M + 64,), 7.0, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    lib.check(L.alpha_engine_batchMatMul(p(out), p(A), p(B), Bt, N, M, K, AK, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = out[:Bt * N * M].view(Bt, N, M).double()
    want = A[..., :K].double() @ B.double()
    assert bool(((got - want).abs() <= K * 2.0 ** -24 * (A[..., :K].double().abs() @ B.double().abs())).all())
    assert bool((out[Bt * N * M:] == 7.0).all())


def test_reduction_split_needs_no_scratch(pkg):
    """A call that never needed scratch still runs in a stream capture, which may not allocate any."""
    import torch
    eng = pkg.submodule("engine").Engine()
    dY, W = torch.randn((8, 1, 1, 2764), device="cuda"), torch.randn((2764, 1, 1, 52), device="cuda")
    want = eng.dconv3D_deltaX(dY, W, 1, 1, 1, 1, 0, 0)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        got = eng.dconv3D_deltaX(dY, W, 1, 1, 1, 1, 0, 0)
    graph.replay()
    torch.cuda.synchronize()
    mag = dY.double().abs().reshape(8, -1) @ W.double().abs().reshape(2764, 52)
    assert bool(((got.double() - want.double()).abs().reshape(8, 52) <= 2 * 2764 * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("algo", ["auto", "simt"])
@pytest.mark.parametrize("shape", [(2, 35, 29, 36, 100, 3, 1, 1), (2, 17, 17, 40, 36, 3, 2, 1), (1, 12, 12, 132, 44, 4, 2, 1), (3, 1, 4, 52, 1380, 1, 1, 0),
                                   (2, 10, 11, 8, 2060, 3, 1, 1)], ids=str)
def test_infinite_weight_reaches_only_the_pixels_of_its_tap(pkg, shape, algo):
    """A tap that falls outside the output is skipped, not multiplied by zero: border pixels of deltaX stay finite."""
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    eng = engine.Engine(engine.CudaFloat32EngineBase(algo=algo))
    N, OH, OW, IC, OC, F, s, p = shape
    IH, IW = (OH - 1) * s + F - 2 * p, (OW - 1) * s + F - 2 * p
    g = torch.Generator(device="cuda").manual_seed(OC)
    dY = torch.rand((N, OH, OW, OC), device="cuda", generator=g) + 0.5
    for oc, fh, fw, ic in ((0, 0, 0, 0), (OC - 1, F - 1, F - 1, IC - 1), (OC // 2, F // 2, 0, 5)):
        W = torch.randn((OC, F, F, IC), device="cuda", generator=g)
        W[oc, fh, fw, ic] = float("inf")
        dX = eng.dconv3D_deltaX(dY, W, IH, IW, s, s, p, p)
        ih, iw = torch.arange(IH, device="cuda") + p - fh, torch.arange(IW, device="cuda") + p - fw
        meets = ((ih >= 0) & (ih % s == 0) & (ih // s < OH))[:, None] & ((iw >= 0) & (iw % s == 0) & (iw // s < OW))
        want = torch.ones((N, IH, IW, IC), dtype=torch.bool, device="cuda")
        want[..., ic] = ~meets
        assert torch.equal(torch.isfinite(dX), want), (oc, fh, fw, ic)


# N, IH, IW, IC, OC, F, s, p: FH * FW * IC just above 16384 with a channel count that is no multiple of 8 (forward, deltaW) or 32 (deltaW)
@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", [(2, 9, 8, 660, 12, 5, 1, 2), (1, 15, 15, 404, 20, 7, 2, 3), (1, 5, 5, 16420, 8, 1, 1, 0)], ids=str)
def test_long_odd_reductions_stay_in_fp32(pkg, shape, mode):
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(IC)
    X, W = torch.randn((N, IH, IW, IC), device="cuda", generator=g), torch.randn((OC, F, F, IC), device="cuda", generator=g)
    dY = torch.randn((N, OH, OW, OC), device="cuda", generator=g)
    Y = eng.conv3D(X, W, s, s, p, p).double()
    assert lib.last_algo() == "simt"
    dW = eng.dconv3D_deltaW(X, dY, F, F, s, s, p, p).double()
    assert lib.last_algo() == "simt"
    conv = lambda x, w: torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), stride=s, padding=p).permute(0, 2, 3, 1)
    assert bool(((Y - conv(X.double(), W.double())).abs() <= F * F * IC * 2.0 ** -24 * conv(X.double().abs(), W.double().abs())).all())
    grad = lambda x, y: torch.nn.grad.conv2d_weight(x.permute(0, 3, 1, 2), (OC, IC, F, F), y.permute(0, 3, 1, 2), stride=s, padding=p).permute(0, 2, 3, 1)
    assert bool(((dW - grad(X.double(), dY.double())).abs() <= N * OH * OW * 2.0 ** -24 * grad(X.double().abs(), dY.double().abs()) + 1e-30).all())


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
def test_long_odd_matrix_product_stays_in_fp32(pkg, mode):
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    g = torch.Generator(device="cuda").manual_seed(1)
    A, B = torch.randn((40, 20004), device="cuda", generator=g), torch.randn((24, 20004), device="cuda", generator=g)
    C = eng.matMulT2(A, B).double()
    assert lib.last_algo() == "simt"
    assert bool(((C - A.double() @ B.double().T).abs() <= 20004 * 2.0 ** -24 * (A.double().abs() @ B.double().abs().T)).all())


def test_more_columns_than_a_grid_dimension(pkg):
    """67188 column tiles of 64: more than gridDim.y holds."""
    import torch
    eng, lib = pkg.submodule("engine").Engine(), pkg.submodule("lib")
    g = torch.Generator(device="cuda").manual_seed(2)
    A, B = torch.randn((4, 4), device="cuda", generator=g), torch.randn((4, 4300000), device="cuda", generator=g)
    C = eng.matMul(A, B)
    assert lib.last_algo() == "simt"
    assert bool(((C.double() - A.double() @ B.double()).abs() <= 4 * 2.0 ** -24 * (A.double().abs() @ B.double().abs())).all())


@pytest.mark.parametrize("shape", [(8, 1, 52, 2764, 1, 1), (4, 9, 20, 36, 3, 2), (3, 6, 132, 100, 3, 1)], ids=str)
def test_bits_do_not_depend_on_scratch(pkg, shape):
    """A reduction split into parts adds them up in the same order with a copy for each as without."""
    import torch
    eng = pkg.submodule("engine").Engine()
    N, OH, IC, OC, F, s = shape
    p = F // 2
    IH = (OH - 1) * s + F - 2 * p
    dY, W = torch.randn((N, OH, OH, OC), device="cuda"), torch.randn((OC, F, F, IC), device="cuda")
    want = eng.dconv3D_deltaX(dY, W, IH, IH, s, s, p, p)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()      # a fresh stream: no block yet
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        got = eng.dconv3D_deltaX(dY, W, IH, IH, s, s, p, p)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
