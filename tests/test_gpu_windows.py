"""Layers of few input channels as convolutions over windows of a filter row, forced for every shape that fits."""
import numpy as np
import pytest

from helpers import gen, metrics, out_hw

pytestmark = pytest.mark.gpu
TOL = {"3xtf32": dict(norm=1e-4, comp=1e-5), "tf32": dict(norm=5e-3, comp=2e-3)}   # the bounds of the other shape tests

# N, IH, IW, IC, OC, FH, FW, sh, sw, ph, pw: filters that do and do not divide by the stride, odd images, one stride only, no
# padding, windows of one chunk and of several, one window per pixel (FH <= sh), strides above the filter
SHAPES = [
    (3, 32, 32, 4, 64, 7, 7, 2, 2, 3, 3), (2, 33, 29, 4, 36, 7, 7, 2, 2, 3, 3), (2, 20, 22, 12, 64, 3, 3, 1, 1, 1, 1), (2, 17, 15, 36, 20, 3, 3, 2, 2, 1, 1),
    (2, 16, 16, 8, 128, 4, 4, 2, 2, 1, 1), (2, 12, 40, 4, 64, 2, 2, 2, 2, 0, 0), (2, 19, 13, 20, 44, 5, 5, 1, 1, 2, 2), (1, 30, 30, 4, 16, 3, 5, 2, 1, 0, 2),
    (1, 31, 31, 4, 32, 3, 3, 1, 3, 1, 1), (1, 26, 26, 8, 32, 3, 2, 4, 3, 1, 0), (5, 9, 9, 40, 100, 3, 3, 1, 1, 1, 1),
]


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_windows(pkg, oracle_mod, shape, mode):
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, FH, FW, sh, sw, ph, pw = shape
    OH, OW = out_hw(IH, IW, FH, FW, sh, sw, ph, pw)
    rng = np.random.default_rng(IH * 1000 + OC)
    X, W, B = gen((N, IH, IW, IC), "relu", rng), gen((OC, FH, FW, IC), "u11", rng), gen((OC,), "u11", rng)
    dY = gen((N, OH, OW, OC), "n01", rng)
    tX, tW, tB, tdY = (torch.from_numpy(a).cuda() for a in (X, W, B, dY))
    lib.set_option("HALO_WINDOW", 2)
    try:
        Y = eng.conv3D(tX, tW, sh, sw, ph, pw, Bias=tB).cpu().numpy()
        fwd = lib.last_plan()
        dW = eng.dconv3D_deltaW(tX, tdY, FH, FW, sh, sw, ph, pw).cpu().numpy()
        algo = lib.last_algo()
    finally:
        lib.set_option("HALO_WINDOW", 1)
    assert lib.device_status() == 0
    assert fwd.startswith("halo") and algo == "dw_window", (fwd, algo)
    ref, mag = oracle_mod.conv3D_f64(X, W, sh, sw, ph, pw, threads=8)
    for op, m in (("fwd", metrics(Y, ref + B, mag + np.abs(B))),
                  ("dw", metrics(dW, *oracle_mod.deconv3D_deltaW_f64(X, dY, FH, FW, sh, sw, ph, pw, threads=8)))):
        assert m["finite"] and m["norm"] <= TOL[mode]["norm"] and m["comp"] <= TOL[mode]["comp"], (op, m)


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", [(4, 40, 40, 3, 64, 7, 2, 3), (4, 41, 43, 4, 36, 3, 2, 1), (4, 40, 40, 8, 64, 4, 2, 1), (4, 30, 30, 12, 64, 5, 1, 2),
                                   (2, 41, 41, 4, 32, 3, 3, 0), (2, 40, 40, 4, 32, 5, 4, 1), (2, 30, 30, 4, 32, 2, 3, 0)], ids=str)
def test_one_infinite_pixel_reaches_only_its_own_outputs(pkg, shape, mode):
    """The rows and columns a window holds are those of the filter: an Inf pixel may not meet a zero weight beyond them."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, F, s, p = shape
    g = torch.Generator(device="cuda").manual_seed(IH)
    X, W = torch.randn((N, IH, IW, IC), device="cuda", generator=g), torch.rand((OC, F, F, IC), device="cuda", generator=g) + 0.5
    lib.set_option("HALO_WINDOW", 2)
    try:
        for n, ih, iw in ((0, 20, 21), (1, 21, 20), (1, 22, 23), (N - 1, IH - 1, IW - 1), (0, 0, 0)):
            Xi = X.clone()
            Xi[n, ih, iw, IC - 1] = float("inf")
            Y = eng.conv3D(Xi, W, s, s, p, p)
            assert lib.last_plan().startswith("halo")
            oh, ow = (torch.arange(d, device="cuda") for d in Y.shape[1:3])
            meets = ((ih + p - oh * s >= 0) & (ih + p - oh * s < F))[:, None] & ((iw + p - ow * s >= 0) & (iw + p - ow * s < F))
            want = torch.ones(Y.shape[:3], dtype=torch.bool, device="cuda")
            want[n] = ~meets
            assert torch.equal(torch.isfinite(Y).all(-1), want) and torch.equal(torch.isfinite(Y).any(-1), want), (n, ih, iw)
    finally:
        lib.set_option("HALO_WINDOW", 1)
    assert lib.device_status() == 0
