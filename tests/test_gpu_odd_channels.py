"""Channel counts that are no multiple of 32: zero-filled last chunks in the halo kernels and channel blocks of any multiple of
32 columns in deltaW, against the fp64 oracle, with the route chosen by cost (HALO_PAD = 1) and forced (2)."""
import re

import numpy as np
import pytest

from helpers import gen, metrics, out_hw

pytestmark = pytest.mark.gpu
TOL = {"3xtf32": dict(norm=1e-4, comp=1e-5), "tf32": dict(norm=5e-3, comp=2e-3)}   # the bounds of the other shape tests

# N, IH, IW, IC, OC, FH, FW, s, p: remainders 4 ... 28 of a chunk, one chunk and several, blocks of 96 and 160 columns, tails in
# the kernel forms that test_forms_of_zero_filled_chunks names
SHAPES = [
    (3, 35, 29, 36, 100, 3, 3, 1, 1), (2, 18, 18, 40, 64, 3, 3, 1, 1), (4, 20, 20, 16, 32, 3, 3, 1, 1), (2, 16, 16, 8, 128, 3, 3, 1, 1),
    (4, 28, 28, 60, 128, 3, 3, 1, 1), (2, 14, 14, 132, 256, 3, 3, 1, 1), (2, 13, 11, 92, 48, 5, 5, 1, 2), (3, 17, 15, 100, 72, 1, 1, 1, 0),
    (2, 24, 24, 96, 96, 3, 3, 1, 1), (2, 16, 16, 192, 40, 3, 3, 1, 1), (2, 12, 12, 320, 64, 3, 3, 1, 1), (2, 33, 31, 44, 20, 3, 3, 2, 1),
    (2, 17, 17, 72, 36, 3, 3, 2, 1), (1, 5, 5, 420, 24, 3, 3, 1, 1), (2, 16, 16, 68, 68, 4, 4, 2, 1), (1, 8, 8, 1028, 8, 1, 1, 1, 0),
    (2, 112, 112, 36, 48, 3, 3, 1, 1),
]


@pytest.mark.parametrize("pad", [1, 2])
@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_zero_filled_chunks(pkg, oracle_mod, shape, mode, pad):
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, FH, FW, s, p = shape
    OH, OW = out_hw(IH, IW, FH, FW, s, s, p, p)
    rng = np.random.default_rng(IC * 1000 + OC)
    X, W, dY = gen((N, IH, IW, IC), "relu", rng), gen((OC, FH, FW, IC), "u11", rng), gen((N, OH, OW, OC), "n01", rng)
    tX, tW, tdY = (torch.from_numpy(a).cuda() for a in (X, W, dY))
    lib.set_option("HALO_PAD", pad)
    try:
        got, algo = {"fwd": eng.conv3D(tX, tW, s, s, p, p)}, {}
        algo["fwd"] = lib.last_algo()
        got["dw"] = eng.dconv3D_deltaW(tX, tdY, FH, FW, s, s, p, p)
        algo["dw"] = lib.last_algo()
        ref = {"fwd": oracle_mod.conv3D_f64(X, W, s, s, p, p, threads=8), "dw": oracle_mod.deconv3D_deltaW_f64(X, dY, FH, FW, s, s, p, p, threads=8)}
        if (IH + 2 * p - FH) % s == 0 and (IW + 2 * p - FW) % s == 0:
            got["dx"] = eng.dconv3D_deltaX(tdY, tW, IH, IW, s, s, p, p)
            ref["dx"] = oracle_mod.deconv3D_deltaX_f64(dY, W, IH, IW, s, s, p, p, threads=8)
    finally:
        lib.set_option("HALO_PAD", 1)
    assert lib.device_status() == 0
    if pad == 2 and IC % 32:       # forced: no patch matrix (a strided forward, and 8-channel steps in tiles under 0.6 full, have the im2col kernel)
        assert algo["dw"] == "dw_halo" and (s > 1 or IC % 8 == 0 or algo["fwd"].startswith("halo")), algo
    for op, y in got.items():
        m = metrics(y.cpu().numpy(), *ref[op])
        assert m["finite"] and m["norm"] <= TOL[mode]["norm"] and m["comp"] <= TOL[mode]["comp"], (op, m)


def test_forms_of_zero_filled_chunks(pkg):
    """Over the shapes above, zero-filled chunks meet every form of the kernels."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    plans = []
    lib.set_option("HALO_PAD", 2)
    lib.set_option("HALO_TAPSTACK", 2)      # wherever the tap-stacked kernel fits (plain TF32)
    try:
        for mode in ("3xtf32", "tf32"):
            eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
            for N, IH, IW, IC, OC, FH, FW, s, p in SHAPES:
                if IC % 32 == 0:
                    continue
                OH, OW = out_hw(IH, IW, FH, FW, s, s, p, p)
                X = torch.zeros((N, IH, IW, IC), device="cuda")
                eng.conv3D(X, torch.zeros((OC, FH, FW, IC), device="cuda"), s, s, p, p)
                plans.append(lib.last_plan())
                eng.dconv3D_deltaW(X, torch.zeros((N, OH, OW, OC), device="cuda"), FH, FW, s, s, p, p)
                plans.append(lib.last_plan())
    finally:
        lib.set_option("HALO_PAD", 1)
        lib.set_option("HALO_TAPSTACK", 1)
    forms = {"CTA pairs": "halo_pair", "single CTA": "halo_row", "tap-stacked": "tapstack", "split reduction": "ksplit=([2-9]|1[0-9])", "strided deltaW": "dw_halo.* strided",
             "tap groups": "tap groups", "stacked planes": "dw_halo stacked", "two half tiles": "dw_halo diagonal"}
    missing = [f for f, text in forms.items() if not any(re.search(text, q) for q in plans)]
    assert not missing, (missing, sorted(set(q.split(" R=")[0].split(" npb")[0] for q in plans)))


def test_long_odd_reductions_keep_their_corrections_apart(pkg):
    """A product over 6148 channels (no multiple of 8) of a row count that is none either stays on the halo kernel, whose side
    columns hold the correction terms: the im2col kernel's single accumulator errs four times as much (4e-5)."""
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    g = torch.Generator(device="cuda").manual_seed(5)
    A, B = torch.randn((995, 6146), device="cuda", generator=g), torch.randn((73, 6146), device="cuda", generator=g)
    C = eng.matMulT2(A, B)
    assert lib.last_algo().startswith("halo"), lib.last_algo()
    ref = A.double() @ B.double().T
    assert float((C.double() - ref).norm() / ref.norm()) <= 3e-5      # the bound stated for FullConnect layers


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", [(4, 35, 29, 36, 100, 3, 1, 1), (3, 21, 27, 4, 64, 5, 1, 2), (3, 33, 31, 44, 68, 3, 2, 1), (2, 19, 18, 12, 132, 7, 2, 3),
                                   (2, 13, 37, 100, 72, 3, 1, 0)], ids=str)
def test_infinite_border_pixel_reaches_only_its_own_taps(pkg, shape, mode):
    """Pixel tiles of deltaW reach past the output, where deltaY is zero but X can still have pixels: an Inf among those may not
    make deltaW NaN at taps that never meet it.  Every route of an odd channel count, with the other elements exact."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IW, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(IH * IC)
    X, dY = torch.randn((N, IH, IW, IC), device="cuda", generator=g), torch.rand((N, OH, OW, OC), device="cuda", generator=g) + 0.5
    pad = torch.nn.functional.pad(X.double(), (0, 0, p, p, p, p))
    cut = lambda t, i, j: t[:, i:i + (OH - 1) * s + 1:s, j:j + (OW - 1) * s + 1:s]
    for route in ({"HALO_PAD": 2}, {"HALO_WINDOW": 2}, {}):
        for k, v in route.items():
            lib.set_option(k, v)
        try:
            for n, ih, iw in ((1, IH - 1, IW - 1), (0, IH - 1, 3), (N - 1, 2, IW - 2), (1, IH // 2, IW // 2)):
                Xi = X.clone()
                Xi[n, ih, iw, 1] = float("inf")
                dW = eng.dconv3D_deltaW(Xi, dY, F, F, s, s, p, p)
                for i in range(F):
                    for j in range(F):
                        oh, ow = ih + p - i, iw + p - j
                        meets = oh % s == 0 and ow % s == 0 and 0 <= oh // s < OH and 0 <= ow // s < OW
                        fin = torch.isfinite(dW[:, i, j])
                        assert bool(fin[:, 1].all()) != meets and bool(fin[:, 1].any()) != meets, (route, (n, ih, iw), i, j)
                        ok = [c for c in range(IC) if c != 1]
                        assert bool(fin[:, ok].all())
                        ref = torch.einsum("nhwo,nhwc->oc", dY.double(), cut(pad, i, j))
                        scale = torch.einsum("nhwo,nhwc->oc", dY.double(), cut(pad, i, j).abs())
                        assert float(((dW[:, i, j].double() - ref).abs() / scale)[:, ok].max()) <= TOL[mode]["comp"]
        finally:
            for k in route:
                lib.set_option(k, 1)
    assert lib.device_status() == 0


@pytest.mark.parametrize("shape", [(64, 14, 14, 148, 64, 3, 1, 1), (8, 28, 28, 68, 128, 5, 1, 2), (8, 28, 28, 20, 48, 5, 1, 2), (32, 16, 16, 100, 64, 3, 2, 1)], ids=str)
def test_small_layers_err_no_more_than_the_patch_product(pkg, shape):
    """Where the product over the patch matrix splits its reduction over idle SMs, a route with longer sums is not taken: the
    2-norm error of the default route is at most that of the patch product (a quarter more for sums in another order)."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    N, IH, IW, IC, OC, F, s, p = shape
    g = torch.Generator(device="cuda").manual_seed(IC)
    X, W = torch.randn((N, IH, IW, IC), device="cuda", generator=g).relu_(), torch.randn((OC, F, F, IC), device="cuda", generator=g)
    ref = torch.nn.functional.conv2d(X.double().permute(0, 3, 1, 2), W.double().permute(0, 3, 1, 2), stride=s, padding=p).permute(0, 2, 3, 1)
    err = {}
    for pad in (1, 0):
        lib.set_option("HALO_PAD", pad)
        try:
            err[pad] = float((eng.conv3D(X, W, s, s, p, p).double() - ref).norm() / ref.norm())
        finally:
            lib.set_option("HALO_PAD", 1)
    assert err[1] <= 1.25 * err[0], err


# N, IH, IC, OC, F, s, p and the options of the route whose error is the measure: the patch product of an odd channel count, the
# stacked planes of whole chunks (a block of 96 or 128 columns would be cheaper unstacked, in sums of the same or twice the length)
@pytest.mark.parametrize("shape,former", [((50, 35, 12, 64, 3, 1, 1), {"HALO_WINDOW": 0, "HALO_PAD": 0}), ((64, 32, 4, 100, 4, 2, 1), {"HALO_WINDOW": 0, "HALO_PAD": 0}),
                                          ((64, 14, 68, 64, 3, 1, 1), {"HALO_WINDOW": 0, "HALO_PAD": 0}), ((8, 28, 352, 256, 5, 1, 2), {"DW_STACKED": 1}),
                                          ((32, 28, 192, 128, 3, 1, 1), {"DW_STACKED": 1})], ids=str)
def test_deltaW_errs_no_more_than_its_former_route(pkg, shape, former):
    """The steps one accumulator takes bound the truncation error of a 3xTF32 deltaW: forms with fewer parts or without stacked
    planes get more parts, or give way (a quarter more for sums in another order)."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    N, IH, IC, OC, F, s, p = shape
    OH, OW = out_hw(IH, IH, F, F, s, s, p, p)
    g = torch.Generator(device="cuda").manual_seed(IC)
    X, dY = torch.randn((N, IH, IH, IC), device="cuda", generator=g).relu_(), torch.randn((N, OH, OW, OC), device="cuda", generator=g)
    pad = torch.nn.functional.pad(X, (0, 0, p, p, p, p))
    ref = torch.stack([torch.stack([dY.double().reshape(-1, OC).T @ pad[:, i:i + (OH - 1) * s + 1:s, j:j + (OW - 1) * s + 1:s].double().reshape(-1, IC)
                                    for j in range(F)], 1) for i in range(F)], 1)
    err = []
    for options in ({}, former):
        saved = {k: lib.get_option(k) for k in options}
        for k, v in options.items():
            lib.set_option(k, v)
        try:
            err.append(float((eng.dconv3D_deltaW(X, dY, F, F, s, s, p, p).double() - ref).norm() / ref.norm()))
        finally:
            for k, v in saved.items():
                lib.set_option(k, v)
    assert err[0] <= 1.25 * err[1], err
