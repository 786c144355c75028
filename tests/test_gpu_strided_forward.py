"""Strided forward convolutions over the phases of the stride lattice (halo kernel), forced for every shape that fits."""
import numpy as np
import pytest

from helpers import gen, metrics, out_hw

pytestmark = pytest.mark.gpu
TOL = {"3xtf32": dict(norm=1e-4, comp=1e-5), "tf32": dict(norm=5e-3, comp=2e-3)}   # the bounds of the other shape tests

# N, IH, IW, IC, OC, FH, FW, sh, sw, ph, pw: odd images whose lattices differ in length, phases without a tap, one stride only,
# stacked images, channel tails, several column tiles, five taps in a row (three of a phase), padding beyond the lattice
SHAPES = [
    (3, 33, 31, 64, 64, 3, 3, 2, 2, 1, 1), (2, 56, 56, 32, 128, 3, 3, 2, 2, 1, 1), (2, 30, 30, 64, 48, 4, 4, 2, 2, 1, 1), (2, 17, 19, 96, 40, 1, 1, 2, 2, 0, 0),
    (2, 21, 20, 32, 300, 5, 5, 2, 2, 2, 2), (2, 16, 40, 44, 36, 2, 2, 2, 2, 0, 0), (4, 9, 9, 64, 32, 3, 3, 2, 2, 1, 1), (2, 24, 24, 32, 32, 3, 3, 2, 1, 1, 1),
    (2, 24, 24, 32, 32, 3, 3, 1, 2, 1, 1), (9, 13, 13, 128, 256, 3, 3, 2, 2, 1, 1), (1, 40, 1, 32, 16, 3, 1, 2, 2, 1, 0), (2, 15, 15, 32, 64, 3, 3, 2, 2, 2, 2),
    (2, 64, 64, 32, 256, 5, 3, 2, 2, 2, 1),
]


@pytest.mark.parametrize("mode", ["3xtf32", "tf32"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_strided_forward(pkg, oracle_mod, shape, mode):
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math=mode))
    N, IH, IW, IC, OC, FH, FW, sh, sw, ph, pw = shape
    rng = np.random.default_rng(IH * 1000 + OC)
    X, W, B = gen((N, IH, IW, IC), "relu", rng), gen((OC, FH, FW, IC), "u11", rng), gen((OC,), "u11", rng)
    lib.set_option("HALO_LATTICE", 2)
    lib.set_option("HALO_PAD", 2)
    try:
        got = eng.conv3D(*(torch.from_numpy(a).cuda() for a in (X, W)), sh, sw, ph, pw, Bias=torch.from_numpy(B).cuda()).cpu().numpy()
        algo = lib.last_algo()
    finally:
        lib.set_option("HALO_LATTICE", 1)
        lib.set_option("HALO_PAD", 1)
    assert lib.device_status() == 0
    OH, OW = out_hw(IH, IW, FH, FW, sh, sw, ph, pw)
    assert algo == "halo_lat" or OH * OW <= 16, algo
    ref, mag = oracle_mod.conv3D_f64(X, W, sh, sw, ph, pw, threads=8)
    m = metrics(got, ref + B, mag + np.abs(B))
    assert m["finite"] and m["norm"] <= TOL[mode]["norm"] and m["comp"] <= TOL[mode]["comp"], (algo, m)


def test_strided_forward_is_chosen_by_cost(pkg):
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    for shape, want in (((32, 112, 112, 128, 64), "halo_lat"), ((512, 16, 16, 64, 128), "igemm"), ((4, 16, 16, 32, 48), "igemm")):
        N, IH, IW, IC, OC = shape
        eng.conv3D(torch.zeros((N, IH, IW, IC), device="cuda"), torch.zeros((OC, 3, 3, IC), device="cuda"), 2, 2, 1, 1)
        assert lib.last_algo() == want, (shape, lib.last_algo())
