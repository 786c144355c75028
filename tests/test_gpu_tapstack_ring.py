"""The tap-stacked kernel (plain TF32, few output channels) where its two issuing threads share a ring of fewer patches than a tile has
chunks, or as many: neither may take a slot's earlier patch for its own.

Bound: both operands truncated to 10 bits (2^-9 of a product), and a truncated addition of 2^-22 for each."""
import pytest

pytestmark = pytest.mark.gpu

# N, IH, IW, IC, OC, FH, FW: ring slots 5, 4, 3, 2, 3 for 5, 7, 4, 9, 3 chunks (turns), 3 for 2 (release first), 6 for 2
SHAPES = [(6, 30, 30, 160, 8, 3, 3), (3, 31, 28, 216, 16, 3, 3), (4, 30, 58, 128, 32, 3, 3), (2, 16, 30, 288, 16, 3, 3), (8, 7, 29, 96, 64, 3, 2), (8, 30, 30, 64, 64, 3, 3), (8, 30, 30, 64, 16, 3, 3)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_more_chunks_than_ring_slots(pkg, shape):
    import torch
    engine, lib = pkg.submodule("engine"), pkg.submodule("lib")
    N, IH, IW, IC, OC, FH, FW = shape
    ph, pw = FH // 2, FW // 2 if FW > 2 else 0
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="tf32"))
    g = torch.Generator(device="cuda").manual_seed(IC)
    X, W = torch.randn((N, IH, IW, IC), device="cuda", generator=g), torch.randn((OC, FH, FW, IC), device="cuda", generator=g)
    conv = lambda x, w: torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), padding=(ph, pw)).permute(0, 2, 3, 1)
    ref, mag = conv(X.double(), W.double()), conv(X.double().abs(), W.double().abs())
    old = {k: lib.set_option(k, v) for k, v in (("HALO_TAPSTACK", 2), ("HALO_PAD", 2))}
    try:
        for _ in range(3):
            Y = eng.conv3D(X, W, 1, 1, ph, pw)
            assert lib.last_algo() == "halo_tapstack", lib.last_plan()
            assert bool(((Y.double() - ref).abs() <= (2.0 ** -9 + FH * FW * IC * 2.0 ** -22) * mag).all())
            # deltaX by the same kernel: the filter rotated, as the output channels of a layer of IC channels
            dX = eng.dconv3D_deltaX(X, W.permute(3, 1, 2, 0).flip((1, 2)).contiguous(), IH if ph else IH - FH + 1, IW - FW + 1 + 2 * pw, 1, 1, FH - 1 - ph, FW - 1 - pw)
            assert lib.last_algo() == "halo_tapstack" and float((dX - Y).abs().max()) <= 1e-5 * float(mag.max())
    finally:
        for k, v in old.items():
            lib.set_option(k, v)
    assert lib.device_status() == 0
