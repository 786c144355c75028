"""SM_BUDGET leaves SMs to a kernel of another stream: no waiting successor of the library's own launches may occupy them."""
import pytest

pytestmark = pytest.mark.gpu


def test_budget_leaves_room_for_another_stream(pkg):
    """Side GEMMs beside a chain of convolutions on half of the SMs end long before the chain does (alone they take a sixth of it)."""
    import torch
    lib, engine = pkg.submodule("lib"), pkg.submodule("engine")
    eng = engine.Engine(engine.CudaFloat32EngineBase(math="3xtf32"))
    X, W = torch.randn((256, 56, 56, 64), device="cuda"), torch.randn((64, 3, 3, 64), device="cuda")
    A = torch.randn((1024, 1024), device="cuda", dtype=torch.bfloat16)
    main, conv, side = torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()

    def both():
        conv.wait_stream(main)
        side.wait_stream(main)
        start, conv_end, side_end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        start.record()
        with torch.cuda.stream(conv):
            for _ in range(10):
                eng.conv3D(X, W, 1, 1, 1, 1)
            conv_end.record()
        with torch.cuda.stream(side):
            for _ in range(100):
                A @ A
            side_end.record()
        main.wait_stream(conv)
        main.wait_stream(side)
        torch.cuda.synchronize()
        return start.elapsed_time(side_end) / start.elapsed_time(conv_end)

    lib.set_option("SM_BUDGET", 74)
    try:
        for _ in range(3):
            both()
        share = sorted(both() for _ in range(9))[4]
    finally:
        lib.set_option("SM_BUDGET", 0)
    assert share <= 0.5, share
