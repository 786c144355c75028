"""The engine's pad-to-4 copies, and pooling gradients of 2 x 2 blocks against the element-wise kernel's order of sums."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,rows4,cols4", [(1, 1, 1, 4), (7, 3, 8, 4), (5, 4, 8, 4), (300, 5, 300, 8), (13, 257, 16, 260), (70000, 3, 70000, 4)])
def test_pad_rows(pkg, rows, cols, rows4, cols4):
    import torch
    lib = pkg.submodule("lib")
    src = torch.randn((rows * cols + 1,), device="cuda")[1:].view(rows, cols)      # not 16-byte aligned
    out = torch.full((rows4 * cols4 + 64,), float("nan"), device="cuda")
    lib.check(lib.load().alpha_pad_rows(src.data_ptr(), rows, cols, out.data_ptr(), rows4, cols4, torch.cuda.current_stream().cuda_stream))
    want = torch.zeros((rows4, cols4), device="cuda")
    want[:rows, :cols] = src
    assert torch.equal(out[:rows4 * cols4].view(rows4, cols4), want) and bool(out[rows4 * cols4:].isnan().all())


def test_engine_pads_any_layout(pkg):
    """Strided and transposed inputs, other data types, one-dimensional tensors: as a zero-filled copy."""
    import torch
    E = pkg.submodule("engine")
    base = torch.randn((6, 5, 7), device="cuda")
    for t in (base, base.transpose(0, 2), base[::2, :, 1:6], base.double(), base[0, 0]):
        c4 = E._pad4(t.shape[-1])
        got = E._pad_last(t, c4)
        assert got.is_contiguous() and got.dtype == t.dtype
        assert torch.equal(got[..., : t.shape[-1]], t) and bool((got[..., t.shape[-1]:] == 0).all())
    neg = torch._neg_view(base)
    assert torch.equal(E._pad_last(neg, 8)[..., :7], -base)
    got = E._pad_both(base, 8, 8)
    assert torch.equal(got[:6, :, :7], base) and bool((got[6:] == 0).all()) and bool((got[:, :, 7:] == 0).all())


def test_pad_rows_beyond_one_launch(pkg):
    """2.1e9 rows of one column: more 16-byte words than a launch indexes."""
    import torch
    lib = pkg.submodule("lib")
    rows = 2100000000
    src = torch.arange(rows, device="cuda", dtype=torch.int32).view(torch.float32)      # (bit patterns)
    out = torch.full((rows + 8, 4), float("nan"), device="cuda")
    lib.check(lib.load().alpha_pad_rows(src.data_ptr(), rows, 1, out.data_ptr(), rows + 4, 4, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out[:rows, 0].view(torch.int32), src.view(torch.int32))
    assert not bool(out[:rows, 1:].any()) and not bool(out[rows:rows + 4].any()) and bool(out[rows + 4:].isnan().all())


# N, IH, IW, IC, F, p: odd images (a last block row of one element), every padding, channel groups of 4 and of 8
@pytest.mark.parametrize("shape", [(2, 13, 11, 8, 3, 1), (1, 12, 14, 12, 3, 0), (2, 7, 9, 20, 3, 2), (3, 10, 13, 16, 2, 0), (2, 9, 8, 4, 2, 1), (1, 3, 3, 24, 3, 1)], ids=str)
def test_stride_two_gradients(pkg, oracle_mod, shape):
    import torch
    eng = pkg.submodule("engine").Engine()
    N, IH, IW, IC, F, p = shape
    g = torch.Generator(device="cuda").manual_seed(IH * 100 + IC)
    X = torch.randn((N, IH, IW, IC), device="cuda", generator=g).mul_(2).round_()         # ties
    Y, index = eng.pool2D_max(X, F, F, 2, 2, p, p, indexed=True)
    OH, OW = Y.shape[1:3]
    dY = torch.randn((N, OH, OW, IC), device="cuda", generator=g)
    want = {k: torch.zeros((N, IH, IW, IC), device="cuda") for k in ("max", "indexed", "avg", "avg_ip")}
    off = torch.arange(N * IH * IW * IC, device="cuda", dtype=torch.int32).view(N, IH, IW, IC)
    alpha = torch.tensor(1.0, device="cuda") / (F * F)
    for oh in range(OH):                          # ascending (oh, ow): the order in which an element adds its windows
        for ow in range(OW):
            h0, w0 = max(oh * 2 - p, 0), max(ow * 2 - p, 0)
            h1, w1 = min(oh * 2 - p + F, IH), min(ow * 2 - p + F, IW)
            s = (slice(None), slice(h0, h1), slice(w0, w1))
            dy = dY[:, oh:oh + 1, ow:ow + 1]
            want["max"][s] += (X[s] >= Y[:, oh:oh + 1, ow:ow + 1]) * dy
            want["indexed"][s] += (off[s] == index[:, oh:oh + 1, ow:ow + 1]) * dy
            want["avg"][s] += (alpha.double() * dy.double()).float()       # one rounding more than the kernel's FMA
            want["avg_ip"][s] += dy / torch.full_like(dy, (h1 - h0) * (w1 - w0))   # (a Python divisor would become a product)
    assert torch.equal(eng.upool2D_max(dY, Y, X, F, F, 2, 2, p, p), want["max"])
    assert torch.equal(eng.upool2D_max_indexed(dY, index, IH, IW, F, F, 2, 2, p, p), want["indexed"])
    assert torch.equal(eng.upool2D_avg(dY, IH, IW, F, F, 2, 2, p, p, ignore_padding=True), want["avg_ip"])
    # four windows at most: each product and sum rounds once
    assert float((eng.upool2D_avg(dY, IH, IW, F, F, 2, 2, p, p) - want["avg"]).abs().max()) <= 8 * 2.0 ** -24 * float(dY.abs().max())
