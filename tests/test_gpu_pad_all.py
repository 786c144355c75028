"""The tensors of one call padded by one launch into one block: as each of them padded by itself."""
import struct

import pytest

pytestmark = pytest.mark.gpu

# (shape, n4, c4) of each tensor: none, one, two and three to pad, first dimensions too, one of a single element
JOBS = [[((4, 3, 8), 4, 8), ((8, 4), 8, 4)], [((4, 3, 7), 4, 8), ((8, 4), 8, 4)], [((2, 5, 5, 3), 2, 4), ((6, 3, 3, 3), 8, 4), ((1, 6), 1, 8)],
        [((1, 1), 4, 4), ((1000, 257), 1000, 260), ((33, 1), 36, 4)], [((5, 6), 8, 8), ((8, 8), 8, 8), ((7, 3), 8, 4)]]


@pytest.mark.parametrize("jobs", JOBS, ids=str)
@pytest.mark.parametrize("layout", ["dense", "transposed", "offset"])
def test_pad_all(pkg, jobs, layout):
    import torch
    E, lib = pkg.submodule("engine"), pkg.submodule("lib")
    make = {"dense": lambda s: torch.randn(s, device="cuda"), "transposed": lambda s: torch.randn(s[::-1], device="cuda").permute(*range(len(s))[::-1]),
            "offset": lambda s: torch.randn(s + (1,), device="cuda").expand(s + (2,))[..., 1]}[layout]
    tensors = [make(s) for s, _, _ in jobs]
    want = [E._pad_both(t, n4, c4) for t, (_, n4, c4) in zip(tensors, jobs)]
    count = lib.launch_count()
    got, block = E._pad_all(*((t, n4, c4) for t, (_, n4, c4) in zip(tensors, jobs)))
    assert lib.launch_count() - count <= 1
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        if isinstance(g, int):
            assert g % 256 == 0
            at = (g - block.data_ptr()) // 4
            g = block[at:at + w.numel()].view(w.shape)
        assert torch.equal(g, w) and g.is_contiguous()


def test_other_types_and_bad_jobs(pkg):
    import torch
    E, lib = pkg.submodule("engine"), pkg.submodule("lib")
    a, b = torch.randn((3, 5), device="cuda").double(), torch.randn((3, 5), device="cuda")
    (x, y), block = E._pad_all((a, 4, 8), (b, 4, 8))
    assert x.dtype == torch.float64 and torch.equal(x[:3, :5], a) and torch.equal(y[:3, :5], b) and block is None
    (x, y), _ = E._pad_all((torch._neg_view(b), 4, 8), (b, 4, 8))
    assert torch.equal(x[:3, :5], -b)
    p = b.data_ptr()
    for job in ((0, 3, 5, p, 4, 8), (p, 3, 5, 0, 4, 8), (p, 0, 5, p, 4, 8), (p, 3, 5, p, 2, 8), (p, 3, 5, p, 4, 4), (p, 3, 5, p, 4, 6), (p, 3, 5, p + 4, 4, 8)):
        assert lib.load().alpha_pad_rows_many(2, struct.pack("12q", *job, *job), None) == -1, job
    assert lib.load().alpha_pad_rows_many(0, b"", None) == -1
