"""Element permutations (small copies and additions) at the edges of their CTAs
(1024 elements) and on both sides of the sizes where the tiled engine takes
over: copies move bits, additions round the product and the sum once each."""
import numpy as np
import pytest
import torch

import exatensor_b200 as XB

pytestmark = pytest.mark.gpu

SHAPES = [([1023], [1]), ([1, 1, 1], [3, 1, 2]), ([31, 33], [2, 1]), ([32, 32], [2, 1]), ([5, 41, 5], [3, 1, 2]),
          ([2] * 12, [12, 1, 11, 2, 10, 3, 9, 4, 8, 5, 7, 6]), ([2] * 18, list(range(18, 0, -1))),
          ([3, 5, 7, 2, 11], [4, 2, 5, 1, 3])]
# just below and just above the limits of copies (24 and 32 MB) and of 4-byte additions (64 MB)
LARGE = [(4, [251, 251, 99], [3, 1, 2]), (4, [251, 251, 101], [3, 1, 2]), (8, [63, 64, 65, 16], [4, 2, 3, 1]),
         (8, [65, 64, 65, 16], [4, 2, 3, 1]), (4, [255, 256, 257], [2, 3, 1]), (4, [257, 256, 257], [2, 3, 1])]


def moved(x, dims, perm):
    """The permuted tensor by torch: index k of the input becomes index perm[k]."""
    r = len(dims)
    src = [perm.index(p + 1) for p in range(r)]
    return x.view(tuple(reversed(dims))).permute([r - 1 - src[r - 1 - q] for q in range(r)]).contiguous().view(-1)


@pytest.mark.parametrize("kind,dt", [(XB.R4, torch.float32), (XB.R8, torch.float64), (XB.C4, torch.complex64),
                                     (XB.C8, torch.complex128)])
@pytest.mark.parametrize("dims,perm", SHAPES)
def test_small_copies_and_additions(xt, dev, kind, dt, dims, perm):
    n = int(np.prod(dims))
    g = torch.Generator(device="cuda").manual_seed(n + kind)
    x = torch.randn(n, dtype=dt, device="cuda", generator=g)
    y = torch.randn(n, dtype=dt, device="cuda", generator=g)
    want = moved(x, dims, perm)
    out = torch.zeros_like(y)
    n0 = xt.launch_count()
    xt.tensor_copy(kind, dims, perm, x.data_ptr(), out.data_ptr(), stream=torch.cuda.current_stream())
    assert xt.launch_count() - n0 == 1
    assert torch.equal(out, want)
    if dt.is_complex:
        xt.tensor_copy(kind, dims, perm, x.data_ptr(), out.data_ptr(), conj_bits=2, stream=torch.cuda.current_stream())
        assert torch.equal(out, want.conj().resolve_conj())
    xt.tensor_add(kind, dims, perm, y.data_ptr(), x.data_ptr(), 0.5, stream=torch.cuda.current_stream())
    g = torch.Generator(device="cuda").manual_seed(n + kind)
    torch.randn(n, dtype=dt, device="cuda", generator=g)
    y0 = torch.randn(n, dtype=dt, device="cuda", generator=g)
    assert torch.equal(y, y0 + want * 0.5)  # a power of two: the product is exact


@pytest.mark.parametrize("es,dims,perm", LARGE)
def test_sizes_around_the_limits(xt, dev, es, dims, perm):
    n = int(np.prod(dims))
    dt, kind = (torch.float32, XB.R4) if es == 4 else (torch.float64, XB.R8)
    x = torch.arange(n, dtype=dt, device="cuda")
    out, d = torch.zeros_like(x), torch.ones_like(x)
    want = moved(x, dims, perm)
    for _ in range(2):  # the first call of a shape may time its plans
        xt.tensor_copy(kind, dims, perm, x.data_ptr(), out.data_ptr(), stream=torch.cuda.current_stream())
        assert torch.equal(out, want)
    xt.tensor_add(kind, dims, perm, d.data_ptr(), x.data_ptr(), 2.0, stream=torch.cuda.current_stream())
    assert torch.equal(d, want * 2 + 1)
