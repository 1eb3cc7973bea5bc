"""One-kernel contractions over every tile shape, K split and row box that the planner
takes (golden/direct_cases.json: kind, tile shape, split, box, pattern, extents; the
smallest found for each; tests/test_direct_plan_emul.py checks that the planner takes
them there), in all four data kinds.

Operands are whole numbers of up to 2 bits and alpha is 1/2, so that every product and
sum is exact in the data's own type and results are compared bit for bit with a
64-bit reference.  NaN and infinities in both operands give the IEEE pattern, and
the other entries keep their bits."""
import json
import os
import re

import pytest
import torch

import exatensor_b200 as XB
from tests.test_gpu_routes import install_plain

pytestmark = pytest.mark.gpu
CASES = json.load(open(os.path.join(os.path.dirname(__file__), "golden", "direct_cases.json")))
KIND = {"R4": (XB.R4, torch.float32), "R8": (XB.R8, torch.float64), "C4": (XB.C4, torch.complex64),
        "C8": (XB.C8, torch.complex128)}


def operands(kind, pattern, extents, seed):
    """(labels, dims, [D, L, R]) as contiguous tensors in torch's (reversed) order."""
    ext = {x.split("=")[0]: int(x.split("=")[1]) for x in extents.split()}
    g = [x.replace(",", "") for x in re.findall(r"\(([^)]*)\)", pattern)]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = KIND[kind][1]

    def whole(n):
        real = torch.randint(-2, 3, (n * (2 if dt.is_complex else 1),), device="cuda", generator=gen).to(torch.float64)
        return (torch.view_as_complex(real.view(n, 2)) if dt.is_complex else real).to(dt)

    dims = [[ext[x] for x in s] for s in g]
    out = []
    for d in dims:
        n = 1
        for x in d:
            n *= x
        out.append(whole(n).view(tuple(reversed(d))))
    return g, dims, out


def reference(g, d, l, r, conj):
    """D + L R / 2 in 64 bits; complex products from four real ones, as sums of terms are."""
    eq = "%s,%s->%s" % (g[1][::-1], g[2][::-1], g[0][::-1])
    if not l.dtype.is_complex:
        return torch.einsum(eq, l.double(), r.double()) * 0.5 + d.double()
    lr, li, rr, ri = l.real.double(), l.imag.double() * (-1.0 if conj else 1.0), r.real.double(), r.imag.double()
    re = torch.einsum(eq, lr, rr) - torch.einsum(eq, li, ri)
    im = torch.einsum(eq, lr, ri) + torch.einsum(eq, li, rr)
    # alpha is the complex number (1/2, 0): an infinity times its imaginary part is NaN
    return torch.complex(re * 0.5 - im * 0.0 + d.real.double(), im * 0.5 + re * 0.0 + d.imag.double())


def parts(x):
    return [x.real, x.imag] if x.dtype.is_complex else [x]


@pytest.mark.parametrize("ci", range(len(CASES)), ids=lambda i: "%s-%d-%d-%d" % tuple(CASES[i][:4]))
def test_every_shape_split_and_box(xt, dev, ci):
    kind, _, _, _, pattern, extents = CASES[ci]
    dtk, dt = KIND[kind]
    g, dims, (d, l, r) = operands(kind, pattern, extents, ci)
    conj = dt.is_complex and ci % 2 == 1
    pat = pattern.replace("L(", "L+(") if conj else pattern
    nan, inf = float("nan"), float("inf")
    install_plain()
    try:
        for plant in (False, True):
            if plant:
                lf, rf = [torch.view_as_real(x).view(-1) if dt.is_complex else x.view(-1) for x in (l, r)]
                lf[lf.numel() // 3] = nan
                lf[lf.numel() - 1] = -inf
                rf[rf.numel() // 2] = inf
            out = d.clone()
            n0 = xt.launch_count()
            xt.tensor_contract(pat, dtk, dims[0], out.data_ptr(), dims[1], l.data_ptr(), dims[2], r.data_ptr(), 0.5,
                               stream=torch.cuda.current_stream())
            assert xt.launch_count() - n0 == 1
            want = reference(g, d, l, r, conj)
            for a, b in zip(parts(out), parts(want)):
                a = a.double()
                for f in (torch.isnan, torch.isposinf, torch.isneginf):
                    assert torch.equal(f(a), f(b)), f.__name__
                fin = torch.isfinite(b)
                assert torch.equal(a[fin], b[fin])
    finally:
        XB.selector_install(0, None, None, None)
