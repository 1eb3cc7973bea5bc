"""Where TB_METHOD_AUTO sends FP64 products, and the operand orders of the
tensor-core path.

Long R8 and C8 products that the selector leaves to the plain method run with
15 moduli; short ones in one kernel.  Tolerance of the former: operands keep 51
bits (2^-51 each, relative to a row's largest value, about 1.7 times the rms of
uniform data) and the FP64 reference itself carries about sqrt(K) 2^-54.

The fused path's rows run in blocks of eight of the left operand's contiguous
group when D's fastest group is another one: groups shorter than a block, whole
blocks, and blocks with a remainder."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import exatensor_b200 as XB
import oracle as O
from tests.test_gpu_contract import oracle_dd
from tests.test_gpu_permute import rand_host

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("kind,dt,m,n,k,moduli", [(XB.R8, torch.float64, 1400, 1100, 1290, 15),
                                                  (XB.C8, torch.complex128, 900, 700, 1000, 15),
                                                  (XB.R8, torch.float64, 1300, 1200, 200, 0)])
def test_long_products_keep_51_bits(xt, dev, kind, dt, m, n, k, moduli):
    g = torch.Generator(device="cuda").manual_seed(k)
    real = torch.float64
    mk = lambda *s: (torch.rand(*s, dtype=real, device="cuda", generator=g) * 2 - 1)  # noqa: E731
    l, r, d = [mk(*s) if dt == real else torch.complex(mk(*s), mk(*s)) for s in ((m, k), (n, k), (n, m))]
    want = r @ l.T + d  # D(i,j), i fastest; L(k,i) and R(k,j) with k fastest
    plain = np.zeros(16 * 8 + 8 + 64 + 8 + 8 * XB.SELECT_PLANS + XB.SELECT_PLANS, np.float32)
    plain[-XB.SELECT_PLANS + 1:] = 9.0
    # a caller's network that picks the plain method keeps it: one kernel, no residues
    XB.selector_install(8, plain, np.zeros(16, np.float32), np.ones(16, np.float32))
    try:
        out = d.clone()
        xt.tensor_contract("D(i,j)+=L(k,i)*R(k,j)", kind, [m, n], out.data_ptr(), [k, m], l.data_ptr(), [k, n],
                           r.data_ptr(), 1.0, stream=torch.cuda.current_stream())
        st = xt.last_contract_stats()
        assert st.method == XB.METHOD_TTGT and st.moduli == 0
        assert (torch.linalg.norm(out - want) / torch.linalg.norm(want)).item() <= 4e-15
    finally:
        XB.selector_install(0, None, None, None)
    out = d.clone()
    # below the size rule's 4e9 operations: picked plain, then refined
    xt.tensor_contract("D(i,j)+=L(k,i)*R(k,j)", kind, [m, n], out.data_ptr(), [k, m], l.data_ptr(), [k, n], r.data_ptr(),
                       1.0, stream=torch.cuda.current_stream())
    st = xt.last_contract_stats()
    assert st.moduli == moduli and (not moduli or st.residue_bits >= 51)
    assert (torch.linalg.norm(out - want) / torch.linalg.norm(want)).item() <= 4e-15


def install_plain():
    """A caller's network that always picks the plain method."""
    p = np.zeros(16 * 8 + 8 + 64 + 8 + 8 * XB.SELECT_PLANS + XB.SELECT_PLANS, np.float32)
    p[-XB.SELECT_PLANS + 1:] = 9.0
    XB.selector_install(8, p, np.zeros(16, np.float32), np.ones(16, np.float32))


def spread_operands(kind, name, m, n, k, g):
    """L as (m, k), R as (n, k) by the name of their magnitudes along k."""
    real = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=g) * 2 - 1  # noqa: E731
    mk = real if kind == XB.R8 else lambda *s: torch.complex(real(*s), real(*s))
    l, r = mk(m, k), mk(n, k)
    x = torch.arange(k, dtype=torch.float64, device="cuda")
    if name == "graded":       # energy denominators: 1e-8 .. 1 along k in one operand, the inverse in the other
        w = torch.pow(10.0, -8 * x / k)
        l, r = l * w, r / w
    elif name == "steep":      # 1 .. 2^-60
        w = torch.pow(2.0, -torch.floor(60 * x / k))
        l, r = l * w, r / w
    elif name == "half":       # half of L tiny where R has values, R zero on the other half
        l, r = l * torch.where(x < k // 2, 1.0, 1e-10), r * (x >= k // 2)
    elif name == "lognormal":
        l = l * torch.exp(3 * torch.randn(m, k, dtype=torch.float64, device="cuda", generator=g))
        r = r * torch.exp(3 * torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g))
    elif name == "one row":
        l[7] *= torch.pow(2.0, -torch.floor(60 * x / k))
    elif name == "one column":
        r[5] *= torch.pow(2.0, -torch.floor(60 * x / k))
    elif name == "subnormal row":
        l[3] *= 1e-310
    elif name == "zero row and column":
        l[3], r[n - 1] = 0, 0
    elif name == "rows of all sizes":
        l = l * torch.pow(10.0, torch.linspace(-150, 150, m, dtype=torch.float64, device="cuda"))[:, None]
    return l.contiguous(), r.contiguous()


@pytest.mark.parametrize("k_first", [True, False])
@pytest.mark.parametrize("kind,m,n,k", [(XB.R8, 1400, 1100, 1290), (XB.C8, 900, 700, 1000), (XB.C8, 1300, 1200, 259)])
@pytest.mark.parametrize("name,residues", [
    ("uniform", True), ("zero row and column", True), ("rows of all sizes", True), ("graded", False), ("steep", False),
    ("half", False), ("lognormal", False), ("one row", False), ("one column", False), ("subnormal row", False)])
def test_fp64_products_keep_every_element(xt, dev, kind, m, n, k, k_first, name, residues):
    """Whatever the magnitudes along k, every element of a product that the selector
    leaves to the plain method is as close as an FP64 sum: within 2 sqrt(K) 2^-53
    of sum |l| |r| (rounding errors of K random terms; the alternative, a fixed point
    below a row's largest value, loses all digits of "steep").  Where the magnitudes
    allow it the product runs as residues, else as the one-kernel form, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(k + len(name))
    l, r = spread_operands(kind, name, m, n, k, g)
    pattern, ld, rd = ("D(i,j)+=L(k,i)*R(k,j)", [k, m], [k, n]) if k_first else ("D(i,j)+=L(i,k)*R(j,k)", [m, k], [n, k])
    lt, rt = (l, r) if k_first else (l.T.contiguous(), r.T.contiguous())

    def run():
        d = torch.full((n, m), float("nan"), dtype=l.dtype, device="cuda")
        xt.tensor_contract(pattern, kind, [m, n], d.data_ptr(), ld, lt.data_ptr(), rd, rt.data_ptr(), 1.0,
                           accumulative=False, stream=torch.cuda.current_stream())
        return d

    XB.selector_install(0, None, None, None)  # the size rule, which leaves these products to the plain method
    got, st = run(), xt.last_contract_stats()
    assert st.moduli == 15 and st.residue_bits >= 51
    install_plain()
    try:
        plain = run()
        assert xt.last_contract_stats().moduli == 0
    finally:
        XB.selector_install(0, None, None, None)
    assert torch.equal(got, plain) != residues
    rows, cols = [0, 3, 7, 8, m // 2, m - 1], [0, 5, n // 2, n - 1]
    wide = np.longdouble if kind == XB.R8 else np.clongdouble
    lh, rh = l[rows].cpu().numpy().astype(wide), r[cols].cpu().numpy().astype(wide)
    err = np.abs(got[cols][:, rows].cpu().numpy() - rh @ lh.T)
    # (k 2^-1074: products that round among the subnormal numbers)
    assert (err <= 2 * np.sqrt(k) * 2.0 ** -53 * (np.abs(rh) @ np.abs(lh).T) + k * 5e-324).all()


def test_refused_residues_with_nan_and_accumulation(xt, dev):
    """Falling magnitudes and a NaN row, D accumulated: the one-kernel form updates D once."""
    m, n, k = 1400, 1100, 1290
    g = torch.Generator(device="cuda").manual_seed(2)
    l, r = spread_operands(XB.R8, "steep", m, n, k, g)
    l[11, 4] = float("nan")
    d0 = torch.rand(n, m, dtype=torch.float64, device="cuda", generator=g)
    outs = []
    XB.selector_install(0, None, None, None)
    for network in (False, True):
        if network:
            install_plain()
        try:
            d = d0.clone()
            xt.tensor_contract("D(i,j)+=L(k,i)*R(k,j)", XB.R8, [m, n], d.data_ptr(), [k, m], l.data_ptr(), [k, n],
                               r.data_ptr(), -0.5, stream=torch.cuda.current_stream())
        finally:
            XB.selector_install(0, None, None, None)
        outs.append(d)
    assert torch.isnan(outs[0][:, 11]).all() and torch.equal(outs[0].nan_to_num(), outs[1].nan_to_num())


MEASURED = """
import torch
import exatensor_b200 as XB
XB.device_init(0)
a, b, c, d = 395, 470, 294, 417
l, r = torch.rand(d * c * a, device="cuda"), torch.rand(c * b * d, device="cuda")
out = torch.zeros(b * a, device="cuda")
for _ in range(3):
    XB.tensor_contract("D(a,b)+=L(a,c,d)*R(d,b,c)", XB.R4, [a, b], out.data_ptr(), [a, c, d], l.data_ptr(), [d, b, c],
                       r.data_ptr(), 1.0, accumulative=False, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    st = XB.last_contract_stats()
print("ran", st.method, st.tile_n, st.tile_m)
"""


def test_a_measured_choice_runs():
    """What timing the candidates chose (on the second call of a large shape, by the
    shipped network) is what runs, then and later."""
    env = dict(os.environ, TB_SELECT_TRACE="1")
    r = subprocess.run([sys.executable, "-c", MEASURED], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = [x for x in r.stderr.splitlines() if x.startswith("tb_select:")]
    assert line, "the candidates were timed"
    pick = int(line[-1].split("->")[1])
    ran = [int(x) for x in r.stdout.split("ran")[1].split()]
    if pick == 0:
        assert ran[0] == XB.METHOD_TTGT
    else:
        assert ran == [XB.METHOD_FUSED, 128 if pick == 1 else 256, 256 if pick == 3 else 128]


@pytest.mark.parametrize("dtk,tol", [(O.R8, 1e-12), (O.C8, 1e-12), (O.R4, 1e-4), (O.C4, 1e-4)])
@pytest.mark.parametrize("c", [3, 8, 19, 24])
def test_blocked_rows(xt, dev, dtk, tol, c):
    pattern, ext = "D(a,b,c,d)+=L(c,k,a,l)*R(l,d,k,b)", dict(a=9, b=5, c=c, d=7, k=6, l=40)
    ddims, ldims, rdims = [[ext[x] for x in g] for g in ("abcd", "ckal", "ldkb")]
    d, l, r = [rand_host(dtk, int(np.prod(x)), 3 + i) for i, x in enumerate((ddims, ldims, rdims))]
    ref = oracle_dd(pattern, d, ddims, l, ldims, r, rdims, 0.5, True)
    dd, ld, rd = dev.put(d), dev.put(l), dev.put(r)
    xt.tensor_contract(pattern, dtk, ddims, dd.data_ptr(), ldims, ld.data_ptr(), rdims, rd.data_ptr(), 0.5,
                       plan=xt.make_plan(XB.METHOD_FUSED), stream=dev.stream())
    assert O.rel_frobenius(dev.get(dd, d.dtype, d.size), ref) <= tol
    xt.device_check(dev.stream())


@pytest.mark.parametrize("kind,n,tile", [(XB.R8, 129, 192), (XB.R8, 192, 192), (XB.R8, 193, 256), (XB.R8, 575, 192),
                                         (XB.C8, 190, 192), (XB.C8, 65, 192), (XB.R8, 128, 128)])
def test_residue_tile_of_192_columns(xt, dev, kind, n, tile):
    """The N tile of residue products without a request, at its edges (complex
    products have 2n real columns); same tolerance as 14 moduli elsewhere."""
    m, k = 200, 300
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda *s: (torch.rand(*s, dtype=torch.float64, device="cuda", generator=g) * 2 - 1)  # noqa: E731
    l, r, d = [mk(*s) if kind == XB.R8 else torch.complex(mk(*s), mk(*s)) for s in ((m, k), (n, k), (n, m))]
    want = r @ l.T + d
    xt.tensor_contract("D(i,j)+=L(k,i)*R(k,j)", kind, [m, n], d.data_ptr(), [k, m], l.data_ptr(), [k, n], r.data_ptr(),
                       1.0, plan=xt.make_plan(XB.METHOD_FUSED), stream=torch.cuda.current_stream())
    assert xt.last_contract_stats().tile_n == tile
    assert (torch.linalg.norm(d - want) / torch.linalg.norm(want)).item() <= 1e-13
    xt.device_check(dev.stream())


def test_output_over_an_operand_is_multiplied_from_copies(xt, dev):
    """D starts inside L, and L's infinity lies where another row of D goes: the
    product still sees the old L.  (The infinity's row is infinite, other entries are
    sums of 300 FP64 products.)"""
    m, n, k, off = 96, 80, 300, 3
    rng = np.random.default_rng(4)
    x = rng.uniform(-1, 1, k * m + n * m + off)
    x[5] = np.inf  # L(5, 0); also D(2, 0)
    r = rng.uniform(-1, 1, n * k)
    lm, rm = x[:k * m].reshape(k, m), r.reshape(k, n)
    with np.errstate(invalid="ignore"):
        want = rm.T @ lm
    buf, rd = dev.put(x), dev.put(r)
    xt.tensor_contract("D(a,b)+=L(a,k)*R(b,k)", XB.R8, [m, n], buf.data_ptr() + 8 * off, [m, k], buf.data_ptr(), [n, k],
                       rd.data_ptr(), 1.0, accumulative=False, stream=dev.stream())
    st = xt.last_contract_stats()
    got = dev.get(buf, np.float64)[off:off + n * m].reshape(n, m)
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fin = np.isfinite(want)
    assert fin.sum() >= (m - 1) * n and np.array_equal(np.isfinite(got), fin)
    assert np.linalg.norm(got[fin] - want[fin]) <= 4e-15 * np.linalg.norm(want[fin])
    assert st.method == XB.METHOD_TTGT and st.moduli == 0


def test_more_groups_than_the_one_kernel_form_holds(xt, dev):
    """14 free indices of extent 2 in an order that nothing merges: the plain method runs, not residues."""
    rank, k = 14, 300
    a = "abcdefghijlmno"[:rank]
    perm = list(range(0, rank, 2)) + list(range(1, rank, 2))
    pattern = "D(%s,z)+=L(k,%s)*R(k,z)" % (",".join(a), ",".join(a[i] for i in perm))
    rng = np.random.default_rng(5)
    l, r = rng.uniform(-1, 1, k << rank), rng.uniform(-1, 1, 3 * k)
    dd, ld, rd = dev.put(np.zeros(3 << rank)), dev.put(l), dev.put(r)
    xt.tensor_contract(pattern, XB.R8, [2] * rank + [3], dd.data_ptr(), [k] + [2] * rank, ld.data_ptr(), [k, 3],
                       rd.data_ptr(), 1.0, accumulative=False, stream=dev.stream())
    st = xt.last_contract_stats()
    assert st.method == XB.METHOD_TTGT and st.moduli == 0
    # numpy's axes run the other way round
    lt = l.reshape([2] * rank + [k])            # axes: index perm[rank-1], ..., perm[0], k
    c = np.tensordot(r.reshape(3, k), lt, axes=([1], [rank]))  # z, perm[rank-1], ..., perm[0]
    axis = {perm[rank - 1 - i]: i + 1 for i in range(rank)}
    want = c.transpose([0] + [axis[rank - 1 - i] for i in range(rank)]).ravel()
    assert np.linalg.norm(dev.get(dd, np.float64) - want) <= 4e-15 * np.linalg.norm(want)


def test_short_of_scratch_the_one_kernel_form_runs():
    """With no memory for the residue planes (0.1 GB here) a long FP64 product runs in one
    kernel, and the call that succeeded leaves no error text.  In a process of its own,
    whose scratch pool gives everything back."""
    code = "import exatensor_b200 as X; X.device_init(0); import tests.test_gpu_routes as t; t.short_of_scratch(X)"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def short_of_scratch(xt):
    from cuda.bindings import driver as cu
    m, n, k = 1400, 1100, 1290
    g = torch.Generator(device="cuda").manual_seed(1)
    l, r = [torch.rand(x, k, dtype=torch.float64, device="cuda", generator=g) - 0.5 for x in (m, n)]
    d = torch.zeros(n, m, dtype=torch.float64, device="cuda")

    def run():
        xt.tensor_contract("D(i,j)+=L(k,i)*R(k,j)", XB.R8, [m, n], d.data_ptr(), [k, m], l.data_ptr(), [k, n],
                           r.data_ptr(), 1.0, accumulative=False, stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
        return xt.last_contract_stats()

    install_plain()  # (both forms run once, so that their kernels are loaded before memory runs short)
    run()
    XB.selector_install(0, None, None, None)
    assert run().moduli == 15
    want = r @ l.T
    d.zero_()
    text = xt.lib().tb_last_error()
    err, pool = cu.cuDeviceGetDefaultMemPool(torch.cuda.current_device())
    assert cu.cuMemPoolTrimTo(pool, 0)[0] == cu.CUresult.CUDA_SUCCESS
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    try:
        st = run()
        assert xt.lib().tb_last_error() == text
    finally:
        del fill
        torch.cuda.empty_cache()
    assert st.method == XB.METHOD_TTGT and st.moduli == 0
    assert torch.linalg.norm(d - want) <= 4e-15 * torch.linalg.norm(want)
