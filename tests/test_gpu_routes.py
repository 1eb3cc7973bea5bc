"""Where TB_METHOD_AUTO sends FP64 products, and the operand orders of the
tensor-core path.

Long R8 and C8 products that the selector leaves to the plain method run with
15 moduli; short ones in one kernel.  Tolerance of the former: operands keep 51
bits (2^-51 each, relative to a row's largest value, about 1.7 times the rms of
uniform data) and the FP64 reference itself carries about sqrt(K) 2^-54.

The fused path's rows run in blocks of eight of the left operand's contiguous
group when D's fastest group is another one: groups shorter than a block, whole
blocks, and blocks with a remainder."""
import numpy as np
import pytest
import torch

import exatensor_b200 as XB
import oracle as O
from tests.test_gpu_contract import oracle_dd
from tests.test_gpu_permute import rand_host

pytestmark = pytest.mark.gpu


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
    sums of 300 FP64 products and an accumulated old element.)"""
    m, n, k, off = 96, 80, 300, 3
    rng = np.random.default_rng(4)
    x = rng.uniform(-1, 1, k * m + n * m + off)
    x[5] = np.inf  # L(5, 0); also D(2, 0)
    r = rng.uniform(-1, 1, n * k)
    lm, rm, d0 = x[:k * m].reshape(k, m), r.reshape(k, n), x[off:off + n * m].reshape(n, m)
    with np.errstate(invalid="ignore"):
        want = rm.T @ lm + d0
    buf, rd = dev.put(x), dev.put(r)
    xt.tensor_contract("D(a,b)+=L(a,k)*R(b,k)", XB.R8, [m, n], buf.data_ptr() + 8 * off, [m, k], buf.data_ptr(), [n, k],
                       rd.data_ptr(), 1.0, stream=dev.stream())
    st = xt.last_contract_stats()
    got = dev.get(buf, np.float64)[off:off + n * m].reshape(n, m)
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fin = np.isfinite(want)
    assert fin.sum() >= (m - 2) * n and np.array_equal(np.isfinite(got), fin)
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
