"""One-kernel contractions (what TB_METHOD_AUTO runs for small, narrow and
output-bound products) against the double-double oracle: every data kind, tile
edges and remainders, K splits, row boxes, both operand orders, conjugation,
alpha and beta.

Tolerance (relative Frobenius): the sums are FP64, so a K-term product is within
(K + 3) 2^-53 of the exact one on data without cancellation beyond sqrt(K);
4-byte kinds add the rounding of the operand D, of the result and of alpha,
2^-24 each."""
import random

import numpy as np
import pytest

import exatensor_b200 as XB
import oracle as O
from tests.test_gpu_contract import oracle_dd, run_gpu
from tests.test_gpu_permute import rand_host

pytestmark = pytest.mark.gpu

# extents chosen around the tiles' edges (16, 32, 64, 128 rows and columns, 8 to 32 contracted values)
CASES = [
    ("D(a,b)+=L(a,k)*R(k,b)", dict(a=31, b=33, k=32)),
    ("D(a,b)+=L(k,a)*R(b,k)", dict(a=129, b=15, k=7)),
    ("D(a,b)+=L(b,k)*R(k,a)", dict(a=17, b=300, k=1)),
    ("D(a,b)+=L(a,k)*R(k,b)", dict(a=5, b=7, k=1500)),
    ("D(a)+=L(k,a)*R(k)", dict(a=70, k=65)),
    ("D(a,b)+=L(b)*R(a)", dict(a=40, b=9)),
    ("D(a,b,i,j)+=L(a,b,c,d)*R(c,d,i,j)", dict(a=11, b=11, c=11, d=11, i=5, j=5)),
    ("D(a,b,c,d)+=L(c,k,a,l)*R(l,d,k,b)", dict(a=9, b=7, c=13, d=6, k=5, l=8)),
    ("D(a,b,c,d)+=L(d,b,e,a)*R(e,c)", dict(a=35, b=6, c=12, d=19, e=18)),
    ("D(a,b,c,d,e)+=L(e,f,b,a,d)*R(c,f)", dict(a=16, b=5, c=17, d=3, e=33, f=9)),
    ("D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)", dict(a=5, b=6, c=4, d=7, e=3, f=5, g=19)),
    ("D(a,b,c)+=L(d,c,a)*R(b,d)", dict(a=64, b=128, c=2, d=24)),
]


@pytest.mark.parametrize("dtk", [O.R4, O.R8, O.C4, O.C8])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_against_double_double(xt, dev, dtk, ci):
    pattern, ext = CASES[ci]
    rng = random.Random(100 * ci + dtk)
    letters = [[x for x in g.split(")")[0].split(",")] for g in pattern.split("(")[1:]]
    ddims, ldims, rdims = [[ext[x] for x in g] for g in letters]
    d, l, r = [rand_host(dtk, int(np.prod(x)), 7 * ci + k) for k, x in enumerate((ddims, ldims, rdims))]
    if dtk in (O.C4, O.C8) and ci % 2:
        pattern = pattern.replace("L(", "L+(")
    alpha = 0.75 - 0.5j if dtk in (O.C4, O.C8) else -0.75
    accumulative = rng.random() < 0.7
    ref = oracle_dd(pattern, d, ddims, l, ldims, r, rdims, alpha, accumulative)
    n0 = xt.launch_count()
    got = run_gpu(xt, dev, pattern, d, ddims, l, ldims, r, rdims, alpha, accumulative, XB.METHOD_AUTO)
    assert xt.launch_count() - n0 == 1  # one kernel, no permutation pass
    k = int(np.prod([v for x, v in ext.items() if x in letters[1] and x in letters[2]]))
    tol = (k + 3) * 2.0 ** -53 if dtk in (O.R8, O.C8) else 4 * 2.0 ** -24
    assert O.rel_frobenius(got, ref) <= tol, (pattern, ext)


def test_nan_stays_in_its_row_and_beta_zero_ignores_d(xt, dev):
    l, r = rand_host(O.R8, 33 * 21, 1), rand_host(O.R8, 21 * 18, 2)
    l[5] = np.nan  # row 5 of L(a,k)
    got = run_gpu(xt, dev, "D(a,b)+=L(a,k)*R(k,b)", np.full(33 * 18, np.nan), [33, 18], l, [33, 21], r, [21, 18], 1.0,
                  False, XB.METHOD_AUTO).reshape(18, 33)
    assert np.isnan(got[:, 5]).all() and np.isfinite(np.delete(got, 5, axis=1)).all()
