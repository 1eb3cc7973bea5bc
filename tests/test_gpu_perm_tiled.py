"""The tiled permutation engine on the sizes that the element kernel takes otherwise
(it still runs larger ones): with TB_PERM_ELEM=0 the tests of permutations and of
the fused addition run again in a child process, and additions of every data kind,
conjugated and with odd extents, are compared with the oracle bit for bit.  The
switch is read once per process; trace lines show that the tiled kernels ran."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ENV = dict(os.environ, TB_PERM_ELEM="0", TB_PERM_TRACE="1")

SHAPES = [([90, 30, 90, 30], [(2, 1, 3, 4), (1, 4, 3, 2), (4, 2, 3, 1)]), ([37, 41, 29], [(3, 1, 2), (2, 1, 3), (1, 3, 2)]),
          ([64, 48, 80], [(3, 2, 1), (2, 3, 1)]), ([3, 300, 250], [(3, 1, 2)]), ([129, 257], [(2, 1)]),
          ([8, 6, 10, 4, 12, 5], [(6, 1, 5, 2, 4, 3)]), ([1023], [(1,)])]


def child():
    import numpy as np

    sys.path.insert(0, ROOT)
    import exatensor_b200 as XB
    import oracle as O
    from tests.conftest import Dev
    from tests.test_gpu_permute import rand_host

    XB.device_init(0)
    bad, n = [], 0
    for dtk in (O.R4, O.R8, O.C4, O.C8):
        cplx = dtk in (O.C4, O.C8)
        scale = 0.37 - 0.2j if cplx else 0.37
        for dims, perms in SHAPES:
            vol = int(np.prod(dims))
            l, d0 = rand_host(dtk, vol, 60), rand_host(dtk, vol, 70)
            for perm in perms:
                for conj in ((0, 2, 3) if cplx else (0,)):
                    ref = O.tensor_add(list(perm), d0.copy(), l, dims, scale, conj)
                    dd, ld = Dev.put(d0), Dev.put(l)
                    XB.tensor_add(dtk, dims, list(perm), dd.data_ptr(), ld.data_ptr(), scale, conj, Dev.stream())
                    n += 1
                    if not np.array_equal(Dev.get(dd, d0.dtype, vol).view(np.uint8), ref.view(np.uint8)):
                        bad.append([dtk, dims, list(perm), conj])
    XB.device_check(Dev.stream())
    print(json.dumps({"cases": n, "bad": bad}))


def test_additions_by_the_tiled_engine():
    r = subprocess.run([sys.executable, "-c", "import tests.test_gpu_perm_tiled as t; t.child()"], cwd=ROOT, env=ENV,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["cases"] == 96 and out["bad"] == [], out["bad"][:10]
    assert r.stderr.count("kernel=") >= out["cases"] - 8  # (the contiguous shape may be a plain copy of rows)


def test_permutation_tests_by_the_tiled_engine():
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-s", "-m", "gpu", "tests/test_gpu_permute.py",
                        "tests/test_gpu_elementwise.py", "-k", "not full_size and not measured"], cwd=ROOT, env=ENV,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:]
    assert r.stderr.count("kernel=") >= 500
