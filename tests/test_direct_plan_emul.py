"""CPU replay of the one-kernel contraction's plan and index arithmetic
(tests/emul/direct_emul.cpp): random patterns, extents with remainders, every
tile shape, K split and row box, in exact integers against plain loops."""
import os
import random
import subprocess

import pytest

import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "exatensor_b200", "csrc")
PATTERNS = ["D(a,b,i,j)+=L(a,b,c,d)*R(c,d,i,j)", "D(a,i,b,j)+=L(a,k,c,i)*R(c,b,k,j)",
            "D(a,b,c,d)+=L(c,k,a,l)*R(l,d,k,b)", "D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)",
            "D(a,b,c,d)+=L(d,b,e,a)*R(e,c)", "D(a,b,c)+=L(d,c,a)*R(b,d)", "D(a,b,c,d)+=L(e,b)*R(a,e,c,d)",
            "D(a,b)+=L(a,c,d)*R(d,b,c)", "D(a)+=L(k,a)*R(k)", "D(a,b)+=L(b)*R(a)", "D(a,b)+=L()*R(b,a)"]


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("direct") / "direct_emul")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "emul", "direct_emul.cpp"),
                    os.path.join(CSRC, "tb_direct_plan.cpp"), os.path.join(CSRC, "tb_pattern.cpp"), "-o", exe],
                   check=True)
    return exe


def labels(pattern):
    return [[x for x in part.split(")")[0].split(",") if x] for part in pattern.split("(")[1:]]


def test_shapes_match_the_kernels():
    """The shapes in the emulation are those the launch table instantiates."""
    src = open(os.path.join(CSRC, "tb_direct.cu")).read()
    import re
    v = [tuple(int(x) for x in m) for m in re.findall(r"Variant<E, (\d+), (\d+), (\d+), (\d+), (\d+), (\d+), \d+, (\d+)>", src)]
    got = [(wm * mi * 8, wn * ni * 8, bk * kw, wm * wn * kw * 32, occ) for wm, wn, kw, mi, ni, bk, occ in v]
    em = open(os.path.join(HERE, "emul", "direct_emul.cpp")).read()
    want = [tuple(int(x) for x in m) for m in re.findall(r"\{(\d+), (\d+), (\d+), (\d+), (\d+)\}", em)]
    assert got == want


@pytest.fixture(scope="module")
def info(tmp_path_factory):
    return build_info(tmp_path_factory)


def build_info(tmp_path_factory):
    """plans(cases): (variant, split, box, a_on_k, b_on_k, predicted us) per (pattern, extents, es, cplx), None where declined."""
    exe = str(tmp_path_factory.mktemp("direct_info") / "direct_plan_info")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "emul", "direct_plan_info.cpp"),
                    os.path.join(CSRC, "tb_direct_plan.cpp"), os.path.join(CSRC, "tb_pattern.cpp"), "-o", exe],
                   check=True)

    def plans(cases):
        lines = []
        for pat, ext, es, cplx in cases:
            g = labels(pat)
            flat = [len(x) for x in g] + [ext[c] for x in g for c in x] + list(O.parse_pattern(pat)[0]) + [es, int(cplx)]
            lines.append(" ".join(map(str, flat)))
        out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.splitlines()
        assert len(out) == len(cases)
        return [None if x == "DECLINED" else tuple(float(y) for y in x.split()) for x in out]

    return plans


def test_device_cases_cover_the_shapes(info):
    """The planner takes the tile shape, split and box for which each case of the device
    test (tests/test_gpu_direct_shapes.py) is listed; together they hold every shape that
    it takes for products of up to 1e9 multiply-adds."""
    import json
    cases = json.load(open(os.path.join(HERE, "golden", "direct_cases.json")))
    es = {"R4": 4, "R8": 8, "C4": 8, "C8": 16}
    got = info([(c[4], {x.split("=")[0]: int(x.split("=")[1]) for x in c[5].split()}, es[c[0]], c[0][0] == "C") for c in cases])
    assert [c[:4] for c in cases] == [[c[0], int(p[0]), int(p[1]), int(p[2])] for c, p in zip(cases, got)]
    for kind, shapes in (("R4", 7), ("R8", 7), ("C4", 5), ("C8", 6)):
        mine = [c for c in cases if c[0] == kind]
        assert {c[1] for c in mine} == set(range(shapes))
        assert {c[2] for c in mine} == {1, 2, 4, 8} and {c[3] for c in mine} == {0, 1}


def test_clusters_that_do_not_fit_at_once_are_predicted_slower(info):
    """416 CTAs in clusters of eight, of which 384 are resident: measured 3.9 ms (R4, 395
    x 470 x 122598).  The model has to stay within a third of that, or products that the
    tensor cores run in 2.0 ms come here; a shape of which five CTAs per SM fit does
    not wait (2183 x 33 x 24640, measured 0.40 ms)."""
    long_sum, fits = info([("D(a,b)+=L(a,c,d)*R(d,b,c)", dict(a=395, b=470, c=294, d=417), 4, False),
                           ("D(a,b,c)+=L(a,d,e,c)*R(e,b,d)", dict(a=37, b=33, c=59, d=140, e=176), 4, False)])
    assert long_sum[5] > 3950 / 1.33
    assert fits[5] < 400 * 1.33


def test_every_index_once(emul):
    rng = random.Random(5)
    lines = []
    for n in range(420):
        pat = rng.choice(PATTERNS)
        d, l, r = labels(pat)
        ext = {x: rng.choice([1, 2, 3, 5, 7, 8, 11, 16, 17, 19, 23, 33]) for x in set(d + l + r)}
        dims = [[ext[x] for x in g] for g in (d, l, r)]
        while True:  # bounded work for the plain loops
            work = 1
            for x in ext.values():
                work *= x
            if work <= 600000:
                break
            big = max(ext, key=ext.get)
            ext[big] = max(1, ext[big] // 2)
            dims = [[ext[x] for x in g] for g in (d, l, r)]
        cp = O.parse_pattern(pat)[0]
        cplx = rng.random() < 0.3
        es = rng.choice([8, 16] if cplx else [4, 8])
        force = rng.random() < 0.75
        variant = rng.randrange(6 if cplx else 7) if force else -1
        split = rng.choice([1, 2, 4, 8]) if force and rng.random() < 0.5 else 0
        box = rng.choice([0, 1]) if force else -1
        flat = [len(d), len(l), len(r)] + [x for g in dims for x in g] + list(cp) + [es, int(cplx), variant, split, box]
        lines.append(" ".join(map(str, flat)))
    out = subprocess.run([emul], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == len(lines)
    bad = [(i, o) for i, o in zip(lines, out) if o.startswith("BAD")]
    assert not bad, bad[:5]
    ok = [o for o in out if o.startswith("OK")]
    assert len(ok) > 150 and any("box=1" in o for o in ok) and any("split=8" in o for o in ok)
