"""CPU replay of the element permutation's order (tests/emul/elem_perm_emul.cpp):
random shapes and permutations, unit extents, ranks up to and past the plan's
limit."""
import os
import random
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "exatensor_b200", "csrc")


def test_every_element_once(tmp_path):
    exe = str(tmp_path / "elem")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "emul", "elem_perm_emul.cpp"),
                    os.path.join(CSRC, "tb_perm_plan.cpp"), "-o", exe], check=True)
    rng = random.Random(8)
    lines = ["8 0", "8 1 1 1", "4 1 17 1", "8 3 1 5 1 3 2 1", "8 18 " + "2 " * 18 + " ".join(str(18 - i) for i in range(18))]
    for _ in range(500):
        rank = rng.randint(1, 7)
        dims = [rng.choice([1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 40]) for _ in range(rank)]
        while True:
            vol = 1
            for x in dims:
                vol *= x
            if vol <= 60000:
                break
            dims[dims.index(max(dims))] //= 2
        perm = list(range(1, rank + 1))
        rng.shuffle(perm)
        lines.append(" ".join(map(str, [rng.choice([4, 8, 16]), rank] + dims + perm)))
    out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == len(lines)
    assert out[4].startswith("DECLINED")
    bad = [x for x in zip(lines, out) if x[1].startswith("BAD")]
    assert not bad, bad[:5]
