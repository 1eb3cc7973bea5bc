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


# (element bytes, addition, extents, permutation, alignment, tiled); measured on B200, us, element kernel / tiled engine
CHOICES = [
    (8, 1, [16] * 6, [6, 2, 4, 1, 5, 3], 256, 1),          # 321 / 77: sectors leave L2 before their next use
    (8, 1, [16] * 6, [6, 5, 4, 3, 2, 1], 256, 1),          # 350 / 93
    (16, 1, [64] * 4, [4, 3, 2, 1], 256, 1),               # 279 / 140
    (4, 0, [2048, 2048], [2, 1], 256, 1),                  # 20.8 / 11.6: whole vectors in 2-D tiles
    (4, 1, [2048, 4096], [2, 1], 256, 1),                  # 40 / 25
    (8, 0, [1697, 1698], [2, 1], 256, 0),                  # odd extents
    (8, 1, [158, 158, 158], [3, 2, 1], 256, 0),            # 24.9 / 43: tiles that end in parts
    (4, 1, [3, 5242880], [2, 1], 256, 0),                  # 39 / 201: warps share lines
    (8, 1, [51, 40, 80, 36], [3, 1, 2, 4], 256, 0),        # 33 / 76: long rows, few of them
    (8, 1, [40] * 4, [3, 1, 4, 2], 256, 0),                # small
    (4, 0, [1024, 1024], [2, 1], 256, 0),
    (4, 0, [24 << 18], [1], 256, 0),                       # contiguous
    (4, 1, [2048, 4096], [1, 2], 256, 0),
]


def test_tiled_engine_where_it_is_ahead(tmp_path):
    exe = str(tmp_path / "choice")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(HERE, "emul", "elem_choice.cpp"),
                    os.path.join(CSRC, "tb_perm_plan.cpp"), "-o", exe], check=True)
    lines = [" ".join(map(str, [es, add, len(d)] + d + p + [al])) for es, add, d, p, al, _ in CHOICES]
    out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.split()
    assert [int(x) for x in out] == [c[-1] for c in CHOICES], out
