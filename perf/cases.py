"""Cases whose speed is measured, through the package's public entry points.

The work of this library is dense tensor contraction, index permutation (copy),
permuted addition and block-sparse contraction, in R4, R8, C4 and C8.  Each
case is a dict of plain values; prepare() makes its tensors on the GPU, run()
makes one pass, exact() gives the result in 64 bits by plain torch.

Tensors are in Fortran order (first index fastest), so a tensor with extents
(n1, ..., nk) is a contiguous torch tensor of shape (nk, ..., n1).
"""
import math
import re

import numpy as np
import torch

import exatensor_b200 as tb
from exatensor_b200.blocksparse import BlockSparseTensor, contraction_tasks, random_keys, random_segments

KIND = {"R4": tb.R4, "R8": tb.R8, "C4": tb.C4, "C8": tb.C8}
DTYPE = {"R4": torch.float32, "R8": torch.float64, "C4": torch.complex64, "C8": torch.complex128}

LADDER = "D(a,b,i,j)+=L(a,b,c,d)*R(c,d,i,j)"   # coupled-cluster particle-particle ladder
RING = "D(a,i,b,j)+=L(a,k,c,i)*R(c,b,k,j)"     # coupled-cluster ring term
MIXED = "D(a,b,c,d)+=L(c,k,a,l)*R(l,d,k,b)"    # contracted and free indices interleaved
TRIPLES = "D(a,b,c,d,e,f)+=L(d,e,g,a)*R(g,f,b,c)"  # six-index output, one contracted index
# index transformations and contractions of the shapes of the reference's contraction corpus
CORPUS = [
    "D(a,b,c)+=L(b,d,a)*R(d,c)", "D(a,b,c)+=L(d,c,a)*R(b,d)", "D(a,b,c,d)+=L(d,b,e,a)*R(e,c)",
    "D(a,b,c,d)+=L(e,b,a,d)*R(c,e)", "D(a,b,c,d,e)+=L(e,f,b,a,d)*R(c,f)", "D(a,b,c,d)+=L(e,b)*R(a,e,c,d)",
    "D(a,b)+=L(a,c)*R(c,b)", "D(a,b)+=L(a,c,d)*R(d,b,c)", "D(a,b,c)+=L(a,c,d)*R(d,b)",
    "D(a,b,c)+=L(a,d,e,c)*R(e,b,d)", "D(a,b,c,d)+=L(a,e,b,f)*R(d,f,c,e)", "D(a,b,c,d)+=L(e,a,f,c)*R(b,f,d,e)",
    "D(a,b,c,d,e,f)+=L(d,f,g,b)*R(g,e,a,c)", "D(a,b,c,d,e,f)+=L(g,e,b,c)*R(d,f,g,a)",
]


def contract_case(pattern, kind, extents, alpha=1.0, accumulate=True, **more):
    """extents: "a=96 b=96 ..." (one entry for each index letter)."""
    return dict(op="contract", pattern=pattern, kind=kind, extents=extents, alpha=alpha, accumulate=accumulate, **more)


def ladder(kind, v, o, **more):
    return contract_case(LADDER, kind, "a=%d b=%d c=%d d=%d i=%d j=%d" % (v, v, v, v, o, o), **more)


def listed():
    return [
        # one block of a small blocked calculation, as a program that works block by block calls it thousands of
        # times: latency and launches
        dict(ladder("R8", 11, 5, alpha=0.5), name="contract_r8_block"),
        # an ordinary block with interleaved indices: the 40^6 single-block contraction
        contract_case(MIXED, "R8", "a=40 b=40 c=40 d=40 k=40 l=40", alpha=0.5, name="contract_r8_mixed40"),
        # the ladder of a medium molecule, double precision
        dict(ladder("R8", 96, 24), name="contract_r8_ladder96"),
        # the headline workload: virtual extent 192, occupied extent 48
        dict(ladder("R8", 192, 48), name="contract_r8_ladder192"),
        # ring term in complex double precision with odd extents, the left operand conjugated
        contract_case(RING.replace("L(", "L+("), "C8", "a=61 b=61 c=61 i=23 j=23 k=23", name="contract_c8_ring61"),
        # the ladder in single precision
        dict(ladder("R4", 128, 32), name="contract_r4_ladder128"),
        # an index transformation (one short index replaces a long one), single precision, result overwritten
        contract_case("D(a,b,c,d)+=L(d,b,e,a)*R(e,c)", "R4", "a=72 b=72 c=24 d=72 e=72", accumulate=False,
                      name="contract_r4_transform72"),
        # perturbative triples: a six-index result from one contracted index, bound by the result's traffic
        contract_case(TRIPLES, "R8", "a=19 b=19 c=19 d=19 e=19 f=19 g=19", alpha=-1.0, name="contract_r8_triples19"),
        # 256 MiB permutations: a full reversal of four indices, and a rank-5 tensor of odd extents
        dict(op="copy", kind="R8", dims="76 76 76 76", perm="4 3 2 1", name="copy_r8_reverse76"),
        dict(op="copy", kind="R4", dims="37 37 37 37 37", perm="3 1 5 2 4", name="copy_r4_rank5"),
        # antisymmetrisation-like update of an ordinary 40^4 block
        dict(op="add", kind="R8", dims="40 40 40 40", perm="3 1 4 2", alpha=-0.37, name="add_r8_40"),
        # block-sparse ladder: uneven segments, 30% of the blocks present, every block pair in one grouped call
        dict(op="blocks", kind="R8", nseg=4, lo=8, hi=48, presence=0.3, layout=1, name="blocks_r8"),
    ]


# ---- drawn cases ---------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_contract(rng):
    pattern = rng.choice([LADDER, RING, MIXED, TRIPLES, rng.choice(CORPUS), rng.choice(CORPUS)])
    kind = rng.choice(["R8", "R8", "R8", "R4", "R4", "C8", "C4"])
    cplx = kind[0] == "C"
    letters = sorted(set("".join(_labels(pattern)[k] for k in range(3))))
    flops = math.exp(rng.uniform(math.log(1e6), math.log(6e11 if kind[1] == "4" else 1e12)))
    products = flops / (8 if cplx else 2)
    # each index's extent around the geometric mean, occupied ones (i, j, k) shorter
    w = {x: rng.uniform(-0.5, 0.5) - (1.0 if x in "ijk" else 0.0) for x in letters}
    base = (math.log(products) - sum(w.values())) / len(letters)
    ext = {x: max(2, int(round(math.exp(base + w[x])))) for x in letters}
    es = {"R4": 4, "R8": 8, "C4": 8, "C8": 16}[kind]

    def volume():
        return sum(math.prod(ext[x] for x in g) for g in _labels(pattern)) * es

    while volume() > 1 << 30:
        big = max(ext, key=ext.get)
        ext[big] = max(2, int(ext[big] * 0.9))
    if cplx and rng.random() < 0.5:
        pattern = pattern.replace("L(", "L+(")
    return contract_case(pattern, kind, " ".join("%s=%d" % (x, ext[x]) for x in letters),
                         alpha=rng.choice([1.0, 0.5, -0.25]), accumulate=rng.random() < 0.8)


def _draw_permutation(rng, op):
    kind = rng.choice(["R8", "R8", "R4", "R4", "C8"])
    es = {"R4": 4, "R8": 8, "C8": 16}[kind]
    rank = rng.randint(2, 6)
    volume = math.exp(rng.uniform(math.log(1 << 16), math.log(1 << 28))) / es
    w = [rng.uniform(-0.7, 0.7) for _ in range(rank)]
    base = (math.log(volume) - sum(w)) / rank
    dims = [max(2, int(round(math.exp(base + x)))) for x in w]
    perm = list(range(1, rank + 1))
    while perm == sorted(perm):
        rng.shuffle(perm)
    case = dict(op=op, kind=kind, dims=" ".join(map(str, dims)), perm=" ".join(map(str, perm)))
    if op == "add":
        case["alpha"] = rng.choice([1.0, -0.37])
    return case


def draw(rng):
    op = rng.choice(["contract"] * 6 + ["copy"] * 3 + ["add"] * 2 + ["blocks"])
    if op == "contract":
        return _draw_contract(rng)
    if op in ("copy", "add"):
        return _draw_permutation(rng, op)
    return dict(op="blocks", kind=rng.choice(["R8", "R8", "R4"]), nseg=rng.randint(2, 4), lo=rng.randint(4, 12),
                hi=rng.randint(20, 56), presence=0.3, layout=rng.randint(2, 1000000))


# ---- what a case stands for ------------------------------------------------------
def _labels(pattern):
    return [g.replace(",", "") for g in re.findall(r"\(([^)]*)\)", pattern)]


def _extents(case):
    return {x.split("=")[0]: int(x.split("=")[1]) for x in case["extents"].split()}


def _dims(case):
    e = _extents(case)
    return [[e[x] for x in g] for g in _labels(case["pattern"])]


def _ints(text):
    return [int(x) for x in text.split()]


def _random(kind, n, gen, device="cuda"):
    """Uniform in [-1, 1), real and imaginary parts alike."""
    real = torch.float64 if kind[1] == "8" else torch.float32
    x = torch.empty(2 * n if kind[0] == "C" else n, dtype=real, device=device)
    x.uniform_(-1.0, 1.0, generator=gen)
    return torch.view_as_complex(x.view(n, 2)) if kind[0] == "C" else x


def _dense(kind, dims, gen):
    return _random(kind, math.prod(dims), gen).view(tuple(reversed(dims)))


_ready = []


def _inputs(case, seed):
    if not _ready:
        tb.device_init(torch.cuda.current_device())
        _ready.append(True)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if case["op"] == "contract":
        dd, ld, rd = _dims(case)
        letters = _labels(case["pattern"])
        k = math.prod(_extents(case)[x] for x in letters[1] if x in letters[2])
        left = _dense(kind, ld, gen)
        left *= 1.0 / math.sqrt(k)  # results of order one, whatever the contracted length
        return dict(d=_dense(kind, dd, gen), l=left, r=_dense(kind, rd, gen), dd=dd, ld=ld, rd=rd)
    if case["op"] in ("copy", "add"):
        dims, perm = _ints(case["dims"]), _ints(case["perm"])
        out = [0] * len(dims)
        for k, p in enumerate(perm):  # index k of the input becomes index p of the output
            out[p - 1] = dims[k]
        return dict(l=_dense(kind, dims, gen), d=_dense(kind, out, gen), dims=dims, perm=perm)
    # block-sparse: the block structure belongs to the case, the values to the seed
    rng = np.random.default_rng(case["layout"])
    es = 8 if kind == "R8" else 4
    virt, occ = random_segments(1, case["nseg"], case["lo"], case["hi"], rng)[0], \
        random_segments(1, case["nseg"], case["lo"], max(case["lo"], case["hi"] // 2), rng)[0]
    lseg, rseg = [virt] * 4, [virt, virt, occ, occ]
    lkeys, rkeys = random_keys(lseg, case["presence"], rng), random_keys(rseg, case["presence"], rng)
    if not any(a[2:] == b[:2] for a in lkeys for b in rkeys):
        lkeys, rkeys = lkeys + [(0, 0, 0, 0)], rkeys + [(0, 0, 0, 0)]
    left, right = BlockSparseTensor(lseg, lkeys, es), BlockSparseTensor(rseg, rkeys, es)
    for t in (left, right):
        t.data.view(DTYPE[kind]).copy_(_random(kind, max(1, t.volume), gen))
    out, tasks, pairs = contraction_tasks(LADDER, left, right, elem_bytes=es)
    return dict(d=out, l=left, r=right, tasks=tasks, pairs=pairs)


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"], state["kind"] = case, KIND[case["kind"]]
    if case["op"] == "blocks":
        state["plan"] = tb.BlockSparsePlan(LADDER, state["kind"], state.pop("tasks"))
        state["out"] = state["d"].data.view(DTYPE[case["kind"]])
    return state


def run(state):
    case = state["case"]
    if case["op"] == "contract":
        tb.tensor_contract(case["pattern"], state["kind"], state["dd"], state["d"].data_ptr(), state["ld"],
                           state["l"].data_ptr(), state["rd"], state["r"].data_ptr(), case["alpha"],
                           accumulative=case["accumulate"])
        return state["d"]
    if case["op"] == "copy":
        tb.tensor_copy(state["kind"], state["dims"], state["perm"], state["l"].data_ptr(), state["d"].data_ptr())
        return state["d"]
    if case["op"] == "add":
        tb.tensor_add(state["kind"], state["dims"], state["perm"], state["d"].data_ptr(), state["l"].data_ptr(),
                      case["alpha"])
        return state["d"]
    state["plan"].execute()
    return state["out"]


def work(case):
    es = {"R4": 4, "R8": 8, "C4": 8, "C8": 16}[case["kind"]]
    if case["op"] == "contract":
        dd, ld, rd = _dims(case)
        d = math.prod(dd) * (2 if case["accumulate"] else 1)
        products = math.prod(_extents(case).values())
        return {"bytes": (d + math.prod(ld) + math.prod(rd)) * es,
                "flops": (8 if case["kind"][0] == "C" else 2) * products}
    if case["op"] in ("copy", "add"):
        n = math.prod(_ints(case["dims"]))
        return {"bytes": (2 if case["op"] == "copy" else 3) * n * es, "flops": 0 if case["op"] == "copy" else 2 * n}
    rng = np.random.default_rng(case["layout"])
    virt = random_segments(1, case["nseg"], case["lo"], case["hi"], rng)[0]
    occ = random_segments(1, case["nseg"], case["lo"], max(case["lo"], case["hi"] // 2), rng)[0]
    lseg, rseg = [virt] * 4, [virt, virt, occ, occ]
    lkeys, rkeys = random_keys(lseg, case["presence"], rng), random_keys(rseg, case["presence"], rng)
    if not any(a[2:] == b[:2] for a in lkeys for b in rkeys):
        lkeys, rkeys = lkeys + [(0, 0, 0, 0)], rkeys + [(0, 0, 0, 0)]
    size = lambda seg, key: math.prod(seg[k][s] for k, s in enumerate(key))  # noqa: E731
    dseg, dkeys, flops = [virt, virt, occ, occ], set(), 0
    for a in set(lkeys):
        for b in set(rkeys):
            if a[2:] == b[:2]:
                dkeys.add(a[:2] + b[2:])
                flops += 2 * size(lseg, a) * occ[b[2]] * occ[b[3]]
    elems = sum(size(lseg, x) for x in set(lkeys)) + sum(size(rseg, x) for x in set(rkeys)) + \
        2 * sum(size(dseg, x) for x in dkeys)
    return {"bytes": elems * es, "flops": flops}


def tolerance(case):
    if case["op"] in ("copy", "add"):
        return "exact"  # a copy moves bits; an addition is one product and one sum, each rounded once
    # measured against exact(): 8-byte kinds up to 4e-14, 4-byte kinds up to 1.3e-5
    return {"rel": 2e-13} if case["kind"][1] == "8" else {"rel": 5e-5}


def exact(case, seed):
    s = _inputs(case, seed)
    wide = torch.complex128 if case["kind"][0] == "C" else torch.float64
    if case["op"] == "contract":
        pattern = case["pattern"]
        gd, gl, gr = _labels(pattern)
        left = s["l"].to(wide)
        if "L+(" in pattern:
            left = left.conj()
        right = s["r"].to(wide)
        # torch's index order is the reverse of the tensor's
        prod = torch.einsum("%s,%s->%s" % (gl[::-1], gr[::-1], gd[::-1]), left, right)
        prod *= case["alpha"]
        if case["accumulate"]:
            prod += s["d"]
        return prod
    if case["op"] in ("copy", "add"):
        rank, perm = len(s["dims"]), s["perm"]
        src = [0] * rank  # input index that output index p takes
        for k, p in enumerate(perm):
            src[p - 1] = k
        moved = s["l"].permute([rank - 1 - src[rank - 1 - q] for q in range(rank)])
        return moved.clone() if case["op"] == "copy" else s["d"].to(wide) + moved.to(wide) * case["alpha"]
    out = torch.zeros(s["d"].data.numel() // s["d"].elem_bytes, dtype=wide, device="cuda")

    def block(t, key):
        off, dims = t.blocks[key]
        flat = t.data.view(DTYPE[case["kind"]])
        return flat[off:off + math.prod(dims)].view(tuple(reversed(dims))).to(wide)

    for dk, lk, rk in s["pairs"]:
        off, dims = s["d"].blocks[dk]
        out[off:off + math.prod(dims)] += torch.einsum("dcba,jidc->jiba", block(s["l"], lk), block(s["r"], rk)).reshape(-1)
    return out
