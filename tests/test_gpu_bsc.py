"""GPU checks of block-sparse contractions run as one grouped launch
(tb_bsc_*), against the per-block loop of plain contractions that the
reference's hierarchical layer issues (one talsh_tensor_contract per block)."""
import numpy as np
import pytest

import exatensor_b200 as XB
import oracle as O
from exatensor_b200 import blocksparse as BS

pytestmark = pytest.mark.gpu
PATTERN = "D(a,b,i,j)+=L(a,b,c,d)*R(c,d,i,j)"


def make_problem(xt, dev, dtk, nseg=3, lo=8, hi=24, presence=0.5, seed=7):
    rng = np.random.default_rng(seed)
    es = xt.ELEM_BYTES[dtk]
    segs = BS.random_segments(4, nseg, lo, hi, rng)   # a, b, c, d of L
    segr = [segs[2], segs[3]] + BS.random_segments(2, nseg, lo, hi, rng)  # c, d, i, j of R
    L = BS.BlockSparseTensor(segs, BS.random_keys(segs, presence, rng), es)
    R = BS.BlockSparseTensor(segr, BS.random_keys(segr, presence, rng), es)
    xt.fill_uniform(dtk, L.volume, L.data.data_ptr(), seed + 1, stream=dev.stream())
    xt.fill_uniform(dtk, R.volume, R.data.data_ptr(), seed + 2, stream=dev.stream())
    D, tasks, pairs = BS.contraction_tasks(PATTERN, L, R)
    xt.fill_uniform(dtk, D.volume, D.data.data_ptr(), seed + 3, stream=dev.stream())
    return L, R, D, tasks, pairs


def per_block_loop(xt, dev, dtk, D, tasks, alpha, accumulative, method=XB.METHOD_TTGT):
    """The reference's scheme: one plain contraction per block task."""
    import torch
    out = D.data.clone()
    base = D.data.data_ptr()
    if not accumulative:
        for key, (off, dims) in D.blocks.items():
            n = int(np.prod(dims)) * D.elem_bytes
            out[off * D.elem_bytes: off * D.elem_bytes + n].zero_()
    for dp, dd, lp, ld, rp, rd in tasks:
        xt.tensor_contract(PATTERN, dtk, dd, out.data_ptr() + (dp - base), ld, lp, rd, rp, alpha,
                           accumulative=True, plan=xt.make_plan(method), stream=dev.stream())
    torch.cuda.synchronize()
    return out


def values(D, buf, dtype):
    a = buf.cpu().numpy().view(dtype)
    parts = [a[off: off + int(np.prod(dims))] for off, dims in D.blocks.values()]
    return np.concatenate(parts)


@pytest.mark.parametrize("dtk,tol", [(O.R8, 1e-12), (O.R4, 1e-4)])
@pytest.mark.parametrize("accumulative,alpha", [(True, 1.0), (False, 0.5)])
def test_grouped_matches_per_block_loop(xt, dev, dtk, tol, accumulative, alpha):
    import torch
    L, R, D, tasks, pairs = make_problem(xt, dev, dtk)
    assert len(tasks) > len(D.blocks)  # some output blocks receive several products
    ref = per_block_loop(xt, dev, dtk, D, tasks, alpha, accumulative)
    plan = XB.BlockSparsePlan(PATTERN, dtk, tasks, alpha=alpha, accumulative=accumulative, stream=dev.stream())
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    xt.device_check(dev.stream())
    dt = O.NP_DTYPE[dtk]
    got, want = values(D, D.data, dt), values(D, ref, dt)
    assert O.rel_frobenius(got, want) <= tol
    inf = plan.info()
    assert inf.tasks == len(tasks) and inf.out_blocks == len(D.blocks)
    plan.close()


def test_graph_replay_is_deterministic(xt, dev):
    import torch
    L, R, D, tasks, _ = make_problem(xt, dev, O.R8, seed=11)
    plan = XB.BlockSparsePlan(PATTERN, O.R8, tasks, accumulative=False, stream=dev.stream())
    plan.execute(stream=dev.stream())
    first = D.data.clone()
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    assert torch.equal(first, D.data)
    plan.execute(stream=dev.stream(), graph=False)
    torch.cuda.synchronize()
    assert torch.equal(first, D.data)
    plan.close()


def test_autotune_leaves_output_and_keeps_accuracy(xt, dev):
    import torch
    L, R, D, tasks, _ = make_problem(xt, dev, O.R8, seed=13)
    before = D.data.clone()
    plan = XB.BlockSparsePlan(PATTERN, O.R8, tasks, accumulative=True, stream=dev.stream())
    plan.autotune(stream=dev.stream())
    torch.cuda.synchronize()
    assert torch.equal(before, D.data)
    inf = plan.info()
    assert inf.tile_n in (128, 256) and inf.slices in (6, 7)
    assert inf.tune_ms[0] > 0 and inf.tune_ms[2] > 0
    ref = per_block_loop(xt, dev, O.R8, D, tasks, 1.0, True)
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    assert O.rel_frobenius(values(D, D.data, np.float64), values(D, ref, np.float64)) <= 1e-12
    plan.close()


def test_one_block_against_the_oracle(xt, dev):
    """One output block receiving several products, checked against the
    double-double oracle."""
    import torch
    L, R, D, tasks, pairs = make_problem(xt, dev, O.R8, nseg=2, presence=1.0, seed=17)
    key = next(iter(D.blocks))
    mine = [(t, p) for t, p in zip(tasks, pairs) if p[0] == key]
    assert len(mine) >= 2
    plan = XB.BlockSparsePlan(PATTERN, O.R8, [t for t, _ in mine], alpha=-0.75, accumulative=False,
                              stream=dev.stream())
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    off, dims = D.blocks[key]
    n = int(np.prod(dims))
    got = D.data.cpu().numpy().view(np.float64)[off: off + n]
    lv = L.data.cpu().numpy().view(np.float64)
    rv = R.data.cpu().numpy().view(np.float64)
    cptrn, *_ = O.parse_pattern(PATTERN)
    acc = np.zeros(n)
    for _, (_, lk, rk) in mine:
        lo, ldims = L.blocks[lk]
        ro, rdims = R.blocks[rk]
        O.contract(cptrn, acc, dims, lv[lo: lo + int(np.prod(ldims))].copy(), ldims,
                   rv[ro: ro + int(np.prod(rdims))].copy(), rdims, -0.75, 0, True, mode=1)
    assert O.rel_frobenius(got, acc) <= 1e-12
    plan.close()


def test_mismatched_block_is_rejected(xt, dev):
    L, R, D, tasks, _ = make_problem(xt, dev, O.R8, seed=19)
    dp, dd, lp, ld, rp, rd = tasks[0]
    bad = [(dp, dd, lp, ld, rp, rd), (dp, dd, lp, [x + 1 for x in ld], rp, rd)]
    with pytest.raises(XB.TBError):
        XB.BlockSparsePlan(PATTERN, O.R8, bad, stream=dev.stream())


def fixed_problem(xt, dev, dtk, segl, segr, seed):
    """Every block present, with the given segment extents (L: a b c d; R: c d i j)."""
    import itertools
    es = xt.ELEM_BYTES[dtk]
    L = BS.BlockSparseTensor(segl, list(itertools.product(*[range(len(s)) for s in segl])), es)
    R = BS.BlockSparseTensor(segr, list(itertools.product(*[range(len(s)) for s in segr])), es)
    xt.fill_uniform(dtk, L.volume, L.data.data_ptr(), seed + 1, stream=dev.stream())
    xt.fill_uniform(dtk, R.volume, R.data.data_ptr(), seed + 2, stream=dev.stream())
    D, tasks, pairs = BS.contraction_tasks(PATTERN, L, R)
    return L, R, D, tasks


@pytest.mark.parametrize("dtk,tol", [(O.R8, 1e-12), (O.R4, 1e-4)])
@pytest.mark.parametrize("tile_n", [128, 256])
def test_wide_blocks_and_long_block_sums(xt, dev, dtk, tol, tile_n):
    """Output blocks of many N tiles (items are issued N tile by N tile),
    and one output block whose pairs sum 1056 K blocks of INT8 planes
    (more than one exact INT32 pass holds, so passes end at pair
    boundaries), against the per-block loop of plain contractions."""
    import torch
    probs = [
        # 11 pairs of K = 96 * 128 into one 128 x 64 block
        ([[16], [8], [96] * 11, [128]], [[96] * 11, [128], [8], [8]]),
        # 256 x 3072 blocks: 24 (12) N tiles of 128 (256) columns
        ([[16], [16], [8], [8, 16]], [[8], [8, 16], [64], [48]]),
    ]
    for i, (segl, segr) in enumerate(probs):
        L, R, D, tasks = fixed_problem(xt, dev, dtk, segl, segr, 40 + i)
        ref = per_block_loop(xt, dev, dtk, D, tasks, 1.0, False)
        plan = XB.BlockSparsePlan(PATTERN, dtk, tasks, accumulative=False, plan=xt.make_plan(tile_n=tile_n),
                                  stream=dev.stream())
        plan.execute(stream=dev.stream())
        torch.cuda.synchronize()
        xt.device_check(dev.stream())
        assert plan.info().tile_n == tile_n
        dt = O.NP_DTYPE[dtk]
        assert O.rel_frobenius(values(D, D.data, dt), values(D, ref, dt)) <= tol, (i, tile_n)
        plan.close()


def matrix_task(d, l, r, m, n, k):
    """D(a,i) += L(a,c) R(c,i) as one block task."""
    return (d.data_ptr(), [m, n], l.data_ptr(), [m, k], r.data_ptr(), [k, n])


MEMORY = """
import torch
import exatensor_b200 as XB
from tests.test_gpu_bsc import matrix_task
XB.device_init(0)
m, n, k = 50000, 256, 25000
l, r, d = [torch.empty(x, dtype=torch.float64, device="cuda").uniform_(-1, 1) for x in (m * k, k * n, m * n)]
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
plan = XB.BlockSparsePlan("D(a,i)+=L(a,c)*R(c,i)", XB.R8, [matrix_task(d, l, r, m, n, k)], accumulative=False,
                          stream=torch.cuda.current_stream())
plan.execute(stream=torch.cuda.current_stream())
torch.cuda.synchronize()
held = before - torch.cuda.mem_get_info()[0]
plan.close()
print("held", held, before - torch.cuda.mem_get_info()[0])
"""


def test_closed_plans_give_their_memory_back(xt):
    """Of a closed plan's 16 GB of planes at most the pool's 12 GB stay with the library
    (in a process of its own, whose pool starts empty)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", MEMORY], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    held, kept = [int(x) for x in r.stdout.split("held")[1].split()]
    assert held > 16 << 30
    assert kept <= (12 << 30) + (64 << 20)


ARITHMETIC = [("residues", {}), ("slices", dict(moduli=-1)), ("slices", dict(slices=7))]


def plan_of(xt, dev, tasks, arithmetic, options, **kw):
    plan = XB.BlockSparsePlan(PATTERN, O.R8, tasks, plan=xt.make_plan(**options), stream=dev.stream(), **kw)
    assert (plan.moduli() > 0) == (arithmetic == "residues")
    return plan


@pytest.mark.parametrize("arithmetic,options", ARITHMETIC)
def test_each_arithmetic_replays_tunes_and_matches(xt, dev, arithmetic, options):
    """Grouped result, graph replay, launches without the graph, and tuning, by residues
    and by slices (six, and seven so that the tuner times both), against the
    per-block loop."""
    import torch
    L, R, D, tasks, _ = make_problem(xt, dev, O.R8, seed=23)
    d0 = D.data.clone()
    ref = per_block_loop(xt, dev, O.R8, D, tasks, -0.75, True)
    plan = plan_of(xt, dev, tasks, arithmetic, options, alpha=-0.75)
    outs = []
    for graph in (True, True, False):
        D.data.copy_(d0)
        plan.execute(stream=dev.stream(), graph=graph)
        torch.cuda.synchronize()
        outs.append(D.data.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert O.rel_frobenius(values(D, outs[0], np.float64), values(D, ref, np.float64)) <= 1e-12
    D.data.copy_(d0)
    plan.autotune(stream=dev.stream())
    torch.cuda.synchronize()
    assert torch.equal(D.data, d0)
    inf = plan.info()
    timed = [x > 0 for x in inf.tune_ms]
    assert timed == ([True] * 4 if options.get("slices") == 7 else [True, False, True, False])
    assert arithmetic == "residues" or inf.slices in (6, 7)
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    xt.device_check(dev.stream())
    assert O.rel_frobenius(values(D, D.data, np.float64), values(D, ref, np.float64)) <= 1e-12
    plan.close()


@pytest.mark.parametrize("arithmetic,options", ARITHMETIC[:2])
@pytest.mark.parametrize("tile_n", [128, 256])
def test_each_arithmetic_on_wide_blocks(xt, dev, arithmetic, options, tile_n):
    """256 x 3072 output blocks, and blocks whose rows and columns end inside tiles."""
    import torch
    for segl, segr in [([[16], [16], [8], [8, 16]], [[8], [8, 16], [64], [48]]),
                       ([[13, 5], [11], [7], [9]], [[7], [9], [17], [3, 31]])]:
        L, R, D, tasks = fixed_problem(xt, dev, O.R8, segl, segr, 60)
        ref = per_block_loop(xt, dev, O.R8, D, tasks, 1.0, False)
        plan = plan_of(xt, dev, tasks, arithmetic, dict(options, tile_n=tile_n), accumulative=False)
        plan.execute(stream=dev.stream())
        torch.cuda.synchronize()
        xt.device_check(dev.stream())
        assert O.rel_frobenius(values(D, D.data, np.float64), values(D, ref, np.float64)) <= 1e-12
        plan.close()


@pytest.mark.parametrize("arithmetic,options", ARITHMETIC[:2])
def test_nan_and_infinity_in_a_block(xt, dev, arithmetic, options):
    """Rows and columns of the output whose operand rows hold a NaN or an infinity are NaN
    throughout; all others are what they are without them."""
    import torch
    segl, segr = [[13], [11], [7], [9]], [[7], [9], [17], [3, 31]]
    L, R, D, tasks = fixed_problem(xt, dev, O.R8, segl, segr, 70)
    plan = plan_of(xt, dev, tasks, arithmetic, options, accumulative=False)
    plan.execute(stream=dev.stream())
    clean = {k: D.data.view(torch.float64)[o:o + int(np.prod(d))].clone() for k, (o, d) in D.blocks.items()}
    lv, rv = L.data.view(torch.float64), R.data.view(torch.float64)
    off = L.blocks[(0, 0, 0, 0)][0]
    lv[off + 5 + 13 * 2 + 13 * 11 * 3] = float("nan")       # a = 5, b = 2
    lv[off + 7 + 13 * 10 + 13 * 11 * 20] = float("inf")     # a = 7, b = 10
    off = R.blocks[(0, 0, 0, 1)][0]
    rv[off + 4 + 63 * 8 + 63 * 17 * 30] = float("-inf")     # i = 8, j = 30 of the second block
    plan.execute(stream=dev.stream())
    torch.cuda.synchronize()
    for key, (o, dims) in D.blocks.items():
        got = D.data.view(torch.float64)[o:o + int(np.prod(dims))].view(tuple(reversed(dims)))  # j, i, b, a
        want = clean[key].view(tuple(reversed(dims))).clone()
        want[:, :, 2, 5] = float("nan")
        want[:, :, 10, 7] = float("nan")
        if key[3] == 1:
            want[30, 8] = float("nan")
        assert torch.equal(torch.isnan(got), torch.isnan(want)), key
        assert torch.equal(got.nan_to_num(), want.nan_to_num()), key
    plan.close()
