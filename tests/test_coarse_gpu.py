"""The cluster kernel that runs the coarse end of the V-cycle (k_coarse), one
V-cycle at a time against the CPU oracle, at the sizes where its layout can go
wrong: rows that end inside a quad of cells, levels swept on one CTA and in
slabs of one, two and three planes, a coarsest level that is swept (on one CTA
and in slabs) or applied as a dense operator, a single level, no smoothing on
one side.

Tolerances: FP32 as the other V-cycle comparisons, 2e-4 of the maximum (FMA
contraction through up to 60 sweeps).  With 16-bit storage the kernel is held
to the separate sweeps of the same storage: about twenty roundings of relative
size 2^-11 lie between the two, 1e-2 of the maximum.
"""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from pfflip import _native as N
from pfflip import scenes
from pfflip._arrays import DeviceArray
from pfflip.poisson import MGPCG

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(a):
    return DeviceArray(torch.as_tensor(np.ascontiguousarray(a)).to(DEV, torch.float32))


def vcycle(res, bx, by, bz, b, **kw):
    g = MGPCG(res, DEV, **kw)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    z = DeviceArray.zeros(res, device=DEV)
    for _ in range(2):  # the second cycle starts from whatever the first left behind
        g.precondition(dev(b), z)
    return g, z.numpy().astype(np.float64)


def off(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


# extents: (first level, swept levels on a cluster, dense operator)
SHAPES = {
    (4, 4, 4): (0, 0, 0),  # a single level on one CTA
    (13, 11, 9): (0, 0, 0),  # a single odd level, swept; rows of 9
    (21, 23, 27): (0, 1, 0),  # a single odd level in slabs
    (24, 24, 24): (0, 2, 1),  # slabs, one CTA, dense 6^3
    (20, 20, 22): (0, 2, 0),  # 10 x 10 x 11 swept
    (30, 22, 18): (0, 2, 0),  # rows of 18 and 9
    (38, 44, 38): (0, 2, 0),  # three quads a thread, coarsest 19 x 22 x 19 in slabs
    (48, 32, 40): (0, 3, 1),  # two levels on the same CTAs
    (16, 64, 24): (0, 2, 1),  # one plane per slab
    (62, 30, 34): (0, 2, 0),  # four planes a slab, three quads a thread
    (64, 48, 48): (1, 2, 1),  # a launched level above
    (62, 60, 68): (1, 1, 0),  # a launched level above a swept 31 x 30 x 34
}


@pytest.mark.parametrize("stencil", ["flux", "reference"])
@pytest.mark.parametrize("res", SHAPES)
def test_coarse_vcycle_matches_oracle(res, stencil):
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=31)
    g, z = vcycle(res, bx, by, bz, b, pre=3, post=3, stencil=stencil)
    assert g.bottom_info() == SHAPES[res]
    o = O.OracleMGPCG(res, pre=3, post=3, stencil=stencil)
    o.build_hierarchy(bx, by, bz)
    assert off(z, o.precondition(b).astype(np.float64)) < 2e-4


@pytest.mark.parametrize("pre,post", [(0, 2), (2, 0), (1, 1)])
def test_coarse_vcycle_sweep_counts(pre, post):
    res = (24, 20, 36)
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=32)
    _, z = vcycle(res, bx, by, bz, b, pre=pre, post=post)
    o = O.OracleMGPCG(res, pre=pre, post=post)
    o.build_hierarchy(bx, by, bz)
    assert off(z, o.precondition(b).astype(np.float64)) < 2e-4


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("res", [(24, 24, 24), (30, 22, 18), (48, 32, 40), (62, 30, 34)])
def test_coarse_vcycle_16bit_matches_separate_sweeps(res, precision, monkeypatch):
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=33)
    z = {}
    for mode in ("cta", ""):
        monkeypatch.setenv("PFFLIP_MG_BOTTOM", mode)
        g, z[mode] = vcycle(res, bx, by, bz, b, pre=2, post=2, precision=precision)
    # bfloat16 keeps 8 bits where binary16 keeps 11
    assert off(z[""], z["cta"]) < (1e-2 if precision == "fp16" else 8e-2)


@pytest.mark.parametrize("stencil", ["flux", "reference"])
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("res,first", [((15, 15, 17), 0), ((27, 15, 9), 0), ((13, 11, 9), 0), ((28, 28, 5), 0),
                                       ((54, 30, 18), 0)])
def test_16bit_swept_coarsest_level_is_swept_in_binary64(res, first, precision, stencil, monkeypatch):
    """A coarsest level of up to 4096 cells, whatever its rows are padded to.  Two
    binary64 solves of it, with their sums in different orders, differ by some
    1e-14 and round to the same 16-bit values: none may differ by half a 16-bit
    step, 2^-12 (2^-9) of its size.  A binary32 one differs by some 1e-6 before the
    rounding, which showed at 1 to 3 values of these levels in FP16.  54 x 30 x 18
    has such a level below a smoothed one, whose sweeps the other kernel rounds:
    16-bit tolerance."""
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=36)
    z = {}
    for mode in ("cta", ""):
        monkeypatch.setenv("PFFLIP_MG_BOTTOM", mode)
        g, z[mode] = vcycle(res, bx, by, bz, b, pre=2, post=2, precision=precision, stencil=stencil)
    assert g.bottom_info()[0] == first
    if g.nlev > 1:
        assert off(z[""], z["cta"]) < (1e-2 if precision == "fp16" else 8e-2)
        return
    step = 2.0 ** (-12 if precision == "fp16" else -9)
    assert not (np.abs(z[""] - z["cta"]) > step * np.abs(z["cta"])).any()


def solves(g, res, b, tol, max_iter, one=True):
    """(iterations, residual, x) of the one-launch solve and of the launched CG
    (verbose solves take that one; with `one` False both do)."""
    out = []
    for verbose in (False, True):
        x, rhs = DeviceArray.zeros(res, device=DEV), dev(b)
        before = N.launch_count()
        it, rel = g.solve(rhs, x, tol=tol, max_iter=max_iter, verbose=verbose)
        assert (N.launch_count() - before == 1) == (one and not verbose)
        out.append((it, rel, x.numpy().astype(np.float64)))
    return out


@pytest.mark.parametrize("precision,stencil,tol", [("fp32", "flux", 1e-6), ("fp32", "reference", 1e-4), ("fp16", "flux", 1e-6)])
@pytest.mark.parametrize("res", [(4, 4, 4), (16, 16, 16), (13, 11, 9), (21, 23, 27), (20, 20, 22), (32, 32, 32),
                                 (38, 44, 38), (40, 40, 40)])
def test_one_launch_solve_matches_launched_cg(res, precision, stencil, tol):
    """Same iterations within 1; the solutions differ by what the tolerance
    leaves open, 10 tol of the maximum as in the comparisons with binary64."""
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=34)
    g = MGPCG(res, DEV, pre=3, post=3, precision=precision, stencil=stencil)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    # the binary64 operator of 8^3 cells leaves no room for the CG vectors
    one = precision == "fp32" or res not in ((16, 16, 16), (32, 32, 32))
    (i1, r1, x1), (i2, r2, x2) = solves(g, res, b, tol, 200, one)
    assert r1 < tol and r2 < tol and abs(i1 - i2) <= 1, (i1, r1, i2, r2)
    assert abs(x1.mean()) < 1e-6 * np.abs(x1).max()
    assert off(x1, x2) < 10 * tol


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("coarsest,max_iter,one", [(60, 1000, True), (60, 4000, False), (2000, 200, False), (2000, 10, True)])
def test_one_launch_is_bounded_in_time(coarsest, max_iter, one, precision):
    """A launch that could take above 0.25 s is left to the launched CG."""
    res = (13, 11, 9)  # one level, swept
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=38)
    g = MGPCG(res, DEV, coarsest=coarsest, precision=precision)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    x, rhs = DeviceArray.zeros(res, device=DEV), dev(b)
    before = N.launch_count()
    it, rel = g.solve(rhs, x, tol=1e-5, max_iter=max_iter)
    assert (N.launch_count() - before == 1) == one
    assert rel < 1e-5


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("max_iter", [0, 1, 2, 3])
@pytest.mark.parametrize("res", [(16, 16, 16), (13, 11, 9), (32, 32, 32)])
def test_one_launch_solve_leaves_the_vectors_of_the_launched_cg(res, max_iter, precision):
    """x, rhs and the last two residuals, as the launched CG leaves them, from
    vectors that hold something else before.  The iterates of the two part by
    rounding: 1e-4 of the maximum (of b for the residuals), 1e-2 where the
    preconditioner keeps 16 bits."""
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=37)
    g = MGPCG(res, DEV, pre=2, post=2, precision=precision)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    left = []
    for verbose in (False, True):
        for a in (g.x, g.rhs, g.res_v, g.r_prev):
            a.fill_(7.0)
        out = DeviceArray.zeros(res, device=DEV)
        g.solve(dev(b), out, tol=1e-30, max_iter=max_iter, verbose=verbose)
        left.append([a.numpy().astype(np.float64) for a in (g.x, g.rhs, g.res_v, g.r_prev, out)])
    for k, (a, c) in enumerate(zip(*left)):
        scale = np.abs(c if k in (0, 4) else left[1][1]).max()
        assert np.abs(a - c).max() <= (1e-4 if precision == "fp32" else 1e-2) * scale, k
    x, out = left[0][0], left[0][4]
    assert np.abs(x - x.mean() - out).max() <= 1e-6 * max(np.abs(x).max(), 1e-30)


@pytest.mark.parametrize("precision,stencil", [("fp32", "flux"), ("fp32", "reference"), ("fp16", "flux"), ("bf16", "flux")])
@pytest.mark.parametrize("res", [(13, 11, 9), (21, 23, 27), (24, 24, 24), (30, 22, 18), (40, 40, 40)])
def test_one_launch_solve_matches_binary64(res, precision, stencil):
    """The one-launch solve against the CPU oracle in binary64 at 1e-12: within
    10 tol of the maximum, as the other solves."""
    tol = 1e-6 if stencil == "flux" else 1e-4
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=39)
    g = MGPCG(res, DEV, pre=3, post=3, precision=precision, stencil=stencil)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    x, rhs = DeviceArray.zeros(res, device=DEV), dev(b)
    before = N.launch_count()
    it, rel = g.solve(rhs, x, tol=tol, max_iter=300)
    assert N.launch_count() - before == 1 and rel < tol, (it, rel)
    x64, _, _ = O.fp64_reference_solve(bx, by, bz, b.astype(np.float64), tol=1e-12)
    assert off(x.numpy().astype(np.float64), x64) < 10 * tol


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_launched_graph_and_eager_solves_are_bitwise_equal(precision):
    """Above the sizes that run in one launch, where use_graphs matters."""
    res = (64, 48, 48)
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=40)
    outs = []
    for graphs in (True, False, True):
        g = MGPCG(res, DEV, pre=3, post=3, use_graphs=graphs, precision=precision)
        g.build_hierarchy(dev(bx), dev(by), dev(bz))
        x, rhs = DeviceArray.zeros(res, device=DEV), dev(b)
        before = N.launch_count()
        outs.append((g.solve(rhs, x, tol=1e-6, max_iter=100), x.numpy()))
        assert N.launch_count() - before > 10
    for o in outs[1:]:
        assert o[0] == outs[0][0] and np.array_equal(o[1], outs[0][1])


@pytest.mark.parametrize("res", [(16, 16, 16), (32, 32, 32), (13, 11, 9)])
def test_one_launch_solve_stops_like_the_launched_cg(res):
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=35)
    g = MGPCG(res, DEV, pre=2, post=2)
    g.build_hierarchy(dev(bx), dev(by), dev(bz))
    for rhs, max_iter in ((np.zeros_like(b), 10), (b, 0), (b, 1), (b, 4)):
        (i1, r1, x1), (i2, r2, x2) = solves(g, res, rhs, 1e-30, max_iter)
        assert i1 == i2 and abs(r1 - r2) <= 1e-4 * r2, (max_iter, r1, r2)
        # the iterates of the two paths part by rounding
        assert np.abs(x1 - x2).max() <= 1e-4 * max(np.abs(x2).max(), 1e-30)
    bad = b.copy()
    bad[1, 2, 3] = np.nan
    with pytest.warns(RuntimeWarning):
        g.solve(dev(bad), DeviceArray.zeros(res, device=DEV))
