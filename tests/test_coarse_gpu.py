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


SHAPES = [
    (4, 4, 4),  # a single level on one CTA
    (13, 11, 9),  # a single odd level, swept; rows of 9
    (21, 23, 27),  # a single odd level in slabs
    (24, 24, 24),  # slabs, one CTA, dense 6^3
    (20, 20, 22),  # 10 x 10 x 11 swept
    (30, 22, 18),  # rows of 18 and 9
    (38, 44, 38),  # three quads a thread, coarsest 19 x 22 x 19 in slabs
    (48, 32, 40),  # two levels on the same CTAs
    (16, 64, 24),  # one plane per slab
    (62, 30, 34),  # a launched level above 31 x 15 x 17
]


@pytest.mark.parametrize("stencil", ["flux", "reference"])
@pytest.mark.parametrize("res", SHAPES)
def test_coarse_vcycle_matches_oracle(res, stencil):
    bx, by, bz, b, _ = scenes.solve_problem(res, seed=31)
    _, z = vcycle(res, bx, by, bz, b, pre=3, post=3, stencil=stencil)
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
