"""Particle state in and out of the simulator: set_particles and read_particles
against the arrays themselves (copies: the tolerance is zero), for counts around
a warp and a block, every kind of source (host, device, strided, other dtypes)
and of destination (device, strided device, host, none)."""

import numpy as np
import pytest
import torch

from pfflip import Config, Simulator
from pfflip._arrays import as_tensor

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def state(n):
    rng = np.random.default_rng(n + 1)
    pos = rng.random((n, 3), dtype=np.float32)
    vel = rng.standard_normal((n, 3)).astype(np.float32)
    return pos, vel, rng.integers(0, 3, n).astype(np.int32)  # type 2 is not liquid


def sources(kind, pos, vel, typ):
    if kind == "host":
        return pos, vel, typ
    t = [torch.from_numpy(a).to(DEV) for a in (pos, vel, typ)]
    if kind == "strided":
        wide = [torch.zeros(len(pos), 7, device=DEV) for _ in range(2)]
        for w, a in zip(wide, t):
            w[:, 1:6:2] = a
        return wide[0][:, 1:6:2], wide[1][:, 1:6:2], t[2].repeat_interleave(2)[::2]
    if kind == "double":
        return t[0].double(), t[1].double(), t[2].long()
    return t


@pytest.mark.parametrize("kind", ["host", "device", "strided", "double"])
@pytest.mark.parametrize("n", [0, 1, 31, 257, 5000])
def test_particles_round_trip(n, kind):
    pos, vel, typ = state(n)
    sim = Simulator(Config(res=(6, 5, 4), dx=0.25, ppc=8, droplets=False, device=DEV))
    sim.set_particles(*sources(kind, pos, vel, typ))
    assert np.array_equal(sim.ptype.numpy(), (typ == 1).astype(np.int32))
    outs = [(None, None), tuple(torch.empty(n, 3, device=DEV) for _ in range(2)),
            tuple(torch.empty(n, 6, device=DEV)[:, ::2] for _ in range(2)),
            tuple(torch.empty(n, 3) for _ in range(2)), (None, torch.empty(n, 3, device=DEV))]
    for po, vo in outs:
        x, v = sim.read_particles(po, vo)
        assert (po is None or x is po) and (vo is None or v is vo)
        torch.cuda.synchronize()
        assert np.array_equal(x.cpu().numpy(), pos) and np.array_equal(v.cpu().numpy(), vel)


def test_read_particles_keeps_the_rules_of_in_place_writes():
    """Device tensors given to read_particles are written as by an in-place copy:
    a leaf that requires grad is refused, a tensor that autograd has saved is seen
    to have changed, inference tensors are refused outside inference mode, a
    tangent is dropped, and of overlapping outputs the velocities come last."""
    n = 300
    pos, vel, typ = state(n)
    sim = Simulator(Config(res=(6, 5, 4), dx=0.25, ppc=8, droplets=False, device=DEV))
    sim.set_particles(pos, vel, typ)
    new = lambda *a: torch.zeros(*a, device=DEV)  # noqa: E731
    for bad in ((new(n, 3).requires_grad_(), new(n, 3)), (new(n, 3), new(n, 3).requires_grad_())):
        with pytest.raises(RuntimeError):
            sim.read_particles(*bad)
    with torch.inference_mode():
        frozen = new(n, 3)
    with pytest.raises(RuntimeError):
        sim.read_particles(frozen, new(n, 3))
    for k in range(2):
        out = (new(n, 3), new(n, 3))
        p = torch.ones(1, device=DEV, requires_grad=True)
        y = (p * out[k]).sum()
        sim.read_particles(*out)
        assert np.array_equal(out[0].cpu().numpy(), pos) and np.array_equal(out[1].cpu().numpy(), vel)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.backward()
    import torch.autograd.forward_ad as fw

    with fw.dual_level():
        dual = fw.make_dual(new(n, 3), torch.ones(n, 3, device=DEV))
        sim.read_particles(dual, new(n, 3))
        primal, tangent = fw.unpack_dual(dual)
        assert np.array_equal(primal.cpu().numpy(), pos) and (tangent is None or not tangent.any())
    buf = new(n + 1, 3)
    sim.read_particles(buf[:n], buf[1:])
    assert np.array_equal(buf[1:].cpu().numpy(), vel) and np.array_equal(buf[0].cpu().numpy(), pos[0])


@pytest.mark.parametrize("res,ppc", [((6, 5, 4), 8), ((16, 16, 16), 8), ((33, 9, 12), 27)])
def test_phase_field_and_gradient_match_the_step_kernels(res, ppc):
    """phase_field forms the cell grid alone and its gradient in one pass: equal
    to the step's stages (same sums) and, for the gradient, to the general
    adjoint gather within the rounding of eight products, 1e-5 of the maximum."""
    import ctypes as C

    from pfflip import _native as N
    from pfflip import scenes
    from pfflip.adjoint import DiffSim

    cfg = Config(res=res, dx=1.0 / max(res), ppc=ppc, droplets=False, device=DEV)
    pos, _, typ = scenes.dam_break(cfg)
    ds = DiffSim(cfg, typ, 1e-3)
    x = torch.from_numpy(pos).to(DEV).requires_grad_(True)
    phi = ds.phase_field(x)
    w = torch.randn(res, device=DEV, generator=torch.Generator(DEV).manual_seed(1))
    (gx,) = torch.autograd.grad(phi, x, w)
    s = ds.sim
    s.set_particles(pos, np.zeros_like(pos), typ)
    s._p2g()
    s._phase_field_and_coefficients()
    assert np.abs(s.phi_cell.numpy() - phi.detach().cpu().numpy()).max() < 1e-5
    gcell = torch.empty_like(w)
    N.call("pf_adj_phase_cell", C.byref(s._g), N.ptr(s.cell_mass), w.data_ptr(), float(s.rho_min), float(cfg.alpha_phi),
           float(s.rho_0l), gcell.data_ptr(), N.stream())
    ga, gb = (torch.zeros(len(pos), 4, device=DEV) for _ in range(2))
    N.call("pf_adj_p2g", C.byref(s._g), len(pos), s._pos4.data_ptr(), s._vel4.data_ptr(), float(cfg.rho_l),
           float(cfg.rho_g), float(np.float32(cfg.r_p)), *(None,) * 6, gcell.data_ptr(), ga.data_ptr(), gb.data_ptr(),
           N.stream())
    ref = torch.empty(len(pos), 3, device=DEV)
    ref[s._ids().long()] = ga[:, :3]
    assert (ref - gx).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("hook", [lambda t: t.double(), lambda t: t.cpu(), lambda t: t.bfloat16()])
def test_phase_field_gradient_under_saved_tensor_hooks(hook):
    """What autograd saves may come back in another type, place or precision:
    the gradient is that of the particles as they were, with the slope of phi at
    the mass that came back, against the general adjoint gather at 1e-5 of the
    maximum (the rounding of eight products)."""
    import ctypes as C

    from pfflip import _native as N
    from pfflip import scenes
    from pfflip.adjoint import DiffSim

    cfg = Config(res=(12, 10, 8), dx=1.0 / 12, ppc=8, droplets=False, device=DEV)
    pos, _, typ = scenes.dam_break(cfg)
    ds = DiffSim(cfg, typ, 1e-3)
    s = ds.sim
    x = torch.from_numpy(pos).to(DEV).requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(hook, lambda t: t):
        phi = ds.phase_field(x)
    mass = hook(as_tensor(s.cell_mass)).to(DEV, torch.float32)
    w = torch.randn(cfg.res, device=DEV, generator=torch.Generator(DEV).manual_seed(1))
    gcell = torch.empty_like(w)
    N.call("pf_adj_phase_cell", C.byref(s._g), mass.data_ptr(), w.data_ptr(), float(s.rho_min), float(cfg.alpha_phi),
           float(s.rho_0l), gcell.data_ptr(), N.stream())
    ga, gb = (torch.zeros(len(pos), 4, device=DEV) for _ in range(2))
    N.call("pf_adj_p2g", C.byref(s._g), len(pos), s._pos4.data_ptr(), s._vel4.data_ptr(), float(cfg.rho_l),
           float(cfg.rho_g), float(np.float32(cfg.r_p)), *(None,) * 6, gcell.data_ptr(), ga.data_ptr(), gb.data_ptr(),
           N.stream())
    ref = torch.empty(len(pos), 3, device=DEV)
    ref[s._ids().long()] = ga[:, :3]
    (gx,) = torch.autograd.grad(phi, x, w)
    assert (ref - gx).abs().max() <= 1e-5 * ref.abs().max()
