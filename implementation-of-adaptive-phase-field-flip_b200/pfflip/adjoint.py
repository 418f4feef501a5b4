"""Differentiable uniform PF-FLIP rollout.

The reference step (pfflip/sim.py:168-202) is not differentiable.  Here each
block of ``checkpoint_every`` steps is one ``torch.autograd.Function``.  Its
forward pass runs the plain step on the GPU and keeps only the particle state
at the start of the block.  Its backward pass replays the block to recover
the state before each step.  It then walks the steps in reverse: it re-runs
one step's grid stages and applies the hand-written adjoint kernels of
libpfflip.so (include/pfflip.h, "adjoint"):

    G2P + RK3 + reflection   -> pf_adj_g2p_advect   (scatter onto the faces)
    liquid extrapolation     -> pf_adj_extrapolate  (transposed sweeps)
    projection               -> pf_adj_project      (pressure and beta adjoints)
    pressure solve           -> a second MG-PCG solve with the same operator
    RHS/forces/beta/u = P/m  -> pf_adj_face_sources
    P2G                      -> pf_adj_p2g          (per-particle gather)
    sort                     -> pf_adj_unsort

Positions and velocities cross the autograd boundary as (n, 3) float32 CUDA
tensors in the caller's particle order.  Particle types are fixed.  Discrete
decisions are held fixed, so the gradient is the derivative of the step away
from its clamp/max kinks: sort order, liquid tags, extrapolation masks, wall
clamps and the valid-face test.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _native as N
from ._arrays import as_tensor
from .config import Config


class DiffSim:
    """Differentiable rollout of the uniform PF-FLIP step at a fixed dt.

    ``rollout(x, v, steps)`` returns the particle positions and velocities
    after ``steps`` steps; ``phase_field(x)`` returns the eq. (7) cell phase
    field of a particle set.  Both take part in torch autograd.
    """

    def __init__(self, cfg: Config, ptype, dt: float, checkpoint_every: int = 5, adjoint_tol: float | None = None,
                 adjoint_max_iter: int | None = None):
        from .sim import Simulator

        if cfg.k_div > 0:
            raise N.NativeError(N.PF_ERR_UNSUPPORTED, "the adjoint supports k_div = 0 only")
        if checkpoint_every < 1:
            raise ValueError("checkpoint_every must be >= 1")
        self.cfg = cfg
        self.dt = float(dt)
        self.k = int(checkpoint_every)
        self.adjoint_tol = float(cfg.pcg_tol if adjoint_tol is None else adjoint_tol)
        self.adjoint_max_iter = int(cfg.pcg_max_iter if adjoint_max_iter is None else adjoint_max_iter)
        self.sim = Simulator(cfg)
        if self.sim.has_solids:  # pragma: no cover - a fresh simulator has none
            raise N.NativeError(N.PF_ERR_UNSUPPORTED, "the adjoint does not support solids")
        dev = self.sim.dev
        t = ptype if isinstance(ptype, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(ptype))
        self.ptype = t.to(device=dev, dtype=torch.int32).reshape(-1)
        self.n = int(self.ptype.numel())
        fs = self.sim.face_shapes
        z = lambda s: torch.zeros(s, dtype=torch.float32, device=dev)  # noqa: E731
        self._gu = [z(s) for s in fs]
        self._gus = [z(s) for s in fs]
        self._gul = [z(s) for s in fs]
        self._tmp = [z(s) for s in fs]
        self._gbeta = [z(s) for s in fs]
        self._gmass = [z(s) for s in fs]
        self._gmom = [z(s) for s in fs]
        self._lv = [torch.empty(s, dtype=torch.uint8, device=dev) for s in fs]
        self._lv_tmp = [torch.empty(s, dtype=torch.uint8, device=dev) for s in fs]
        self._gp = z(self.sim.res)
        self._lam = z(self.sim.res)
        self._g4 = [torch.zeros((self.n, 4), dtype=torch.float32, device=dev) for _ in range(4)]
        self.adjoint_solves = []  # (iterations, residual) of every adjoint solve

    # ---------------------------------------------------------------- helpers
    def _load(self, x, v):
        self.sim.set_particles(x.detach(), v.detach(), self.ptype)

    def _to_ids(self, a4):
        """(n, 3) tensor in the caller's order from a float4 stream in array order."""
        out = torch.empty((self.n, 3), dtype=torch.float32, device=self.sim.dev)
        if self.n:
            N.call("pf_unpack_particles", self.n, N.sptr(self.sim._vel4), N.sptr(a4), out.data_ptr(), None, None,
                   N.stream())
        return out

    def _from_ids(self, gx, gv, gx4, gv4):
        """float4 streams in array order from (n, 3) tensors in the caller's order
        (None: zero)."""
        gx, gv = (None if g is None else g.to(device=self.sim.dev, dtype=torch.float32).contiguous() for g in (gx, gv))
        N.call("pf_gather_particles", self.n, N.sptr(self.sim._vel4), N.ptr(gx), N.sptr(gx4), N.ptr(gv), N.sptr(gv4),
               N.stream())

    def _grid_stages(self):
        """One step's forward grid stages on the current particles: sort, P2G,
        phi/beta, forces, solve, projection, extrapolation (no G2P/advection)."""
        s, dt = self.sim, self.dt
        s._p2g()
        s._phase_field_and_coefficients()
        s._add_forces(dt, save_vel_star=True)
        s._pressure_solve(dt)
        s._project(dt)
        s._extrapolate_liquid_velocity()

    def _step_adjoint(self, gpos4, gvel4, out_pos4, out_vel4):
        """Adjoint of the step whose grid stages were just run.  gpos4/gvel4
        hold the adjoints of the particles after the step (sorted order); the
        adjoints before the step's sort land in out_pos4/out_vel4."""
        s, cfg, dt = self.sim, self.cfg, self.dt
        g = C.byref(s._g)
        st = N.stream()
        P = N.ptr
        for a in self._gu + self._gus + self._gul:
            a.zero_()
        lo, hi = s._bounds()
        tmp_p, tmp_v = self._g4[2], self._g4[3]
        N.call("pf_adj_g2p_advect", g, self.n, s._pos4.data_ptr(), s._vel4.data_ptr(),
               *(P(a) for a in s.vel), *(P(a) for a in s.vel_star), *(P(a) for a in s.vel_liq),
               float(cfg.alpha_flip_liquid), float(cfg.alpha_flip_air), dt, lo, hi, 1, 1,
               gpos4.data_ptr(), gvel4.data_ptr(), tmp_p.data_ptr(), tmp_v.data_ptr(),
               *(P(a) for a in self._gu), *(P(a) for a in self._gus), *(P(a) for a in self._gul), st)
        N.call("pf_adj_extrapolate", g, P(s.is_liquid), int(cfg.extrap_cells), *(P(a) for a in self._gul),
               *(P(a) for a in self._tmp), *(P(a) for a in self._lv), *(P(a) for a in self._lv_tmp),
               *(P(a) for a in self._gu), st)
        N.call("pf_adj_project", g, P(s.pressure), *(P(a) for a in s.beta), *(P(a) for a in self._gu), dt,
               P(self._gp), *(P(a) for a in self._gbeta), st)
        it, rel = s.solver.solve(self._gp, self._lam, tol=self.adjoint_tol, max_iter=self.adjoint_max_iter)
        self.adjoint_solves.append((it, rel))
        N.call("pf_adj_face_sources", g, P(s.pressure), P(self._lam), *(P(a) for a in s.beta),
               *(P(a) for a in s.mass), *(P(a) for a in s.mom), P(s.is_liquid), float(1e-12 * s.rho_0l),
               float(s.rho_min), float(cfg.alpha_phi), float(s.rho_0l), float(cfg.rho_l), float(cfg.rho_g), dt,
               *(P(a) for a in self._gu), *(P(a) for a in self._gus), *(P(a) for a in self._gbeta),
               *(P(a) for a in self._gmass), *(P(a) for a in self._gmom), st)
        N.call("pf_adj_p2g", g, self.n, s._pos4.data_ptr(), s._vel4.data_ptr(), float(cfg.rho_l), float(cfg.rho_g),
               float(np.float32(cfg.r_p)), *(P(a) for a in self._gmass), *(P(a) for a in self._gmom), None,
               tmp_p.data_ptr(), tmp_v.data_ptr(), st)
        N.call("pf_adj_unsort", self.n, s._perm.data_ptr(), tmp_p.data_ptr(), tmp_v.data_ptr(),
               out_pos4.data_ptr(), out_vel4.data_ptr(), st)

    # ---------------------------------------------------------------- blocks
    def _forward_block(self, x, v, nsteps):
        self._load(x, v)
        for _ in range(nsteps):
            self.sim.step(self.dt)
        return self._to_ids(self.sim._pos4), self._to_ids(self.sim._vel4)

    def _field_arrays(self):
        s = self.sim
        return (*s.vel, *s.vel_star, *s.vel_liq, *s.beta, *s.mass, *s.mom, s.is_liquid, s.pressure)

    def _take_fields(self):
        """The sort permutation and the grid fields of the step just run, handed
        over as they are: the simulator goes on with fresh arrays, of which its
        next step writes every element."""
        s = self.sim
        perm, s._perm = s._perm, torch.empty_like(s._perm)
        fields = [a.tensor for a in self._field_arrays()]
        for a in self._field_arrays():
            a.tensor = torch.empty_like(a.tensor)
        return perm, fields

    def _own(self, perm, fields):
        self.sim._perm = perm
        for a, t in zip(self._field_arrays(), fields):
            a.tensor = t

    def _give_back(self, snap):
        """Make a step's state, as its grid stages left it, the simulator's."""
        s = self.sim
        p4, v4, taken = snap
        # copied back: the simulator's own streams may have been allocated on
        # another stream than this pass's, so they are neither dropped nor replaced
        s._pos4.copy_(p4)
        s._vel4.copy_(v4)
        self._own(*taken)
        s.solver.build_hierarchy(*s.beta)  # the adjoint solve uses this step's operator
        s._particles_changed()

    def _backward_block(self, x, v, nsteps, gx, gv):
        """Replay the block once, keeping each step's grid state (its sorted
        particles, permutation and fields: about 0.1 GB per step at 64^3 / 8
        ppc), then walk the steps in reverse, restoring that state for each
        step's adjoint instead of recomputing the step's grid stages."""
        s = self.sim
        self._load(x, v)
        own = s._perm, [a.tensor for a in self._field_arrays()]
        try:
            return self._replay_and_walk_back(nsteps, gx, gv)
        finally:  # the arrays the simulator was made with are its own again, after an error too
            self._own(*own)

    def _replay_and_walk_back(self, nsteps, gx, gv):
        s = self.sim
        s._particles_changed()  # step 0 sorts again (the identity), so its permutation maps onto this order
        snaps = []
        for k in range(nsteps):
            self._grid_stages()
            if k < nsteps - 1:  # the last step's state is used where it stands
                p4, v4 = s._pos4.clone(), s._vel4.clone()
                s._g2p_advect(self.dt, do_g2p=True, do_advect=True)
                snaps.append((p4, v4, self._take_fields()))
        ga, gb = self._g4[0], self._g4[1]
        self._from_ids(gx, gv, ga, gb)
        for k in range(nsteps - 1, -1, -1):
            if k < nsteps - 1:
                self._give_back(snaps.pop())
            # ga/gb are in the order of the arrays after the step, which is the
            # order after the step's sort; the result is in the order before it
            nxt_p, nxt_v = torch.empty_like(ga), torch.empty_like(gb)
            self._step_adjoint(ga, gb, nxt_p, nxt_v)
            ga, gb = nxt_p, nxt_v
        # step 0's sort was the identity on the loaded order, so the snapshot's
        # ids give the order ga/gb use
        return self._to_ids(ga), self._to_ids(gb)

    def rollout(self, x, v, steps: int):
        """Positions and velocities after ``steps`` steps of size dt."""
        left = int(steps)
        while left > 0:
            m = min(self.k, left)
            x, v = _Block.apply(x, v, self, m)
            left -= m
        return x, v

    def phase_field(self, x):
        """eq. (7) cell phase field of the particles at x (shape = cfg.res)."""
        return _Phase.apply(x, self)

    def _phase_forward(self, x):
        """phi of the particles at x, and what its gradient needs: the sorted
        particles, their places in the caller's order and the cell mass."""
        s, cfg = self.sim, self.cfg
        self._load(x, torch.zeros_like(x))
        # the cell grid alone: phi depends on nothing else
        N.call("pf_p2g", C.byref(s._g), self.n, N.sptr(s._pos4), N.sptr(s._vel4), s._cell_start.data_ptr(),
               float(cfg.rho_l), float(cfg.rho_g), float(np.float32(cfg.r_p)), *(None,) * 6, N.ptr(s.cell_mass),
               N.ptr(s.cell_wsum), N.stream())
        N.call("pf_phase_cell", C.byref(s._g), N.ptr(s.cell_mass), float(s.rho_min), float(cfg.alpha_phi),
               float(s.rho_0l), N.ptr(s.phi_cell), N.stream())
        return as_tensor(s.phi_cell).clone(), s._pos4.clone(), s._ids().clone(), as_tensor(s.cell_mass).clone()

    def _phase_backward(self, pos4, ids, cell_mass, gphi):
        s, cfg = self.sim, self.cfg
        gcell = torch.empty_like(cell_mass)
        N.call("pf_adj_phase_cell", C.byref(s._g), cell_mass.data_ptr(), gphi.data_ptr(), float(s.rho_min),
               float(cfg.alpha_phi), float(s.rho_0l), gcell.data_ptr(), N.stream())
        gx = torch.empty((self.n, 3), dtype=torch.float32, device=s.dev)
        N.call("pf_adj_phase_particles", C.byref(s._g), self.n, N.sptr(pos4), N.sptr(ids), float(cfg.rho_l),
               float(cfg.rho_g), float(np.float32(cfg.r_p)), gcell.data_ptr(), N.sptr(gx), N.stream())
        return gx


class _Block(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, v, dsim, nsteps):
        ctx.dsim = dsim
        ctx.nsteps = nsteps
        ctx.save_for_backward(x.detach().clone(), v.detach().clone())
        with torch.no_grad():
            return dsim._forward_block(x, v, nsteps)

    @staticmethod
    def backward(ctx, gx, gv):
        x, v = ctx.saved_tensors
        with torch.no_grad():
            ax, av = ctx.dsim._backward_block(x, v, ctx.nsteps, gx, gv)
        return ax, av, None, None


class _Phase(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, dsim):
        ctx.dsim = dsim
        with torch.no_grad():
            phi, pos4, ids, cell_mass = dsim._phase_forward(x.detach())
        # the streams hold integers in their words, which a saved-tensor hook may
        # not keep (and the kernel writes to the places that ids names), so only
        # the mass is saved as autograd saves
        ctx.particles = pos4, ids
        ctx.save_for_backward(cell_mass)
        return phi

    @staticmethod
    def backward(ctx, gphi):
        (mass,) = ctx.saved_tensors
        dev = ctx.dsim.sim.dev
        with torch.no_grad():
            mass, gphi = (t.to(device=dev, dtype=torch.float32).contiguous() for t in (mass, gphi))
            gx = ctx.dsim._phase_backward(*ctx.particles, mass, gphi)
        return gx, None


class RTAmplitudeGradient:
    """Gradient of the final interface-height variance of the Rayleigh-Taylor
    scene with respect to its 16 mode amplitudes a_k.

    The liquid (heavy, rho_l) tags are piecewise constant in a_k, so the
    amplitudes enter through the particle positions instead: the jittered
    lattice is tagged by its reference height (heavy above Ly/2) and displaced
    vertically by D a, D[p, k] = Ly sin^2(pi y/Ly) cos(2 pi (m_k x + n_k z))
    (scenes.rt_profile), which carries the plane Ly/2 onto the interface
    0.5 + sum_k a_k cos(...).  After ``steps`` steps the light-phase height of
    every (x, z) column is h = dx sum_y (1 - phi) and the loss is the variance
    of h over the columns.  d loss / d a = D^T (d loss / d x0) through the
    adjoint rollout (DiffSim) and the adjoint of eq. (7)."""

    def __init__(self, cfg: Config, dt: float, steps: int, checkpoint_every: int = 5,
                 adjoint_tol: float | None = 1e-6, n_modes: int = 16):
        from . import scenes

        pos_ref, ptype, amps, waves = scenes.rayleigh_taylor_lattice(cfg, n_modes)
        self.cfg = cfg
        self.steps = int(steps)
        self.amps0 = np.asarray(amps, np.float64)
        self.waves = np.asarray(waves)
        self.pos_ref_host = pos_ref
        self.ptype = ptype
        self.ds = DiffSim(cfg, ptype, dt, checkpoint_every=checkpoint_every, adjoint_tol=adjoint_tol)
        dev = self.ds.sim.dev
        ref = torch.from_numpy(pos_ref).to(dev)
        self.pos_ref = ref
        self.profile = scenes.rt_profile(ref.double(), self.waves, cfg.domain_size, xp=torch).float()

    def positions(self, a):
        """Initial positions for amplitudes a ((n_modes,) tensor)."""
        dy = self.profile @ a.to(device=self.profile.device, dtype=torch.float32)
        x = self.pos_ref
        return torch.stack((x[:, 0], x[:, 1] + dy, x[:, 2]), dim=1)

    def interface_variance(self, phi):
        h = (1.0 - phi.double()).sum(dim=1) * self.cfg.dx  # (nx, nz) light-phase column heights
        return ((h - h.mean()) ** 2).mean()

    def loss(self, a):
        x0 = self.positions(a)
        xT, _ = self.ds.rollout(x0, torch.zeros_like(x0), self.steps)
        return self.interface_variance(self.ds.phase_field(xT))

    def gradient(self, a=None):
        """(loss, d loss / d a) at amplitudes a (default: the seeded ones)."""
        a = torch.tensor(self.amps0 if a is None else a, dtype=torch.float64, device=self.ds.sim.dev,
                         requires_grad=True)
        loss = self.loss(a)
        loss.backward()
        return float(loss.detach()), a.grad.double().cpu().numpy()
