"""Velocity-Verlet NVE molecular dynamics on the device, driven by the evaluator.

Positions, velocities and forces stay in HBM; a step is two kernels around one
evaluation from device-resident positions.  The neighbor graph is built with a skin and rebuilt
when the largest displacement since the last build exceeds skin/2, the reuse test of the
reference's calculator (symmetrix/source/symmetrix/calculator.py:2894-2899).
Units: eV, Angstrom, amu, fs.
"""
from __future__ import annotations

import numpy as np

from .evaluator import MACEB200, runs_own

ACCEL = 9.648533212331e-3      # (eV/A/amu) -> A/fs^2
KINETIC = 103.642696562621     # amu*A^2/fs^2 -> eV
KB = 8.617333262e-5            # eV/K
MASSES = {8: 15.999, 22: 47.867, 38: 87.62}


def maxwell_boltzmann(masses, temperature, seed):
    """Velocities (A/fs) at ``temperature`` with zero total momentum."""
    rng = np.random.default_rng(seed)
    masses = np.asarray(masses, dtype=np.float64)
    sigma = np.sqrt(KB * temperature / (masses * KINETIC))
    v = rng.normal(size=(len(masses), 3)) * sigma[:, None]
    v -= (masses[:, None] * v).sum(axis=0) / masses.sum()
    return v


class NVEIntegrator:
    def __init__(self, evaluator, positions, cell, types, masses, velocities, dt_fs=1.0, skin=0.5):
        import torch

        self.torch = torch
        self.ev = evaluator
        self.cell = np.asarray(cell, dtype=np.float64).reshape(3, 3)
        self.types = np.asarray(types, dtype=np.int32)
        self.dt = float(dt_fs)
        self.skin = float(skin)
        dev = torch.device("cuda")
        self.x = torch.from_numpy(np.asarray(positions, dtype=np.float64).reshape(-1, 3).copy()).to(dev)
        self.v = torch.from_numpy(np.asarray(velocities, dtype=np.float64).copy()).to(dev)
        self.m = torch.from_numpy(np.asarray(masses, dtype=np.float64).copy()).to(dev)[:, None]
        self.n = self.x.shape[0]
        self.rebuilds = 0
        self._build()
        self.f, self.potential = self._forces()

    def _build(self):
        host = self.x.cpu().numpy()
        res = self.ev._prepare_periodic_factorized_graph(self.types, host, self.cell, np.linalg.inv(self.cell),
                                                         self.ev.r_cut + self.skin)
        self.generation = res["generation"]
        self.x_ref = self.x.clone()
        self.rebuilds += 1

    def _evaluate(self, moved):
        if moved > (0.5 * self.skin) ** 2:
            self._build()
        self.ev.compute_positions_device(self.generation, self.x.data_ptr())

    def _forces(self):
        from .distributed import _as_tensor

        torch = self.torch
        self._evaluate(float(((self.x - self.x_ref) ** 2).sum(dim=1).max()))
        _e, f_ptr, _v = self.ev.device_results()
        forces = _as_tensor(torch, f_ptr, (self.n, 3), torch.float64, self.x.device).clone()
        return forces, self.ev.energy

    def kinetic(self):
        return float(0.5 * KINETIC * (self.m * self.v * self.v).sum())

    def _plain(self):
        """The state is as it was set up here, and not tensors of another type, shape or layout put in its place, and neither the
        integrator nor the evaluator has its own forces, kinetic energy or step (a restraint, a bias force)."""
        torch, device = self.torch, self.x_ref.device
        if not runs_own(self, NVEIntegrator, _STEP_METHODS) or not runs_own(self.ev, MACEB200, _EVALUATOR_METHODS):
            return False
        if not isinstance(self.dt, (int, float)):
            return False
        return all(type(t) is torch.Tensor and t.dtype == torch.float64 and t.shape == shape and t.is_contiguous()
                   and t.device == device and not t.requires_grad
                   for t, shape in ((self.x, (self.n, 3)), (self.v, (self.n, 3)), (self.f, (self.n, 3)), (self.m, (self.n, 1)),
                                    (self.x_ref, (self.n, 3))))

    def step(self):
        half = 0.5 * self.dt * ACCEL
        if self._plain():
            stream = self.torch.cuda.current_stream(self.x.device).cuda_stream
            x, v, m = self.x.data_ptr(), self.v.data_ptr(), self.m.data_ptr()
            self._evaluate(self.ev.md_advance(stream, self.n, self.dt, half, x, v, self.f.data_ptr(), m, self.x_ref.data_ptr()))
            forces = self.torch.empty_like(self.x)
            twice_kinetic = self.ev.md_finish(stream, self.n, half, v, m, forces.data_ptr())
            self.f = forces
            self.potential = self.ev.energy
            return self.potential + 0.5 * KINETIC * twice_kinetic
        self.v += half * self.f / self.m
        self.x += self.dt * self.v
        self.f, self.potential = self._forces()
        self.v += half * self.f / self.m
        return self.potential + self.kinetic()

    def run(self, steps):
        """Returns total energies (eV) at step 0..steps."""
        energies = [self.potential + self.kinetic()]
        for _ in range(steps):
            energies.append(self.step())
        return np.array(energies)


# what the integrator and its evaluator must run for the two step kernels to take the tensor expressions' place
_STEP_METHODS = {"_forces": NVEIntegrator._forces, "kinetic": NVEIntegrator.kinetic}
_EVALUATOR_METHODS = {name: getattr(MACEB200, name) for name in ("device_results", "md_advance", "md_finish")}
