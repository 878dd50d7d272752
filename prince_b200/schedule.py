"""Host-side redshift schedule of one solve.

Everything here is scalar bookkeeping evaluated in float64 with the same
expressions as the reference solver, so the device sees the identical step
sizes, window boundaries and per-step scalars:

* the z grid of ``solve`` (``src/prince_cr/solvers/propagation.py:828-832``);
* the rate-cache windows: a refresh at ``z_k`` whenever
  ``|z_k - z_current| > threshold`` (``propagation.py:1383-1387``);
* per step ``h = z[k+1] - z[k]`` (``etd2.py:509-511``), ``dl/dz(z_k)``
  (``propagation.py:360-361``), ``H(z_k) cm2sec`` (the adiabatic loss scale,
  ``interaction_rates.py:1208``) and the injection prefactor
  ``dl/dz(z_k) * 1.0 * cm2sec`` (``propagation.py:366``).
"""

from __future__ import annotations

import math
from dataclasses import dataclass

import numpy as np

from . import constants as C


def z_grid(initial_z, final_z, dz):
    dz_step = -float(abs(dz))
    n_full = int(np.floor((final_z - initial_z) / dz_step))
    zg = initial_z + np.arange(n_full + 1) * dz_step
    if abs(zg[-1] - final_z) > 1e-12:
        zg = np.concatenate([zg, [final_z]])
    return zg


@dataclass
class Schedule:
    z: np.ndarray          # z grid (n_steps + 1)
    window: np.ndarray     # int32 window index of each step
    z_window: np.ndarray   # redshift of each window refresh
    h: np.ndarray
    dldz: np.ndarray
    hc: np.ndarray
    finj: np.ndarray

    @property
    def n_steps(self):
        return int(self.h.size)


def make_schedule(zg, threshold):
    zg = np.asarray(zg, dtype=np.float64)
    n_steps = max(zg.size - 1, 0)
    # Scalar evaluation per step: numpy's vectorised pow/sqrt paths can differ
    # from the scalar ones by an ulp, and the reference evaluates scalars.  Plain
    # floats give the same bits as numpy scalars (both are the C library's pow and
    # sqrt) in a tenth of the time.
    zs = zg[:n_steps].tolist()
    win, starts = [], []
    cur = None
    for z in zs:
        if cur is None or abs(z - cur) > threshold:
            cur = z
            starts.append(z)
        win.append(len(starts) - 1)
    if not starts:
        starts = [zg[0]]
    cm2sec = float(C.PRINCE_UNITS.cm2sec)
    om, ol, h0 = float(C.Omega_m), float(C.Omega_Lambda), float(C.H_0s)
    # the expressions of cosmology.H and cosmology.dldz (tests/test_schedule.py holds them together)
    hz = [h0 * math.sqrt(om * (1 + z) ** 3 + ol) for z in zs]
    dl = [-1.0 / ((1.0 + z) * h * cm2sec) for z, h in zip(zs, hz)]
    return Schedule(
        z=zg,
        window=np.array(win, dtype=np.int32),
        z_window=np.asarray(starts, dtype=np.float64),
        h=zg[1:] - zg[:-1],
        dldz=np.array(dl, dtype=np.float64),
        hc=np.array([h * cm2sec for h in hz], dtype=np.float64),
        finj=np.array([d * 1.0 * cm2sec for d in dl], dtype=np.float64),
    )
