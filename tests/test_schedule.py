"""The schedule's per-step scalars are the cosmology's, bit for bit (no GPU)."""

import numpy as np
import pytest

from prince_b200 import constants as C
from prince_b200.cosmology import H, dldz
from prince_b200.schedule import make_schedule, z_grid


@pytest.mark.parametrize("initial_z,final_z,dz", [(1.0, 0.0, 1e-3), (0.05, 0.0, 1e-3), (6.0, 0.0, 7.3e-3), (3.3, 0.7, 1e-2),
                                                  (0.0123, 0.0, 1e-3)])
def test_step_scalars_are_the_cosmology_s(initial_z, final_z, dz):
    zg = z_grid(initial_z, final_z, dz)
    s = make_schedule(zg, 0.01)
    cm2sec = C.PRINCE_UNITS.cm2sec
    dl = np.array([dldz(z) for z in zg[:-1]])
    assert s.n_steps == zg.size - 1
    assert np.array_equal(s.dldz, dl)
    assert np.array_equal(s.hc, np.array([H(z) * cm2sec for z in zg[:-1]]))
    assert np.array_equal(s.finj, np.array([d * 1.0 * cm2sec for d in dl]))
    assert np.array_equal(s.h, np.diff(zg))
