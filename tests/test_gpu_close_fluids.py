"""Fluid pairs whose squared distance, or product of densities, is a subnormal
float act on each other with finite forces, as in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two", [False, True])  # parameters shared by all fluids, and their own
@pytest.mark.parametrize("rho", [1000.0, 6.0e-20])
def test_subnormal_values(ds, scenes, rho, two):
    r = scenes.Recipe("close")
    r.setDomain((0, 0, 0), (1.0, 1.0, 1.0))
    r.setGravity((0, 0, 0))
    h = 0.05
    p = np.zeros((4, 3))
    p[1, 0] = 1.0e-20 if rho == 1000.0 else 0.01  # squared 1e-40
    p[2], p[3] = (0.03, 0.02, 0.01), (0.02, 0.05, 0.03)
    r.addFluid(p, (0, 0, 0), h, rho, 20.0, 1.0e-6)
    if two:
        r.addFluid(np.array([[0.5, 0.5, 0.5]]), (0, 0, 0), h, 1.5 * rho, 25.0, 2.0e-6)
    r.setSimulationParameterTimeStep(1.0e-7)
    r.setSimulationParameterMaximumTime(1.0)
    r.setSimulationParameterNumFrames(1)
    b, sc = ds.build_scene(r)
    e = ds.Engine(sc)
    e.initialize()
    drho = np.zeros(sc.n_fluid)
    drho[1], drho[2] = 5.0e-4 * rho, 1.0e-3 * rho
    e.upload_fluids(drho=drho)
    e.update(1.0e-7, 1, 1, 1)
    for a in e.download_fluids():
        assert np.isfinite(a).all()
