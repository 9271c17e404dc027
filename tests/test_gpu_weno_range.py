"""WENO weights in FP64 where a flow's fluxes are far from 1: slow flows (u0 is the Mach number times
1.18), whose shear and energy fluxes scale as rho0 u0^2 and rho0 u0^3.  The smoothness indicators'
floor is 1e-6 or 1e-35 times the square of that, and the weights are formed from products of several
of them, so that data without differences (the channel's mean flow along x and z) meet the smallest
products.  Every face is a WENO face (sensor threshold -1).

Bound after one step: 1e-13 of rho, of rho0 c0 (momenta) and of rhoE.  A flux carries the pressure, of
order rho0 c0^2, about a hundred roundings of 1.1e-16 deep, and a step spans less than a cell at the
speed of sound, so that a step leaves at most a few 1e-14 of rho0 c0 in a momentum."""
import numpy as np
import pytest

from conftest import channel_ini, requires_gpu

pytestmark = [pytest.mark.gpu, requires_gpu]


@pytest.mark.parametrize("mach,kw", [
    (0.3, dict(flux_splitting=1, weno_version=1)),
    (1e-3, dict(flux_splitting=1, weno_version=1)),
    (1e-6, dict(flux_splitting=1, weno_version=1)),
    (1e-6, dict(flux_splitting=1)),
    (1e-5, dict(weno_version=1)),
    (1e-6, dict()),
])
def test_slow_mean_flow(tmp_path, mach, kw):
    from oracle_py import Oracle
    from streams_b200 import Case, Solver
    ini = channel_ini(nx=24, ny=20, nz=12, mach=mach, amp=0.0, sensor=-1.0, **kw)
    case = Case(tmp_path, ini)
    s = Solver.from_case(case)
    s.init_run()
    s.advance(1)
    o = Oracle(tmp_path, ini)
    o.init_run()
    o.run(1)
    g = o.ng
    a, b = s.copy_to_field()[:, g:-g, g:-g, g:-g], o.w()[:, g:-g, g:-g, g:-g]
    assert np.isfinite(b).all()
    p = case.params(0)
    scale = [p.rho0] + 3 * [p.rho0 * case.info()["u0"] / mach] + [np.abs(b[4]).max()]
    err = [float(np.abs(a[m] - b[m]).max() / scale[m]) for m in range(5)]
    assert max(err) <= 1e-13, err  # a NaN fails too
