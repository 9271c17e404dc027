"""Launch shapes of the flux and viscous passes against the oracle, one step, at sizes where a shape
can go wrong: lines that fill no tile of 32, rows shorter than a warp (several in a group of x
faces), segments that leave a remainder of faces to a round, blocks of more warps than usual,
columns that fill no viscous tile, stored ghosts, and every width of stencil.

Bound: 1e-12 of each variable's norm after one step, as for the other parity cases: a step is about
a thousand operations deep in each direction, with 2.2e-16 each and no cancellation beyond that of
the transverse momenta (a tenth of the state).

Mixed form: a threshold of -1 or 1.01 makes every face a WENO or a central one, so that no sensor
crosses it differently.  A face flux (of the order of the pressure, 1) is a few roundings of 6e-8 off,
which moves a cell by a third of that a stage (the Courant number over two): 1e-7 to 2e-7 in a step,
bound 1e-6 of rho, rhou, rhoE and, of the perturbation-sized rhov and rhow, 1e-5.  A misplaced face
moves its cell by 1e-2."""
import numpy as np
import pytest

from conftest import channel_ini, requires_gpu

pytestmark = [pytest.mark.gpu, requires_gpu]


def step_errors(tmp_path, ini, tuning=None, steps=1, precision=0):
    from oracle_py import Oracle
    from streams_b200 import Case, Solver
    case = Case(tmp_path, ini)
    s = Solver.from_case(case, precision=precision)
    if tuning:
        s.set_tuning(*tuning)
    s.init_run()
    s.advance(steps)
    o = Oracle(tmp_path, ini)
    o.init_run()
    o.run(steps)
    g = o.ng
    a, b = s.copy_to_field()[:, g:-g, g:-g, g:-g], o.w()[:, g:-g, g:-g, g:-g]
    return [float(np.linalg.norm(a[m] - b[m]) / np.linalg.norm(b[m])) for m in range(5)]


@pytest.mark.parametrize("nx,ny,nz", [(5, 12, 7), (9, 16, 8), (31, 9, 33), (32, 17, 5), (33, 33, 18), (70, 41, 35)])
def test_odd_sizes(tmp_path, nx, ny, nz):
    assert max(step_errors(tmp_path, channel_ini(nx=nx, ny=ny, nz=nz))) <= 1e-12


@pytest.mark.parametrize("tuning", [(1024, 4), (1 << 26, 4), (1 << 26, 5), (4096, 16)])
def test_segments(tmp_path, tuning):
    assert max(step_errors(tmp_path, channel_ini(nx=37, ny=39, nz=34), tuning)) <= 1e-12


@pytest.mark.parametrize("kw", [dict(ep_order=8, weno_scheme=4), dict(ep_order=4, weno_scheme=2), dict(weno_version=1),
                                dict(flux_splitting=1), dict(nkeep=2), dict(ep_order=8, weno_scheme=4, nkeep=-1),
                                dict(ep_order=8, weno_scheme=4, nkeep=2)])
def test_stencil_widths(tmp_path, kw):
    assert max(step_errors(tmp_path, channel_ini(nx=33, ny=20, nz=19, **kw))) <= 1e-12


@pytest.mark.parametrize("precision", [0, 1])
def test_shortest_rows_with_the_widest_stencil(tmp_path, precision):
    """Rows of ng cells: the x pass's buffer at its largest."""
    ini = channel_ini(nx=4, ny=12, nz=5, ep_order=8, weno_scheme=4)
    if precision == 0:
        assert max(step_errors(tmp_path, ini)) <= 1e-12
    else:
        # FP32 fluxes of one step: a few hundred roundings of 6e-8 on perturbations of a tenth
        assert max(step_errors(tmp_path, ini, precision=1)) <= 1e-5


def test_several_groups_of_faces_and_long_lines(tmp_path):
    """Enough x faces for more than one group a warp, and lines longer than a round by far."""
    assert max(step_errors(tmp_path, channel_ini(nx=257, ny=49, nz=67))) <= 1e-12


def test_stored_ghosts_at_odd_sizes(tmp_path):
    from streams_b200.cases import bl_ini
    assert max(step_errors(tmp_path, bl_ini(nx=67, ny=48, nz=21))) <= 1e-12


def test_face_flux_from_lists_equals_inline_at_odd_sizes(tmp_path):
    """The WENO faces from the lists, or inside the passes: the same arithmetic."""
    from streams_b200 import Case, Solver
    ini = channel_ini(nx=45, ny=27, nz=22)
    out = []
    for frac in (0.0, 1.0):
        s = Solver.from_case(Case(tmp_path, ini))
        s.set_weno_split(frac)
        s.init_run()
        s.advance(2)
        out.append(s.copy_to_field())
    d = np.abs(out[0] - out[1]).max() / np.abs(out[0]).max()
    assert d <= 1e-14, d


MIXED_BOUND = (1e-6, 1e-6, 1e-5, 1e-5, 1e-6)


def assert_mixed(tmp_path, ini, tuning=None):
    errs = step_errors(tmp_path, ini, tuning, precision=1)
    assert all(e <= b for e, b in zip(errs, MIXED_BOUND)), errs


@pytest.mark.parametrize("sensor", [-1.0, 1.01])
@pytest.mark.parametrize("nx,ny,nz", [(5, 12, 7), (9, 16, 8), (31, 9, 33), (32, 17, 5), (70, 41, 35), (257, 49, 67)])
def test_odd_sizes_mixed(tmp_path, nx, ny, nz, sensor):
    assert_mixed(tmp_path, channel_ini(nx=nx, ny=ny, nz=nz, sensor=sensor))


@pytest.mark.parametrize("tuning", [(1024, 4), (1 << 26, 5)])
def test_segments_mixed(tmp_path, tuning):
    assert_mixed(tmp_path, channel_ini(nx=37, ny=39, nz=34, sensor=-1.0), tuning)


@pytest.mark.parametrize("kw", [dict(ep_order=8, weno_scheme=4), dict(ep_order=4, weno_scheme=2), dict(weno_version=1),
                                dict(flux_splitting=1)])
def test_stencil_widths_mixed(tmp_path, kw):
    assert_mixed(tmp_path, channel_ini(nx=33, ny=20, nz=19, sensor=-1.0, **kw))


@pytest.mark.parametrize("kw", [dict(nkeep=2), dict(nkeep=-1), dict(ep_order=8, weno_scheme=4, nkeep=2)])
def test_keep_fluxes_mixed(tmp_path, kw):
    assert_mixed(tmp_path, channel_ini(nx=33, ny=20, nz=19, sensor=1.01, **kw))


@pytest.mark.parametrize("sensor", [-1.0, 1.01])
def test_stored_ghosts_at_odd_sizes_mixed(tmp_path, sensor):
    from streams_b200.cases import bl_ini
    assert_mixed(tmp_path, bl_ini(nx=67, ny=48, nz=21, sensor=sensor))


def test_face_flux_from_lists_equals_inline_at_odd_sizes_mixed(tmp_path):
    """Every face a WENO face; the bound of the FP32 roundings, which the compiler may contract
    differently in the two kernels."""
    from streams_b200 import Case, Solver
    ini = channel_ini(nx=45, ny=27, nz=22, sensor=-1.0)
    out = []
    for frac in (0.0, 1.0):
        s = Solver.from_case(Case(tmp_path, ini), precision=1)
        s.set_weno_split(frac)
        s.init_run()
        s.advance(2)
        out.append(s.copy_to_field())
    d = np.abs(out[0] - out[1]).max() / np.abs(out[0]).max()
    assert d <= 1e-6, d


@pytest.mark.parametrize("kw", [dict(gas=True), dict(gas=True, flux_splitting=1), dict(gas=True, nkeep=2),
                                dict(visc_model=2)])
@pytest.mark.parametrize("nx,ny,nz", [(5, 12, 7), (31, 9, 33)])
def test_gas_and_viscosity_laws_at_odd_sizes(tmp_path, nx, ny, nz, kw):
    from streams_b200.cases import SYNTHETIC_CP_POLY
    kw = dict(kw)
    if kw.pop("gas", False):
        kw.update(cp_poly=SYNTHETIC_CP_POLY, mach=2.5)
    assert max(step_errors(tmp_path, channel_ini(nx=nx, ny=ny, nz=nz, **kw))) <= 1e-12


@pytest.mark.parametrize("tuning", [None, (1024, 4096)])
@pytest.mark.parametrize("ny,nz", [(12, 2500), (2500, 4)])
def test_lines_longer_than_a_segment_may_be(tmp_path, ny, nz, tuning):
    """More than 2048 cells in z or y: the second tuning asks for one segment a line and gets two."""
    assert max(step_errors(tmp_path, channel_ini(nx=5, ny=ny, nz=nz), tuning)) <= 1e-12
    assert_mixed(tmp_path, channel_ini(nx=5, ny=ny, nz=nz, sensor=-1.0), tuning)
