"""The step in two launches (k_step_pull, k_step_interface) against the marches
in one launch (MCG_FUSED_PIPE=0): the same arithmetic in the same order, so
populations and fields are equal bit for bit, and the radial sums (float64
atomics in any order) to rounding.

Rows whose last piece of 32 columns is full, ragged or holds a single column,
rows whose columns do not fill 64 bytes, one-plane and one-row grids; states
with no interface, one interface and nothing but interface."""
import numpy as np
import pytest

from helpers import interior
from multicomponent_color_gradient_b200 import Solver, derive

pytestmark = pytest.mark.gpu


def _fields(case, mixture):
    NX, NY, NZ = case["NX"], case["NY"], case["NZ"]
    z, y, x = np.meshgrid(np.arange(NZ), np.arange(NY), np.arange(NX), indexing="ij")
    rng = np.random.default_rng(NX + 1000 * NY)
    if mixture == "pure":
        blue = np.zeros(x.shape)
    elif mixture == "drop":
        d = np.sqrt((x - 0.4 * NX) ** 2 + (y - 0.5 * NY) ** 2 + (z - 0.5 * NZ) ** 2)
        blue = 0.5 * (1 + np.tanh(0.9 * (0.25 * min(NX, NY, NZ) + 1 - d)))
    else:
        blue = 0.5 + 0.3 * (rng.random(x.shape) - 0.5)
    u = [4e-3 * np.sin(2 * np.pi * (a + rng.random())) for a in (y / NY, z / NZ, x / NX)]
    return [np.asarray(a, np.float32) for a in (1 - blue, blue, *u)]


def _run(case, mixture, steps, stats):
    with Solver(case) as S:
        S.init_equilibrium(*_fields(case, mixture))
        if stats:
            S.set_radial_statistics(1)
        S.step(steps)
        return S.tiling()["pipelined"], S.get_populations(), S.get_fields(), S.get_radial()


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic", "closed"])
@pytest.mark.parametrize("mixture", ["pure", "drop", "mixed"])
@pytest.mark.parametrize("shape", [(4, 4, 4), (33, 9, 6), (34, 6, 9), (66, 11, 5), (97, 8, 7), (128, 5, 6), (161, 6, 5),
                                   (256, 6, 7)])
def test_split_step_equals_march(monkeypatch, storage, boundary, mixture, shape):
    NX, NY, NZ = shape
    case = derive(dict(NX=NX, NY=NY, NZ=NZ, boundary=boundary, storage=storage, tau=0.6, sigma=0.01,
                       jet_radius=min(NX, NZ) / 5, inlet_noise=0.01, seed=3, NSTATS_START_STEP=10 ** 9))
    stats = boundary == "jet"
    monkeypatch.delenv("MCG_FUSED_PIPE", raising=False)
    how, pops, fields, radial = _run(case, mixture, 7, stats)
    assert how == 3
    monkeypatch.setenv("MCG_FUSED_PIPE", "0")
    how, mpops, mfields, mradial = _run(case, mixture, 7, stats)
    assert how == 0
    for a, b in zip(pops, mpops):
        np.testing.assert_array_equal(a, b)
    for k in fields:
        np.testing.assert_array_equal(fields[k], mfields[k], err_msg=k)
    assert np.isfinite(pops[0].reshape(27, -1)[:, interior(case)]).all()
    if stats:
        for k in ("sum_uy", "sum_uy2", "sum_ur", "sum_ur2", "sum_uruy"):
            # float32 run sums of at most 32 nodes are the same; their float64
            # totals differ by the order of at most 7*NX*NZ additions
            bound = 7 * NX * NZ * 2.0 ** -53 * 7 * NX * NZ * 0.1
            assert np.abs(radial[k] - mradial[k]).max() <= bound, k


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic", "closed"])
@pytest.mark.parametrize("shape", [(4, 4, 4), (33, 9, 6), (50, 7, 8), (97, 8, 7), (128, 5, 6), (200, 6, 5)])
def test_granular_sequence_equals_split_step(storage, boundary, shape):
    """The launchers one by one (k_moments, k_collide by the same pieces) give
    the split step's populations and fields bit for bit."""
    NX, NY, NZ = shape
    case = derive(dict(NX=NX, NY=NY, NZ=NZ, boundary=boundary, storage=storage, tau=0.6, sigma=0.01,
                       jet_radius=min(NX, NZ) / 5, inlet_noise=0.01, seed=3, NSTATS_START_STEP=10 ** 9))
    out = []
    for granular in (False, True):
        with Solver(case) as S:
            S.init_equilibrium(*_fields(case, "drop"))
            for _ in range(5):
                if not granular:
                    S.step(1)
                    continue
                S.launch_Macros()
                S.launch_collistream()
                if boundary == "jet":
                    S.launch_inlet_bc()
                    S.launch_neumann_bc()
            out.append((*S.get_populations(), *S.get_fields().values()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_back_to_back_steps_equal_waited_steps():
    """Launches of consecutive steps overlap (programmatic dependent launch);
    on a grid small enough to stay in L1 and L2 the result is that of steps
    that are waited for one by one."""
    case = derive(dict(NX=20, NY=12, NZ=10, boundary="periodic", tau=0.6, sigma=0.01, NSTATS_START_STEP=10 ** 9))
    out = []
    for waited in (False, True):
        with Solver(case) as S:
            S.init_equilibrium(*_fields(case, "mixed"))
            for _ in range(200):
                S.step(1)
                if waited:
                    S.synchronize()
            out.append(S.get_populations())
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic"])
@pytest.mark.parametrize("NY,NZ", [(47, 46), (48, 49), (56, 54), (58, 56)])
def test_small_grids_equal_march(monkeypatch, storage, boundary, NY, NZ):
    """Rows of one piece around the sizes up to which k_step_pull holds back the
    next launch (518 blocks of 4 pieces) and every piece has a warp of its own
    in k_step_interface (2960 pieces)."""
    case = derive(dict(NX=30, NY=NY, NZ=NZ, boundary=boundary, storage=storage, tau=0.6, sigma=0.01, jet_radius=6.0,
                       inlet_noise=0.01, seed=3, NSTATS_START_STEP=10 ** 9))
    monkeypatch.delenv("MCG_FUSED_PIPE", raising=False)
    _, pops, fields, _ = _run(case, "drop", 9, False)
    monkeypatch.setenv("MCG_FUSED_PIPE", "0")
    _, mpops, mfields, _ = _run(case, "drop", 9, False)
    for a, b in zip(pops, mpops):
        np.testing.assert_array_equal(a, b)
    for k in fields:
        np.testing.assert_array_equal(fields[k], mfields[k], err_msg=k)


@pytest.mark.parametrize("storage,NY", [("f32", 64), ("f32", 150), ("f16", 64), ("f16", 300)])
def test_pulls_of_buffers_that_fit_l2(monkeypatch, storage, NY):
    """Buffers that fit L2 are pulled with a hint that larger ones are not:
    either way the step is the march's bit for bit."""
    case = derive(dict(NX=66, NY=NY, NZ=66, boundary="periodic", storage=storage, tau=0.6, sigma=0.01,
                       NSTATS_START_STEP=10 ** 9))
    monkeypatch.delenv("MCG_FUSED_PIPE", raising=False)
    _, pops, fields, _ = _run(case, "drop", 4, False)
    monkeypatch.setenv("MCG_FUSED_PIPE", "0")
    _, mpops, mfields, _ = _run(case, "drop", 4, False)
    for a, b in zip(pops, mpops):
        np.testing.assert_array_equal(a, b)
    for k in fields:
        np.testing.assert_array_equal(fields[k], mfields[k], err_msg=k)


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic"])
def test_fields_in_chunks_equal_fields_at_once(storage, boundary):
    """A field read after a step forms and downloads the moments of a large grid
    in z-chunks; after launch_Macros of the same state they are there already
    and come whole.  The ghost planes are the same too."""
    case = derive(dict(NX=130, NY=131, NZ=270, boundary=boundary, storage=storage, tau=0.6, sigma=0.01,
                       jet_radius=8.0, bubble_radius=30.0, seed=2, init_noise=1e-3, NSTATS_START_STEP=10 ** 9))
    with Solver(case) as S:
        S.init_jet() if boundary == "jet" else S.init_bubble()
        S.step(3)
        chunked = S.get_fields()
        at_once = S.get_fields()
        for k in chunked:
            np.testing.assert_array_equal(chunked[k], at_once[k])
        S.step(1)
        only = S.get_stress()
        again = S.get_fields()
    with Solver(case) as S:
        S.init_jet() if boundary == "jet" else S.init_bubble()
        S.step(4)
        want = S.get_fields()
        np.testing.assert_array_equal(S.get_stress(), only)
        for k in want:
            np.testing.assert_array_equal(want[k], again[k])
