"""The split step where its dispatch changes: at the block count up to which
k_step_pull holds back the next launch (518) and the piece count up to which
every piece has a warp of its own in k_step_interface (2960), in float32 rows
that are left unpadded, and on grids of more planes than a launch can have."""
import ctypes as C

import numpy as np
import pytest

from multicomponent_color_gradient_b200 import Solver, derive

pytestmark = pytest.mark.gpu


def _both(monkeypatch, case, steps):
    """Tiling, device bytes and results of the split step, and the march's results."""
    out = []
    z, y, x = np.meshgrid(*[np.arange(case[k]) for k in ("NZ", "NY", "NX")], indexing="ij")
    d = np.sqrt(sum((a - 0.45 * case[k]) ** 2 for a, k in ((x, "NX"), (y, "NY"), (z, "NZ"))))
    blue = 0.5 * (1 + np.tanh(0.9 * (0.3 * min(case["NX"], case["NY"], case["NZ"]) - d)))
    u = [4e-3 * np.sin(2 * np.pi * a / case[k]) for a, k in ((y, "NY"), (z, "NZ"), (x, "NX"))]
    F = [np.asarray(a, np.float32) for a in (1 - blue, blue, *u)]
    for march in (None, "0"):
        if march is None:
            monkeypatch.delenv("MCG_FUSED_PIPE", raising=False)
        else:
            monkeypatch.setenv("MCG_FUSED_PIPE", march)
        with Solver(case) as S:
            S.init_equilibrium(*F)
            S.step(steps)
            b = C.c_uint64()
            S._c("mcg_device_bytes", C.byref(b))
            out.append((S.tiling(), b.value, [*S.get_populations(), *S.get_fields().values()]))
    assert [o[0]["pipelined"] for o in out] == [3, 0]
    return out[0][0], out[0][1], out[0][2], out[1][2]


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic"])
@pytest.mark.parametrize("NY,NZ,blocks", [(46, 46, 484), (30, 76, 518), (30, 77, 525), (42, 76, 740), (49, 65, 756)])
def test_at_the_launch_limits(monkeypatch, storage, boundary, NY, NZ, blocks):
    """One piece a row: blocks below, at and just above 518; with 740 and 756
    blocks 2960 and 2961 pieces."""
    case = derive(dict(NX=30, NY=NY, NZ=NZ, boundary=boundary, storage=storage, tau=0.6, sigma=0.01, jet_radius=6.0,
                       inlet_noise=0.01, seed=3, NSTATS_START_STEP=10 ** 9))
    tiling, _, split, march = _both(monkeypatch, case, 9)
    assert tiling["y_tiles"] * tiling["z_chunks"] == blocks
    for a, b in zip(split, march):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("boundary", ["jet", "periodic"])
@pytest.mark.parametrize("NX", [64, 72, 88, 104, 120, 136, 168, 184, 216, 248])
def test_float32_rows_of_whole_sectors(monkeypatch, boundary, NX):
    """Float32 rows of a multiple of 8 columns, 64 or more, have no padding."""
    case = derive(dict(NX=NX, NY=9, NZ=8, boundary=boundary, tau=0.6, sigma=0.01, jet_radius=3.0,
                       inlet_noise=0.01, seed=3, NSTATS_START_STEP=10 ** 9))
    _, held, split, march = _both(monkeypatch, case, 6)
    for a, b in zip(split, march):
        np.testing.assert_array_equal(a, b)
    monkeypatch.setenv("MCG_FUSED_FIXED_NX", "0")  # plain rows
    _, plain, _, _ = _both(monkeypatch, case, 1)
    assert held == plain


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_more_planes_than_a_launch_has(storage):
    """Above 65535 interior planes, which the split step's grid cannot hold, a
    step is a march: a state that is the same in every plane gives each plane
    the sums of a short grid's."""
    W = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8, np.float32)
    sums = []
    for NZ, how in ((10, 3), (65537, 3), (65538, 0)):
        case = derive(dict(NX=6, NY=5, NZ=NZ, boundary="periodic", storage=storage, tau=0.6, sigma=0.01,
                           NSTATS_START_STEP=10 ** 9))
        row = (0.5 + 0.2 * np.sin(np.arange(30)))[None, None, :].astype(np.float32)
        fr = np.broadcast_to(W[:, None, None] * row, (27, NZ, 30)).reshape(27, -1)
        fb = np.broadcast_to(W[:, None, None] * (1 - row), (27, NZ, 30)).reshape(27, -1)
        with Solver(case) as S:
            S.set_populations(fr, fb)
            S.step(3)
            assert S.tiling()["pipelined"] == (0 if NZ - 2 > 65535 else 3) == how
            sums.append(S.conservation_sums() / (NZ - 2))
    for s in sums[1:]:
        # float64 sums of up to 2e7 equal terms
        np.testing.assert_allclose(s, sums[0], rtol=1e-9, atol=1e-9)
