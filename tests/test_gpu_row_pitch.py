"""Population rows padded to whole pieces of 32 columns: the same results as
rows that are not (MCG_FUSED_FIXED_NX=0, the runtime-pitch kernels), through
every call that touches the buffers, and an adjoint run that finds no room for
padded buffers takes the padding out and gives the same gradient."""
import numpy as np
import pytest

from multicomponent_color_gradient_b200 import McgError, Solver, derive

pytestmark = pytest.mark.gpu


def _case(NX, boundary, storage):
    return derive(dict(NX=NX, NY=9, NZ=8, boundary=boundary, storage=storage, tau=0.6, sigma=0.01, jet_radius=3.0,
                       bubble_radius=3.0, init_noise=1e-3, seed=4, NSTATS_START_STEP=2))


def _walk(S, boundary):
    S.init_jet() if boundary == "jet" else S.init_bubble()
    S.step(4)
    fr, fb = S.get_populations()
    out = [fr, fb, S.conservation_sums()]
    S.set_populations(fb, fr)
    S.step(2)
    S.launch_Macros()
    S.launch_collistream()
    S.step(1)
    out += [*S.get_populations(), *S.get_fields().values(), S.get_stress()]
    assert S.check_finite()
    return out


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["jet", "periodic", "closed"])
@pytest.mark.parametrize("NX", [24, 31, 50, 63, 97, 121, 190, 225])
def test_padded_rows_give_the_same_results(monkeypatch, NX, boundary, storage):
    case = _case(NX, boundary, storage)
    with Solver(case) as S:
        a = _walk(S, boundary)
    monkeypatch.setenv("MCG_FUSED_FIXED_NX", "0")
    with Solver(case) as S:
        b = _walk(S, boundary)
    for u, v in zip(a, b):
        np.testing.assert_allclose(u, v, rtol=1e-12, atol=1e-12 if u.dtype == np.float64 else 0)


def test_adjoint_without_room_for_padding(monkeypatch):
    case = derive(dict(NX=97, NY=34, NZ=34, boundary="periodic", tau=0.7, sigma=0.01, bubble_radius=8.0,
                       NSTATS_START_STEP=10 ** 9))
    N = case["NX"] * case["NY"] * case["NZ"]
    target = np.linspace(-1, 1, N).astype(np.float32)
    with Solver(case) as S:
        S.init_bubble()
        want = S.adjoint_run(target, 12, 8, tape=0)
    with Solver(case) as S:
        S.init_bubble()
        S.step(1)
        fields = S.get_fields()
        S.init_bubble()
        # 7 held states, 2 work and 2 lambda buffers, and about 120 B a node
        # beside them: room for rows of 97 columns, not of 128
        plain, padded = (11 * 216 * (N // 97 * px) for px in (97, 128))
        monkeypatch.setenv("MCG_ADJOINT_MEMORY_MB", str((plain + padded) // 2 + 120 * N >> 20))
        got = S.adjoint_run(target, 12, 8, tape=0)
        np.testing.assert_array_equal(got["dJ_du0"], want["dJ_du0"])
        np.testing.assert_allclose([got[k] for k in ("J", "dJ_dsigma", "dJ_dtau")],
                                   [want[k] for k in ("J", "dJ_dsigma", "dJ_dtau")], rtol=1e-9)
        # the handle goes on from the same state
        S.step(1)
        again = S.get_fields()
        for k in fields:
            np.testing.assert_array_equal(fields[k], again[k])
        monkeypatch.setenv("MCG_ADJOINT_MEMORY_MB", "1")
        with pytest.raises(McgError) as err:
            S.adjoint_run(target, 12, 8)
        assert err.value.status == 2  # MCG_ERR_OOM
