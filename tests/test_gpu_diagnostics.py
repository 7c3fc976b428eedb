"""Conservation sums and the finite check against numpy on the downloaded
populations, on rows shorter than, equal to and longer than a warp's 32
columns and on the smallest grid.

Both sides add the same float32 values in float64, so a sum of n terms is
within n 2^-53 sum|term| of the exact one whatever the order."""
import numpy as np
import pytest

from helpers import CX, CY, CZ, grid, interior
from multicomponent_color_gradient_b200 import Solver, derive

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4), (33, 7, 5), (64, 5, 9), (97, 6, 4), (256, 4, 6)]


def _solver(shape, boundary, storage):
    NX, NY, NZ = shape
    case = derive(dict(NX=NX, NY=NY, NZ=NZ, boundary=boundary, storage=storage, tau=0.7, sigma=0.01, init_noise=1e-2,
                       seed=5, bubble_radius=2.0, NSTATS_START_STEP=10 ** 9))
    S = Solver(case)
    S.init_bubble()
    S.step(3)
    return case, S


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", ["periodic", "closed"])
@pytest.mark.parametrize("shape", SHAPES)
def test_conservation_sums_match_numpy(shape, boundary, storage):
    case, S = _solver(shape, boundary, storage)
    with S:
        got = S.conservation_sums()
        m = interior(case)
        fr, fb = (f.reshape(27, -1)[:, m].astype(np.float64) for f in S.get_populations())
    g = fr + fb
    for k, terms in enumerate((fr, fb, g * CX[:, None], g * CY[:, None], g * CZ[:, None])):
        bound = terms.size * 2.0 ** -53 * np.abs(terms).sum()
        assert abs(got[k] - terms.sum()) <= bound, (k, got[k], terms.sum(), bound)


@pytest.mark.parametrize("shape", SHAPES)
def test_check_finite_sees_one_bad_population(shape):
    case, S = _solver(shape, "closed", "f32")
    NX, NY, NZ = grid(case)
    with S:
        assert S.check_finite()
        fr, fb = S.get_populations()
        corners = [(1, 1, 1), (NX - 2, NY - 2, NZ - 2), (NX - 2, 1, NZ - 2), (1, NY - 2, 1)]
        for n, (x, y, z) in enumerate(corners):
            bad = (fr if n % 2 else fb).copy()
            bad[((7 * n) % 27) * S.N + x + NX * (y + NY * z)] = np.nan if n < 2 else np.inf
            S.set_populations(*((bad, fb) if n % 2 else (fr, bad)))
            assert not S.check_finite()
        S.set_populations(fr, fb)
        assert S.check_finite()
