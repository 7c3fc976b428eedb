"""The reverse step by pieces of 32 columns (k_adj_relax, k_adj_near) on rows
that end inside a piece, at its end and one column after it, with interfaces
across the box's wraps and the ends of pieces, with none and with nothing else:
the bubble's gradient against the oracle's float64 adjoint, the jet's against
float64 central differences.

Tolerances as for the other adjoint tests: the adjoint is float32, each value
within 1e-4 of the largest; the differences (steps 0.02 and 0.01, Richardson)
have a truncation error far below that."""
import numpy as np
import pytest
from scipy import special

from helpers import feq64
from multicomponent_color_gradient_b200 import Solver, derive
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SHAPES = [(5, 5, 5), (20, 9, 8), (33, 8, 10), (34, 10, 7), (66, 7, 8), (97, 6, 7)]


def _fields(case, mixture):
    NX, NY, NZ = case["NX"], case["NY"], case["NZ"]
    z, y, x = np.meshgrid(np.arange(NZ), np.arange(NY), np.arange(NX), indexing="ij")
    rng = np.random.default_rng(NX)
    if mixture == "mixed":
        blue = 0.5 + 0.3 * (rng.random(x.shape) - 0.5)
    else:
        d2 = 0.0
        for a, n in ((x, NX), (y, NY), (z, NZ)):  # around the corner of the periodic interior
            d = np.mod(a - 1, n - 2)
            d2 = d2 + np.minimum(d, n - 2 - d) ** 2
        r = 0.0 if mixture == "pure" else 2.5
        blue = 0.5 * (1 + np.tanh(2.0 * (r - np.sqrt(d2)))) if r else np.zeros(x.shape)
    u = [4e-3 * np.sin(2 * np.pi * (a + rng.random())) for a in (y / NY, z / NZ, x / NX)]
    return [np.asarray(a, np.float32) for a in (1 - blue, blue, *u)]


@pytest.mark.parametrize("mixture", ["pure", "drop", "mixed"])
@pytest.mark.parametrize("shape", SHAPES)
def test_bubble_gradient_matches_oracle(shape, mixture):
    NX, NY, NZ = shape
    case = derive(dict(NX=NX, NY=NY, NZ=NZ, boundary="periodic", tau=0.7, sigma=0.01, beta_recolor=0.7,
                       NSTATS_START_STEP=10 ** 9))
    F = _fields(case, mixture)
    rng = np.random.default_rng(7)
    target = rng.uniform(-1, 1, NX * NY * NZ).astype(np.float32)
    T = 5
    O = Oracle(case, 64)
    G = [f.astype(np.float64).reshape(-1) for f in F]
    O.set_fields(*G)
    O.set_populations(feq64(G[0], *G[2:]).reshape(-1), feq64(G[1], *G[2:]).reshape(-1))
    o = O.adjoint_periodic(target, T)
    with Solver(case) as S:
        for snapshots in (T + 1, 2):
            S.init_equilibrium(*F)
            r = S.adjoint_run(target, T, snapshots)
            assert abs(r["J"] - o["J"]) <= 1e-4 * o["J"]
            assert np.abs(r["dJ_du0"] - o["dJ_du0"]).max() <= 1e-4 * np.abs(o["dJ_du0"]).max()
            for k in ("dJ_dsigma", "dJ_dtau"):
                assert abs(r[k] - o[k]) <= 1e-4 * max(abs(o[k]), 1e-3 * o["J"]), k


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("shape", [(21, 14, 16), (33, 12, 18), (34, 11, 33), (66, 12, 20)])
def test_jet_gradient_matches_differences(shape, storage):
    NX, NY, NZ = shape
    case = derive(dict(NX=NX, NY=NY, NZ=NZ, boundary="jet", storage=storage, tau=0.6, sigma=0.005, jet_radius=4.0,
                       NSTATS_START_STEP=10 ** 9))
    T, t0, y0 = 12, 4, 2
    c0 = np.array([0.1, -0.05, 0, 0, 0, 0, 0, 0], np.float32)
    F = _fields(case, "pure")
    with Solver(case) as S:
        S.set_inlet_bessel(c0)
        S.init_equilibrium(*F)
        r = S.adjoint_jet_run(T, t0, T - 1, y0, 5)

    G = [f.astype(np.float64).reshape(-1) for f in F]
    x = np.arange(NX) - case["jet_x0"]
    z = np.arange(NZ) - case["jet_z0"]
    rad = np.sqrt(x[None, :] ** 2 + z[:, None] ** 2)

    def J(c):
        O = Oracle(dict(case, storage="f32"), 64)
        m = np.ones_like(rad)
        for ck, a in zip(c, special.jn_zeros(0, 8)):
            m += ck * special.j0(a * rad / case["jet_radius"])
        O.set_inlet_profile(m)
        O.set_populations(feq64(G[0], *G[2:]).reshape(-1), feq64(G[1], *G[2:]).reshape(-1))
        O.set_fields(*G)
        total = 0.0
        for t in range(T):
            O.step(1)
            if t >= t0:
                uy = O.get_fields()["uy"].reshape(NZ, NY, NX)[1:-1, y0:-1, 1:-1]
                total += 0.5 * float(np.sum(uy * uy))
        return total

    # float16 states are off by their rounding, 2^-11 of values of order 0.1
    tol = 1e-4 if storage == "f32" else 1e-2
    assert abs(r["J"] - J(c0.astype(np.float64))) <= tol * r["J"]
    for k in (0, 1, 3):
        d = []
        for h in (0.02, 0.01):
            e = np.zeros(8)
            e[k] = h
            d.append((J(c0 + e) - J(c0 - e)) / (2 * h))
        fd = (4 * d[1] - d[0]) / 3
        assert abs(r["dJ_dc"][k] - fd) <= tol * np.abs(r["dJ_dc"]).max(), (k, r["dJ_dc"][k], fd)
