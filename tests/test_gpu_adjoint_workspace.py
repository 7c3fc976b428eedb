"""Device memory that the adjoint runs keep for one another: a run on blocks
that hold another run's values gives the results of a run on new ones, from
several threads at once too, and the memory is given back with the last handle."""
import threading

import numpy as np
import pytest

from multicomponent_color_gradient_b200 import Solver, derive, get_case

pytestmark = pytest.mark.gpu


def _bubble(n):
    case = derive(dict(NX=n, NY=20, NZ=18, bubble_radius=5.0, tau=0.7, sigma=0.01, beta_recolor=0.7,
                       boundary="periodic", NSTATS_START_STEP=10 ** 9))
    S = Solver(case)
    S.init_bubble()
    target = np.linspace(-1, 1, S.N).astype(np.float32)
    return S, lambda: S.adjoint_run(target, 12, 3, tape=4)


def _jet():
    S = Solver(get_case("jet_24x40x24", NSTATS_START_STEP=10 ** 9))
    S.set_inlet_bessel([0.1, -0.05])
    S.init_jet()
    return S, lambda: S.adjoint_jet_run(16, 8, 15, 4, 5)


def _same(a, b):
    # float64 accumulators add block sums in any order; fields are computed alike
    for k in a:
        if k == "ms":
            continue
        if k == "dJ_du0":
            np.testing.assert_array_equal(a[k], b[k])
        else:
            np.testing.assert_allclose(a[k], b[k], rtol=1e-9, atol=0)


def test_runs_on_used_blocks_repeat():
    S0, bubble = _bubble(22)
    S1, bubble2 = _bubble(26)
    S2, jet = _jet()
    first = [f() for f in (bubble, jet, bubble2)]
    for _ in range(2):
        for f, r in zip((bubble2, bubble, jet), (first[2], first[0], first[1])):
            _same(f(), r)
    for S in (S0, S1, S2):
        S.close()


def test_runs_of_several_threads():
    made = [_bubble(22), _bubble(26), _jet()]
    want = [f() for _, f in made]
    got = [None] * 3

    def work(i):
        for _ in range(4):
            got[i] = made[i][1]()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        _same(g, w)
    for S, _ in made:
        S.close()


def test_memory_is_given_back_with_the_last_handle():
    import gc

    import torch

    gc.collect()
    S, run = _bubble(30)
    S.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    S, run = _bubble(30)
    run()
    S.close()
    assert torch.cuda.mem_get_info()[0] >= before
