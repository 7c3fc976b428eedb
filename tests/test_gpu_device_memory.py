"""Calls on a device that is nearly full: memory that the library uses for speed
(rows padded to whole pieces of 32 columns, blocks kept between adjoint runs) is
given up before a call that needs the room fails."""
import contextlib
import ctypes as C
import gc

import numpy as np
import pytest

from multicomponent_color_gradient_b200 import Solver, _lib, derive

pytestmark = pytest.mark.gpu

MB = 1 << 20
# 97 columns are padded to 128: 0.34 GB of 1.4 GB, far above what the allocator
# rounds (2 MB a buffer, fifteen buffers)
CASE = dict(NX=97, NY=160, NZ=160, boundary="periodic", tau=0.7, sigma=0.01, bubble_radius=20.0,
            NSTATS_START_STEP=10 ** 9)
PADDING = 2 * 216 * 160 * 160 * (128 - 97)


@contextlib.contextmanager
def only_free(bytes_free):
    """All but about `bytes_free` of the device's free memory taken."""
    import torch

    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - int(bytes_free), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def device_bytes(S):
    out = C.c_uint64()
    S._c("mcg_device_bytes", C.byref(out))
    return out.value


def walk(S):
    S.init_bubble()
    S.step(3)
    return S.get_fields()


def assert_same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_create_without_room_for_padded_rows():
    """A handle whose padded rows do not fit is made with the rows as they are,
    and gives the same results."""
    case = derive(CASE)
    with Solver(case) as S:
        padded = device_bytes(S)
        want = walk(S)
    plain = padded - PADDING
    with only_free((plain + padded) // 2):
        with Solver(case) as S:
            assert device_bytes(S) == plain
            got = walk(S)
    assert_same(got, want)
    # the padding it did without is there for the next handle
    with Solver(case) as S:
        assert device_bytes(S) == padded


def test_out_of_memory_does_not_reach_the_next_call():
    """A call that found no memory leaves nothing behind that a later launch
    would report as its own failure."""
    with only_free(64 * MB):
        with pytest.raises(_lib.McgError) as err:
            Solver(derive(CASE))
        assert err.value.status == 2  # MCG_ERR_OOM
        with Solver(derive(dict(CASE, NX=24, NY=20, NZ=20, bubble_radius=5.0))) as S:
            walk(S)


def test_output_without_room_beside_padded_rows(tmp_path):
    """A buffer that a handle needs later takes the place of its padding."""
    case = derive(CASE)
    with Solver(case) as S:
        S.init_bubble()
        S.step(3)
        S.write_vti(str(tmp_path / "roomy.vti"))
        S.step(2)
        want = S.get_fields()
    text = 32 * case["NX"] * case["NY"] * case["NZ"]  # base64 of 24 B a node
    with Solver(case) as S:
        S.init_bubble()
        S.step(3)
        padded = device_bytes(S)
        with only_free(text // 2):
            S.write_vti(str(tmp_path / "tight.vti"))
        assert device_bytes(S) == padded - PADDING
        S.step(2)
        assert_same(S.get_fields(), want)
    assert (tmp_path / "tight.vti").read_bytes() == (tmp_path / "roomy.vti").read_bytes()


def adjoint_case():
    case = derive(CASE)
    return case, np.linspace(-1, 1, case["NX"] * case["NY"] * case["NZ"]).astype(np.float32)


def assert_same_gradient(a, b):
    np.testing.assert_array_equal(a["dJ_du0"], b["dJ_du0"])
    # block sums added in any order
    np.testing.assert_allclose([a[k] for k in ("J", "dJ_dsigma", "dJ_dtau")],
                               [b[k] for k in ("J", "dJ_dsigma", "dJ_dtau")], rtol=1e-9)


def test_adjoint_in_the_room_of_the_padding(monkeypatch):
    """An adjoint run that fits beside a handle of plain rows fits beside one of
    padded rows, which gives its padding up."""
    import torch

    case, target = adjoint_case()
    monkeypatch.setenv("MCG_FUSED_FIXED_NX", "0")  # plain rows
    with Solver(case) as S:
        S.init_bubble()
        before = torch.cuda.mem_get_info()[0]
        want = S.adjoint_run(target, 3, 2, tape=2)
        need = before - torch.cuda.mem_get_info()[0]  # kept after the run
    assert need > 4 * PADDING
    monkeypatch.delenv("MCG_FUSED_FIXED_NX")
    with Solver(case) as S:
        S.init_bubble()
        S.step(1)
        fields = S.get_fields()
        S.init_bubble()
        with only_free(need - PADDING // 2):
            got = S.adjoint_run(target, 3, 2, tape=2)
        assert_same_gradient(got, want)
        S.step(1)
        assert_same(S.get_fields(), fields)


def test_memory_kept_between_adjoint_runs_is_there_for_others():
    """What the library keeps between adjoint runs does not stand in the way of
    an allocation beside it, and the next run does without it."""
    import torch

    case, target = adjoint_case()
    with Solver(case) as S:
        S.init_bubble()
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        want = S.adjoint_run(target, 3, 2, tape=2)
        kept = before - torch.cuda.mem_get_info()[0]
        with only_free(-kept // 2):
            pass
        assert_same_gradient(S.adjoint_run(target, 3, 2, tape=2), want)


@pytest.mark.parametrize("at_create", ["0", None])
def test_giving_padding_up_keeps_how_the_step_runs(monkeypatch, at_create):
    """How a handle's step runs is settled when the handle is made, not by the
    environment of the call that takes the padding out."""
    if at_create is not None:
        monkeypatch.setenv("MCG_FUSED_PIPE", at_create)
    else:
        monkeypatch.delenv("MCG_FUSED_PIPE", raising=False)
    case = derive(dict(CASE, NY=34, NZ=34, bubble_radius=8.0))
    N = case["NX"] * case["NY"] * case["NZ"]
    target = np.linspace(-1, 1, N).astype(np.float32)
    with Solver(case) as S:
        how = S.tiling()["pipelined"]
        assert how == (3 if at_create is None else 0)
        S.init_bubble()
        S.step(2)
        want = S.get_fields()
        S.init_bubble()
        if at_create is None:
            monkeypatch.setenv("MCG_FUSED_PIPE", "1")
        else:
            monkeypatch.delenv("MCG_FUSED_PIPE")
        padded = device_bytes(S)
        plain_run, padded_run = (11 * 216 * (N // 97 * px) for px in (97, 128))
        monkeypatch.setenv("MCG_ADJOINT_MEMORY_MB", str((plain_run + padded_run) // 2 + 120 * N >> 20))
        S.adjoint_run(target, 12, 8, tape=0)
        assert device_bytes(S) < padded
        assert S.tiling()["pipelined"] == how
        S.step(2)
        assert_same(S.get_fields(), want)
