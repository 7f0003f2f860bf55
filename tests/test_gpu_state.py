"""State and network rows between host and device in pieces: more than one
piece with a ragged last one, fresh, touched and pinned destinations that do
not start a page, a wet count of one block and less, members of different
sizes, readers on two threads.  Copies and transposes are exact."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FP = ctypes.POINTER(ctypes.c_float)


def _domain(mm, nm, pm=36, om=37):
    from umwm_gb300 import configs

    return configs.fetch_limited(mm=mm, nm=nm, hours=1, dx=3000.0, depth=60.0, pm=pm, om=om, dtg=120, xpl=2, ypl=2)


@pytest.mark.parametrize("mm,nm,pm,om", [(131, 59, 36, 37), (160, 150, 48, 64), (34, 3, 8, 9), (13, 11, 16, 30)])
def test_state_round_trip(lib_built, mm, nm, pm, om):
    import torch

    from helpers import run_gpu

    U = lib_built
    run_gpu(U, _domain(mm, nm, pm, om), max_substeps=1)
    d = U.dims()
    shape = (d["im"], d["pm"], d["om"])
    rng = np.random.default_rng(5)
    F = rng.random(shape, dtype=np.float32)
    u = rng.random(d["im"], dtype=np.float32)
    U.set_state(F, u)
    got, gu = U.get_state()  # fresh pages
    assert np.array_equal(got, F) and np.array_equal(gu, u)
    n = F.size
    for buf in (np.full(n + 7, -1, np.float32), torch.full((n + 7,), -1.0, pin_memory=True).numpy(),
                np.zeros(n + 7, np.float32)):
        at = buf[3:3 + n]
        assert U.lib().umwm_gpu_get_state(at.ctypes.data_as(FP), None) == 0
        assert np.array_equal(at.reshape(shape), F)
        assert np.array_equal(buf[:3], buf[n + 3:n + 6])  # nothing beyond the state is written
    out = [None] * 3
    def read(i):
        out[i] = U.get_state()[0]
    th = [threading.Thread(target=read, args=(i,)) for i in range(3)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert all(np.array_equal(o, F) for o in out)
    U.umwm_finalize()


def test_member_states(lib_built):
    U = lib_built
    U.clear_inputs()
    for mm, nm in ((21, 11), (131, 59), (13, 9)):
        c = _domain(mm, nm)
        c.stage(U)
        U.ensemble_add(c.nml)
    U.ensemble_initialize()
    states = []
    for m in range(3):
        U.select_member(m)
        d = U.dims()
        states.append(np.random.default_rng(m).random((d["im"], d["pm"], d["om"]), dtype=np.float32))
        U.set_state(states[m])
    for m in range(3):
        U.select_member(m)
        assert np.array_equal(U.get_state()[0], states[m])
    U.umwm_finalize()


def test_network_rows_in_pieces(lib_built):
    """Rows are independent: a row of a batch of two pieces is what its part of
    the batch gives alone, to a few bf16 roundings of the hidden layers (another
    batch size may take other tiles): 2% of the largest output, where rows out
    of place would differ by about as much as the outputs themselves."""
    U = lib_built
    U.surrogate_init(37, 36, seed=3)
    X = np.random.default_rng(1).standard_normal((6500, U.SURROGATE_WIDTH), dtype=np.float32)
    X[:, 1341:] = 0
    Y = U.surrogate_forward(X)
    tol = 0.02 * np.abs(Y).max()
    for rows in (slice(6144, 6500), slice(6200, 6300), slice(0, 256)):
        assert np.abs(Y[rows] - U.surrogate_forward(X[rows])).max() <= tol
    T = np.zeros_like(X)
    loss, g = U.surrogate_grad(X[:6400], T[:6400])
    la, ga = U.surrogate_grad(X[:3200], T[:3200])
    lb, gb = U.surrogate_grad(X[3200:6400], T[3200:6400])
    # the mean over both halves' rows
    assert abs(loss - 0.5 * (la + lb)) <= 0.02 * loss
    assert np.abs(g - 0.5 * (ga + gb)).max() <= 0.05 * np.abs(g).max()


@pytest.mark.parametrize("shift", [0, 1, 6000])
def test_network_rows_in_place(lib_built, shift):
    """The outputs may overwrite the inputs: over the same rows, or `shift`
    rows on (12000 rows are two pieces; the same batch gives the same bits)."""
    U = lib_built
    U.surrogate_init(37, 36, seed=3)
    n, w = 12000, U.SURROGATE_WIDTH
    X = np.random.default_rng(2).standard_normal((n, w), dtype=np.float32)
    X[:, 1341:] = 0
    ref = U.surrogate_forward(X)
    for _ in range(3):
        buf = np.empty((n + shift, w), np.float32)
        buf[shift:] = X
        rc = U.lib().umwm_gpu_surrogate_forward(buf[shift:].ctypes.data_as(FP), n, buf.ctypes.data_as(FP))
        assert rc == 0
        np.testing.assert_array_equal(buf[:n], ref)
