"""Buffers allocated on first use when the device is nearly full: the call that
is short of memory reports it, and the model goes on as if it had not been made.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_ocean_buffers_short_of_memory(lib_built):
    import torch

    from umwm_gb300 import configs

    U = lib_built
    case = configs.random_field(mm=301, nm=287, hours=1, dx=2000.0, dtg=60)
    stop = configs._time_str(case.start, 60)
    case.forcing[stop] = case.forcing[case.start]

    def run(short):
        U.clear_inputs()
        case.stage(U)
        U.umwm_initialize(nml_text=case.nml)
        if short:
            d = U.dims()
            spec = 4 * d["im"] * d["pm"] * d["om"]  # bytes of one of the three source terms
            torch.cuda.empty_cache()
            keep = torch.empty(int(torch.cuda.mem_get_info()[0] - 1.4 * spec), dtype=torch.uint8, device="cuda")
            with pytest.raises(U.UmwmError):
                U.set_option("stress_ocn", 1)
            with pytest.raises(U.UmwmError):
                U.get_field("snl")
            del keep
            torch.cuda.empty_cache()
        U.set_option("stress_ocn", 1)
        U.umwm_run(case.start, stop)
        out = U.get_state()[0], U.get_field("snl"), U.get_field("taux_ocntop")
        U.umwm_finalize()
        return out

    for a, b in zip(run(True), run(False)):
        np.testing.assert_array_equal(a, b)


def test_network_batch_short_of_memory(lib_built):
    import torch

    U = lib_built
    U.surrogate_init(37, 36, seed=3)
    X = np.random.default_rng(4).standard_normal((30000, U.SURROGATE_WIDTH), dtype=np.float32)
    X[:, 1341:] = 0
    few = U.surrogate_forward(X[:256])
    torch.cuda.empty_cache()
    keep = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(U.UmwmError):
        U.surrogate_forward(X)
    del keep
    torch.cuda.empty_cache()
    np.testing.assert_array_equal(U.surrogate_forward(X[:256]), few)
    assert np.isfinite(U.surrogate_forward(X)).all()
