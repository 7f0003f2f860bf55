"""The once-per-interval kernels (diagnostics, Stokes drift, stress('ocn'))
and the sea-ice wave height over blocks of 32 points: other direction counts
and level counts than the workloads', fewer levels than warps, wet counts
around a block, against the fp32 oracle with the tolerances of the existing
field tests (1e-3 relative, vectors and profiles of their largest value)."""
import numpy as np
import pytest

from helpers import rel_err, run_gpu, run_oracle, vec_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mm,nm,pm,om,kw", [(20, 17, 36, 37, {}), (35, 3, 8, 9, {}), (34, 3, 16, 64, {}),
                                            (13, 11, 48, 5, {}), (20, 17, 36, 37, {"fice0": 0.5}),
                                            (66, 3, 24, 30, {"fice0": 0.4})])
def test_interval_fields_vs_oracle(lib_built, oracle_mod, mm, nm, pm, om, kw):
    from umwm_gb300 import configs

    U = lib_built
    if nm > 3:
        case = configs.random_field(mm=mm, nm=nm, hours=1, dx=2000.0, pm=pm, om=om, dtg=120, **kw)
    else:
        case = configs.fetch_limited(mm=mm, nm=nm, hours=1, dx=3000.0, depth=60.0, pm=pm, om=om, dtg=120, xpl=2, ypl=2,
                                     **kw)
    stop = configs._time_str(case.start, 120)
    if case.forcing:
        snap = next(iter(case.forcing.values()))
        case.forcing[stop] = snap
    run_gpu(U, case, stop=stop)
    got = {n: U.get_field(n) for n in ("ht", "mwp", "mss", "mwl", "momx", "momy", "cgmxx", "cgmyy", "cgmxy", "dwp", "us",
                                       "vs", "ds", "ustar")}
    rows = U.get_screen()
    U.umwm_finalize()
    o = run_oracle(oracle_mod, case, 32, stop=stop)
    for n in ("ht", "mwp", "mss", "mwl", "ustar"):
        assert rel_err(got[n], o.get(n), 1e-6) < 1e-3, n
    assert vec_err(got["momx"], got["momy"], o.get("momx"), o.get("momy")) < 1e-3
    assert vec_err(got["cgmxx"], got["cgmyy"], o.get("cgmxx"), o.get("cgmyy")) < 1e-3
    us, vs = o.get("us").reshape(got["us"].shape), o.get("vs").reshape(got["vs"].shape)
    top = np.hypot(us, vs).max(1, keepdims=True) + 1e-12
    assert (np.abs(got["us"] - us) / top).max() < 1e-3 and (np.abs(got["vs"] - vs) / top).max() < 1e-3
    # the peak: the same bin, but for two bins within rounding of one another
    assert (np.abs(got["dwp"] - o.get("dwp")) > 1e-3 * o.get("dwp")).mean() <= 0.01
    so = o.get("screen")
    assert rows.shape == so.shape and rel_err(rows[:, 4], so[:, 4], 1e-6) < 1e-3
