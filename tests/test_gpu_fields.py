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


OCN_PAIRS = [("taux_ocntop", "tauy_ocntop"), ("taux_ocnbot", "tauy_ocnbot"), ("taux_snl", "tauy_snl"),
             ("epsx_ocn", "epsy_ocn"), ("epsx_atm", "epsy_atm"), ("tailocnx", "tailocny"), ("taux1", "tauy1"),
             ("taux2", "tauy2"), ("taux3", "tauy3")]


@pytest.mark.parametrize("mm,nm,pm,om,groups,kw", [(20, 17, 36, 37, 2, {}), (20, 17, 36, 37, 4, {}), (35, 3, 8, 9, None, {}),
                                                   (34, 3, 16, 64, 2, {}), (34, 3, 16, 64, 4, {}),
                                                   (13, 11, 48, 5, None, {}), (20, 17, 36, 37, None, {"fice0": 0.5}),
                                                   (66, 3, 24, 30, None, {"fice0": 0.4})])
def test_ocean_fields_vs_oracle(lib_built, oracle_mod, mm, nm, pm, om, groups, kw):
    """stress('ocn') and the source terms that the integration keeps for it, in
    one chunk of levels and in several, against the fp32 oracle: each vector to
    1e-3 of its largest (the field tests' bar), the downshifting part, a
    difference of near-equal terms, to 5e-3 (the bar of its existing test);
    the diagnostics' cross term to 1e-3 of the largest of the tensor."""
    from umwm_gb300 import configs

    U = lib_built
    if nm > 3:
        case = configs.random_field(mm=mm, nm=nm, hours=1, dx=2000.0, pm=pm, om=om, dtg=120, **kw)
    else:
        case = configs.fetch_limited(mm=mm, nm=nm, hours=1, dx=3000.0, depth=20.0, pm=pm, om=om, dtg=120, xpl=2, ypl=2,
                                     **kw)
    stop = configs._time_str(case.start, 120)
    if case.forcing:
        case.forcing[stop] = next(iter(case.forcing.values()))
    U.clear_inputs()
    case.stage(U)
    U.umwm_initialize(nml_text=case.nml)
    if groups is not None:
        U.set_option("direction_groups", groups)
    U.set_option("stress_ocn", 1)
    U.umwm_run(case.start, stop)
    got = {n: U.get_field(n) for n in [n for pair in OCN_PAIRS for n in pair] + ["cgmxx", "cgmxy", "cgmyy", "ssin", "sds"]}
    U.umwm_finalize()
    o = run_oracle(oracle_mod, case, 32, stop=stop)
    for n in ("ssin", "sds"):
        ref = o.get(n)
        assert np.abs(got[n] - ref).max() < 1e-3 * np.abs(ref).max(), n
    for nx, ny in OCN_PAIRS:
        assert vec_err(got[nx], got[ny], o.get(nx), o.get(ny)) < (5e-3 if nx == "taux_snl" else 1e-3), nx
    top = np.hypot(o.get("cgmxx"), o.get("cgmyy")).max()
    assert np.abs(got["cgmxy"] - o.get("cgmxy")).max() < 1e-3 * top
