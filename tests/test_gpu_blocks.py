"""The spectral kernels' block mapping (a warp per 32 consecutive wet points,
the levels shared out over the warps) where it can go wrong: every direction
count with an instance, wet-point counts around a block and a tile, fewer
levels than warps, and the split of the levels, which must not change a bit.
"""
import numpy as np
import pytest

from helpers import lonlat_grid, run_gpu, run_oracle, spec_stats

pytestmark = pytest.mark.gpu


def _case(wet, **kw):
    """A channel of `wet` points in one row (the regional grid's rim is land)."""
    from umwm_gb300 import configs

    return configs.fetch_limited(mm=wet + 2, nm=3, hours=1, dx=3000.0, xpl=2, ypl=2, **kw)


@pytest.mark.parametrize("pm,om", [(8, 37), (12, 20), (16, 33), (24, 9), (32, 25), (36, 64), (48, 37)])
def test_direction_counts_vs_oracle(lib_built, oracle_mod, pm, om):
    """Two substeps against the fp32 oracle.  The tolerance of the existing
    one-substep parity tests (1e-5 relative L2), twice for the two steps."""
    from umwm_gb300 import configs

    U = lib_built
    case = configs.random_field(mm=20, nm=17, hours=1, dx=2000.0, pm=pm, om=om)
    o = run_oracle(oracle_mod, case, 32, max_substeps=2)
    ref = o.get("e")
    for groups in (2,) if pm in (8, 12) else (2, 4):
        run_gpu(U, case, max_substeps=2, groups=groups)
        F, u = U.get_state()
        U.umwm_finalize()
        l2, p999, _ = spec_stats(F, ref)
        assert l2 < 2e-5 and p999 < 1e-3, (groups, l2, p999)
        assert np.abs(u - o.get("ustar")).max() <= 1e-3 * np.abs(o.get("ustar")).max()


@pytest.mark.parametrize("wet", [1, 31, 32, 33, 63, 64, 65, 129])
def test_wet_counts_vs_oracle(lib_built, oracle_mod, wet):
    """Blocks and tiles with a few points, all points and one point."""
    U = lib_built
    case = _case(wet)
    run_gpu(U, case, max_substeps=2)
    F, u = U.get_state()
    U.umwm_finalize()
    o = run_oracle(oracle_mod, case, 32, max_substeps=2)
    l2, p999, _ = spec_stats(F, o.get("e"))
    assert F.shape[0] == wet and l2 < 2e-5 and p999 < 1e-3, (l2, p999)


@pytest.mark.parametrize("option,values", [("direction_groups", (2, 4)), ("integ_groups", (2, 4)),
                                           ("advect_groups", (2, 4)), ("minb_advect", (3, 4, 5)),
                                           ("minb_integ", (3, 4, 5)), ("phys_tma", (0, 1)), ("pf_advect", (0, 3))])
@pytest.mark.parametrize("ice", [False, True])
def test_split_is_bit_identical(lib_built, option, values, ice):
    """How a block's levels are split over warps, and how far ahead its rows
    are fetched, changes no result: 6 substeps with land, currents and (ice)
    points above and below the ice thresholds."""
    from umwm_gb300 import configs

    U = lib_built
    kw = {"fice0": 0.5} if ice else {}
    case = configs.random_field(mm=40, nm=36, hours=1, dx=2000.0, **kw)
    out = []
    for v in values:
        U.clear_inputs()
        case.stage(U)
        U.umwm_initialize(nml_text=case.nml)
        U.set_option("direction_groups", 2)
        U.set_option(option, v)
        U.set_option("max_substeps", 6)
        U.umwm_run(case.start, case.stop)
        out.append((U.get_state(), U.get_field("taux_form"), U.get_field("physics_time_step")))
        U.umwm_finalize()
    for o in out[1:]:
        np.testing.assert_array_equal(o[0][0], out[0][0][0])
        np.testing.assert_array_equal(o[0][1], out[0][0][1])
        np.testing.assert_array_equal(o[1], out[0][1])
        np.testing.assert_array_equal(o[2], out[0][2])


def test_set_state_refreshes_the_mss_prefix(lib_built):
    """A state handed over between runs gives what the same state gives when
    it is read back from the model itself (the prefix of the dissipation's
    mean-square slope is formed again from it)."""
    from umwm_gb300 import configs

    U = lib_built
    case = configs.random_field(mm=40, nm=36, hours=1, dx=2000.0)

    def run(swap):
        U.clear_inputs()
        case.stage(U)
        U.umwm_initialize(nml_text=case.nml)
        U.set_option("max_substeps", 4)
        U.umwm_run(case.start, case.stop)
        if swap:
            F, u = U.get_state()
            U.set_state(3.0 * F, u)  # another state, and back
            U.set_state(F, u)
        U.set_option("max_substeps", 8)
        U.umwm_run(case.start, case.stop)
        F, u = U.get_state()
        U.umwm_finalize()
        return F, u

    F0, u0 = run(False)
    F1, u1 = run(True)
    # the propagation's prefix and k_mss add a level's 36 directions in
    # different orders: a few ulp of the prefix, times (1 + mss_fac chi)^2
    assert np.abs(u1 - u0).max() <= 1e-5 * np.abs(u0).max()
    l2, p999, _ = spec_stats(F1, F0)
    assert l2 < 2e-6 and p999 < 1e-4, (l2, p999)


@pytest.mark.parametrize("pm,om,kw", [(36, 37, {}), (36, 37, {"fice0": 0.5}), (8, 21, {}), (24, 30, {"fice0": 0.4}),
                                      (48, 9, {})])
def test_own_state_set_again_is_neutral(lib_built, pm, om, kw):
    """A run that hands its own state back (another one in between) and goes on
    gives the bits of the run that was never interrupted: the mss prefix and
    the ice's level sums come from the spectrum alone, whoever formed them."""
    from umwm_gb300 import configs

    U = lib_built
    case = configs.random_field(mm=40, nm=36, hours=1, dx=2000.0, pm=pm, om=om, **kw)

    def run(swap):
        U.clear_inputs()
        case.stage(U)
        U.umwm_initialize(nml_text=case.nml)
        U.set_option("max_substeps", 4)
        U.umwm_run(case.start, case.stop)
        if swap:
            F, u = U.get_state()
            U.set_state(3.0 * F, u)
            U.set_state(F, u)
        U.set_option("max_substeps", 8)
        U.umwm_run(case.start, case.stop)
        out = U.get_state() + (U.get_screen(), U.get_field("physics_time_step"))
        U.umwm_finalize()
        return out

    for a, b in zip(run(True), run(False)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("pm,om,groups", [(8, 37, 2), (12, 20, 2), (16, 33, 2), (16, 33, 4), (24, 9, 4), (32, 25, 2), (32, 25, 4),
                                          (48, 37, 2)])
def test_curvilinear_direction_counts_vs_oracle(lib_built, oracle_mod, pm, om, groups):
    """The propagation on a longitude-latitude grid (all four neighbours read,
    the directions turned) with rings of two and of three slots; the tolerances
    of the plain grid's test above."""
    from umwm_gb300 import configs

    U = lib_built
    case = configs.random_field(mm=20, nm=17, hours=1, dx=2000.0, pm=pm, om=om, gridFromFile=True)
    case.gridtopo["lon"], case.gridtopo["lat"] = lonlat_grid(20, 17)
    run_gpu(U, case, max_substeps=2, groups=groups)
    F, u = U.get_state()
    U.umwm_finalize()
    o = run_oracle(oracle_mod, case, 32, max_substeps=2)
    l2, p999, _ = spec_stats(F, o.get("e"))
    assert l2 < 2e-5 and p999 < 1e-3, (l2, p999)
    assert np.abs(u - o.get("ustar")).max() <= 1e-3 * np.abs(o.get("ustar")).max()
