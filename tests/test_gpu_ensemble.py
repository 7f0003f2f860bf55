"""Ensemble (batched) form: members of different sizes advanced as one model.

Each member of an ensemble must give exactly what it gives when run alone:
the kernels are the same, every per-point quantity depends only on the
member's own points, and the only cross-point operations (the dts minimum,
the rotation-rate maximum) are order-independent min/max per member.  So the
comparison is bit-exact.  One member is also checked against the oracle.
"""
import numpy as np
import pytest

from helpers import run_oracle, spec_stats

pytestmark = pytest.mark.gpu


def _members():
    from umwm_gb300 import configs

    return [configs.hurricane(mm=40, nm=36, hours=1, dx=4000.0, dtg=600, seed=3),
            configs.hurricane(mm=56, nm=48, hours=1, dx=3000.0, dtg=600, seed=5),
            configs.hurricane(mm=30, nm=44, hours=1, dx=5000.0, dtg=600, seed=7)]


def _run_alone(U, case):
    U.clear_inputs()
    case.stage(U)
    U.umwm_initialize(nml_text=case.nml)
    U.set_option("max_substeps", -1)
    U.umwm_run(case.start, case.stop)
    F, u = U.get_state()
    out = {"F": F, "ust": u, "ht": U.get_field("ht"), "taux": U.get_field("taux"),
           "screen": U.get_screen()}
    U.umwm_finalize()
    return out


def test_ensemble_members_match_single_runs(lib_built):
    U = lib_built
    members = _members()
    alone = [_run_alone(U, c) for c in members]
    U.clear_inputs()
    for c in members:
        c.stage(U)
        U.ensemble_add(c.nml)
    U.ensemble_initialize()
    assert U.get_field_i("members") == len(members)
    U.umwm_run(members[0].start, members[0].stop)
    for m, ref in enumerate(alone):
        U.select_member(m)
        F, u = U.get_state()
        np.testing.assert_array_equal(F, ref["F"])
        np.testing.assert_array_equal(u, ref["ust"])
        np.testing.assert_array_equal(U.get_field("ht"), ref["ht"])
        np.testing.assert_array_equal(U.get_field("taux"), ref["taux"])
        np.testing.assert_array_equal(U.get_screen(), ref["screen"])
    U.umwm_finalize()


def test_ensemble_member_vs_oracle(lib_built, oracle_mod):
    U = lib_built
    members = _members()
    U.clear_inputs()
    for c in members:
        c.stage(U)
        U.ensemble_add(c.nml)
    U.ensemble_initialize()
    U.set_option("max_substeps", 6)
    U.umwm_run(members[0].start, members[0].stop)
    U.select_member(1)
    o = run_oracle(oracle_mod, members[1], 32, max_substeps=6)
    l2, p999, mx = spec_stats(U.get_state()[0], o.get("e"))
    assert l2 < 1e-4 and p999 < 1e-3, (l2, p999, mx)
    U.umwm_finalize()


@pytest.mark.parametrize("loop", ["host", "persistent"])
def test_members_match_their_single_runs_across_the_size_rule(lib_built, loop):
    """A small domain alone and beside a large one (31 k points): initialize
    takes other direction constants for the two models; with the ensemble's
    choice, set before the run or in its middle, the small domain alone gives the
    member's bits."""
    from umwm_gb300 import configs

    U = lib_built
    small = configs.random_field(mm=40, nm=36, hours=1, dx=2000.0, seed=5)
    large = configs.fetch_limited(mm=180, nm=178, hours=1, dx=2000.0, winds=True, currents=True)
    zero = np.zeros((180, 178), np.float32)
    for t in small.forcing:
        large.forcing[t] = {"uw": zero + 10, "vw": zero + 3, "uc": zero + 0.2, "vc": zero}

    def run(n=6):
        U.set_option("persistent", 1 if loop == "persistent" else 0)
        U.set_option("max_substeps", n)
        U.umwm_run(small.start, small.stop)

    def state():
        F, u = U.get_state()
        return F, u, U.get_field("taux"), U.get_field("physics_time_step"), U.get_screen()

    U.clear_inputs()
    for c in (small, large):
        c.stage(U)
        U.ensemble_add(c.nml)
    U.ensemble_initialize()
    choice = U.stat("direction_constants")
    run(3)
    middle = [(U.select_member(m), U.get_state())[1] for m in (0, 1)]
    run()
    batch = [(U.select_member(m), state())[1] for m in (0, 1)]
    U.umwm_finalize()
    for m, c in enumerate((small, large)):
        U.clear_inputs()
        c.stage(U)
        U.umwm_initialize(nml_text=c.nml)
        assert U.stat("direction_constants") == (choice if m else 6 - choice)  # 2 and 4
        U.set_option("direction_constants", choice)
        run(3)  # (a run that stops starts its interval again)
        run()
        for a, b in zip(state(), batch[m]):
            np.testing.assert_array_equal(a, b)
        U.umwm_finalize()
    # the option between two runs: the prefix of the mean-square slope follows
    U.clear_inputs()
    small.stage(U)
    U.umwm_initialize(nml_text=small.nml)
    U.set_option("direction_constants", choice)
    run(3)
    U.set_option("direction_constants", 6 - choice)
    U.set_state(*middle[0])
    U.set_option("direction_constants", choice)
    run()
    np.testing.assert_array_equal(U.get_state()[0], batch[0][0])
    U.umwm_finalize()


def test_direction_constants_option(lib_built):
    from umwm_gb300 import configs

    U = lib_built
    case = configs.fetch_limited(mm=14, nm=11, hours=1, dx=3000.0, xpl=2, ypl=2, pm=12)
    U.clear_inputs()
    case.stage(U)
    U.umwm_initialize(nml_text=case.nml)
    assert U.stat("direction_constants") == 2
    U.set_option("direction_constants", 2)
    for bad in (3, 4):  # no such construction; none from quarter turns at 12 directions
        with pytest.raises(U.UmwmError):
            U.set_option("direction_constants", bad)
    U.umwm_finalize()
