"""A substep's chain of kernels on both sides of the lines at which its launches
change (dts formed by the pre-pass's last block or by a launch of its own; the
next kernel started early or not): the host-driven loop, the graph loop and the
persistent kernel give the same bits, state, time step and screen lines, with
and without sea ice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 171 points: one block per SM at most; 8 k: the split for small models;
# 17.5 k (548 blocks): dts in the pre-pass; 21.8 k (682): a launch of its own
@pytest.mark.parametrize("mm,nm,kw", [(21, 11, {}), (92, 92, {}), (150, 120, {}), (160, 140, {}),
                                      (21, 11, {"fice0": 0.5}), (150, 120, {"fice0": 0.5}), (160, 140, {"fice0": 0.5})])
def test_loops_agree(lib_built, mm, nm, kw):
    from umwm_gb300 import configs

    U = lib_built
    got = []
    for opt in ("host", "graph", "persistent"):
        case = configs.fetch_limited(mm=mm, nm=nm, hours=1, dx=3000.0, depth=60.0, dtg=600, xpl=2, ypl=2, **kw)
        U.clear_inputs()
        case.stage(U)
        U.umwm_initialize(nml_text=case.nml)
        U.set_option("use_graph", 1 if opt == "graph" else 0)
        U.set_option("persistent", 1 if opt == "persistent" else 0)
        U.set_option("max_substeps", 7)
        U.umwm_run(case.start, case.stop)
        F, u = U.get_state()
        got.append((F, u, U.get_field("dts"), U.get_screen(), U.dims()["substeps"]))
        U.umwm_finalize()
    for g in got[1:]:
        assert g[4] == got[0][4] and g[2] == got[0][2]
        assert np.array_equal(g[3], got[0][3])
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1])


# members' grids: 8 and 132 blocks of 32 points (the split for small models);
# 338 to 604: dts in the pre-pass; 626 and 818: a launch of its own
@pytest.mark.parametrize("grids", [[(20, 17)], [(150, 120)], [(165, 150)], [(40, 36), (60, 48), (30, 44)],
                                   [(100, 60), (90, 90)], [(100, 90), (100, 110)], [(120, 110), (60, 48), (110, 90)],
                                   [(160, 120), (120, 120)]])
def test_loops_agree_with_currents_and_members(lib_built, grids):
    """As above with land and currents (the rotation and the current flag of
    every substep), and with members whose substeps differ in number."""
    from umwm_gb300 import configs

    U = lib_built
    cases = [configs.random_field(mm=mm, nm=nm, hours=1, dx=2000.0 + 300.0 * k, dtg=600, seed=2 + k)
             for k, (mm, nm) in enumerate(grids)]
    stop = configs._time_str(cases[0].start, 600)
    for c in cases:
        c.forcing[stop] = c.forcing[c.start]
    got = []
    for opt in ("host", "graph", "persistent"):
        U.clear_inputs()
        if len(cases) == 1:
            cases[0].stage(U)
            U.umwm_initialize(nml_text=cases[0].nml)
        else:
            for c in cases:
                c.stage(U)
                U.ensemble_add(c.nml)
            U.ensemble_initialize()
        U.set_option("use_graph", 1 if opt == "graph" else 0)
        U.set_option("persistent", 1 if opt == "persistent" else 0)
        U.umwm_run(cases[0].start, stop)
        out = []
        for m in range(len(cases)):
            U.select_member(m)
            out += [*U.get_state(), U.get_screen(), np.float32(U.get_field("dtr")), U.get_field("taux")]
        got.append(out)
        U.umwm_finalize()
    for g in got[1:]:
        for a, b in zip(g, got[0]):
            np.testing.assert_array_equal(a, b)
