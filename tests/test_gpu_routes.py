"""The kernels' short routes at the ends of their ranges, through the public entry points."""
import numpy as np
import pytest

FP64, FP32 = 0, 1
pytestmark = pytest.mark.gpu


def cubic(xs, f, x):
    """The cubic through four nodes at x, in 64 bits."""
    return sum(f[i] * np.prod([(x - xs[j]) / (xs[i] - xs[j]) for j in range(4) if j != i]) for i in range(4))


@pytest.mark.parametrize("prec", [FP64, FP32], ids=["fp64", "fp32"])
def test_tables_beyond_an_axis_that_ends_below_zero(prec):
    """2-D and 3-D tables whose first axis runs from -20 to -5.57: an argument above its last node is
    extrapolated from the last four nodes.  The values are random, so another window is off by about one.
    FP64: 15 (the weights' sum one interval beyond) times rounding, with room.  FP32: an abscissa's rounding of
    1e-6 in an interval of 0.37, times the weights' slope of about 30, is 1e-4, with room."""
    from cudamonsel_b200 import capi
    rng = np.random.default_rng(3)
    a = -20.0 + 0.37 * np.arange(40)
    b, c = np.linspace(0.0, 1.0, 9), np.linspace(0.0, 1.0, 7)
    v2, v3 = rng.random((40, 9)), rng.random((40, 9, 7))
    e = capi.Engine(0)
    e.set_options(1)  # 3-D tables with the window's own abscissae in every step
    t2, t3 = e.table(2, [40, 9], [a, b], v2), e.table(3, [40, 9, 7], [a, b, c], v3)
    xs = a[-1] + 0.37 * np.array([0.001, 0.25, 0.5, 1.0])
    x = np.stack([xs, np.full(4, b[4]), np.full(4, c[3])], axis=1)
    got2, got3 = e.eval_table(t2, x, 3, prec), e.eval_table(t3, x, 3, prec)
    first = e.eval_locate(t2, x, 3, prec)[:, 0]
    e.close()
    assert (first == 36).all()
    tol = 1e-11 if prec == FP64 else 2e-3
    for k in range(4):
        assert abs(got2[k] - cubic(a[-4:], v2[-4:, 4], xs[k])) < tol
        assert abs(got3[k] - cubic(a[-4:], v3[-4:, 4, 3], xs[k])) < tol


@pytest.mark.parametrize("prec", [FP64, FP32], ids=["fp64", "fp32"])
def test_vacuum_steps_take_one_iteration(prec):
    """A primary that starts inside a vacuum box and flies through a stack of them takes one step per wall, and
    each step one iteration of the queue kernels: as many iterations whether or not the boxes have children
    (a region with children takes the full flight), one more than steps for the start.  The resident-steps
    kernel gives the same tallies."""
    from cudamonsel_b200 import capi, scenes

    def box(s, c, h):
        n, p = [], []
        for a in range(3):
            for sg in (-1.0, 1.0):
                n += [sg * (a == k) for k in range(3)]
                p += [c[k] + sg * h[k] * (a == k) for k in range(3)]
        return s.planes(n, p)

    def run(children, options):
        s = scenes.SceneSpec()
        vac = scenes.vacuum(s)
        ch = s.region(None, vac, s.sphere([0.0, 0.0, 0.0], 0.1))
        for k in range(8):
            r = s.region(ch, vac, box(s, [0.0, 0.0, 40e-9 * k], [50e-9, 50e-9, 10e-9]))
            if children:  # a child that the beam misses
                s.region(r, vac, box(s, [45e-9, 45e-9, 40e-9 * k], [1e-9, 1e-9, 1e-9]))
        e = capi.Engine(0)
        h = scenes.replay(s, scenes.EngineBackend(e))
        e.set_options(options)
        b, f, st = e.run(h[ch.idx], np.array([[0.0, 0.0, 1e-9]]), scenes.eV(500.0), 1, 50, 0.0, 3, precision=prec)
        e.close()
        return b, f, st

    b0, f0, s0 = run(False, capi.OPT_QUEUE_STEPS)
    b1, f1, s1 = run(True, capi.OPT_QUEUE_STEPS)
    b2, f2, s2 = run(False, 0)
    print("steps %d, iterations %d, with children %d" % (s0.steps, s0.iterations, s1.iterations))
    assert s0.steps == s1.steps == s2.steps and s0.escapes == 1 and s0.steps == 16
    assert s0.iterations == s1.iterations == s0.steps + 1
    assert np.array_equal(b0, b1) and np.array_equal(f0, f1) and np.array_equal(b0, b2) and np.array_equal(f0, f2)


@pytest.mark.parametrize("prec", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("scene,below", [("features", 131072), ("halfspace", 262144)])
def test_autotuner_starts_from_the_scene_s_own_settings(scene, below, prec):
    """cm_autotune starts from the settings an untuned run of the scene would use; a scene with shape trees
    enters the tail at half as many electrons.  Under CM_OPT_QUEUE_STEPS the tail settings change nothing, so
    the tuner keeps that start unless two runs of one kind differ by its 1 % (six tries)."""
    from cudamonsel_b200 import capi, scenes
    sc = scenes.features() if scene == "features" else scenes.halfspace()
    got = []
    for _ in range(6):
        e = capi.Engine(0)
        h = scenes.build_engine(sc, e)
        e.set_options(capi.OPT_QUEUE_STEPS | sc.spec.options)
        t = e.autotune(h["chamber"], scenes.linescan_pixels(64), scenes.eV(500.0), 300 if prec == FP32 else 100, 50,
                       1e-9, 9, precision=prec)
        e.close()
        got.append((t.tail_below, round(t.ms, 2)))
        if t.tail_below == below:
            break
    print(scene, got)
    assert got[-1][0] == below


@pytest.mark.parametrize("profile", [0, 1])
def test_launch_counts_hold_both_flights(profile):
    """An iteration of the queue kernels launches the fast and the full flight, three event kernels and the
    refill; a tail iteration the resident-steps kernel and the refill."""
    from cudamonsel_b200 import capi, scenes
    e = capi.Engine(0)
    h = scenes.build_engine(scenes.lines(), e)
    _, _, st = e.run(h["chamber"], scenes.linescan_pixels(64), scenes.eV(500.0), 1000, 50, 1e-9, seed=9,
                     precision=FP32, profile=profile)
    e.close()
    n = list(st.kernel_launches)
    print(n, st.step_launches)
    assert n[1] > 0 and n[1] == n[2] == n[3] and n[0] == 2 * n[1]
    assert n[4] == n[1] + st.step_launches and n[5] == 0


def test_steps_that_stay_in_vacuum_take_one_iteration_each():
    """An electron that enters a vacuum region without a far end flies on, staying in the region, to the
    reference's limit of 10^6 steps: the resident-steps kernel takes it through one step per iteration (64 a
    launch), as no such step has an event."""
    from cudamonsel_b200 import capi, scenes
    s = scenes.SceneSpec()
    vac = scenes.vacuum(s)
    ch = s.region(None, vac, s.sphere([0.0, 0.0, 0.0], 0.1))
    s.region(ch, vac, s.planes([0.0, 0.0, -1.0], [0.0, 0.0, 0.0]))
    e = capi.Engine(0)
    h = scenes.replay(s, scenes.EngineBackend(e))
    _, _, st = e.run(h[ch.idx], np.array([[0.0, 0.0, -20e-9]]), scenes.eV(500.0), 1, 50, 0.0, 3, precision=FP32)
    e.close()
    print("steps %d, launches %d, %.0f ms" % (st.steps, st.iterations, st.device_ms))
    assert st.ended_step_limit == 1 and st.escapes == 0 and 1000000 < st.steps < 1000010
    assert st.iterations < st.steps / 64 + 8
