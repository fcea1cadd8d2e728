"""The resident-steps kernel (electrons in shared memory, many steps per launch) against the queue kernels.

Both use the same per-electron functions and lineage-keyed random streams, so tallies and totals are
identical; the cases are the sizes where the kernel's bookkeeping can go wrong."""
import numpy as np
import pytest

FP64, FP32 = 0, 1
pytestmark = pytest.mark.gpu

# (scene, pixels, primaries per pixel, settings of the run through the resident-steps kernel)
CASES = [
    ("lines", 1, 1, {}),                                          # one electron on the whole GPU
    ("lines", 31, 1, dict(tail_steps=1)),                         # flushed after every iteration
    ("lines", 33, 9, dict(tail_steps=3)),                         # two electrons in some blocks, three in others
    ("features", 7, 40, {}),                                      # shape trees
    ("deep", 5, 3, dict(tail_steps=7)),                           # grids; large cascades in few slots
    ("lines", 48, 100, dict(wave=1024, tail_steps=5)),            # a small wave: few slots, refill and pool at work
    ("halfspace", 3, 5000, dict(wave=4096, pool=1)),              # pool overflow and restart
    ("lines", 512, 500, dict(tail_below=1 << 30)),                # more electrons than slots: taken as slots free up
]


def scene_of(name):
    from cudamonsel_b200 import scenes
    if name == "lines":
        return scenes.lines(), 500.0, 120e-9
    if name == "features":
        return scenes.features(), 800.0, 120e-9
    if name == "deep":
        sc, top = scenes.deep_features(seed=3)
        return sc, 5000.0, top + 20e-9
    return scenes.halfspace(), 1000.0, 20e-9


@pytest.mark.parametrize("prec", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name,npix,nprim,settings", CASES)
def test_resident_steps_match_the_queue_kernels(name, npix, nprim, settings, prec):
    from cudamonsel_b200 import capi, scenes
    if prec == FP64 and npix * nprim > 100000:
        nprim = 100
    sc, e_eV, z = scene_of(name)
    e = capi.Engine(0)
    h = scenes.build_engine(sc, e)
    c = scenes.linescan_pixels(npix, z=-z)
    args = (h["chamber"], c, scenes.eV(e_eV), nprim, int(e_eV / 10), 1e-9, 17)
    e.set_tuning(prec, **settings)
    b1, f1, s1 = e.run(*args, precision=prec)
    e.set_tuning(prec)
    e.set_options(capi.OPT_QUEUE_STEPS | (1 if name == "features" else 0))
    b0, f0, s0 = e.run(*args, precision=prec)
    e.close()
    assert s1.step_launches > 0 and s0.step_launches == 0
    assert s1.primaries == npix * nprim
    assert (s1.steps, s1.scatter_events, s1.barrier_events, s1.escapes, s1.secondaries) == (
        s0.steps, s0.scatter_events, s0.barrier_events, s0.escapes, s0.secondaries)
    assert np.array_equal(b1, b0) and np.array_equal(f1, f0)
