"""cm_run_noalloc when its fixed secondary pool overflows: the resident-steps run is repeated with the queue
kernels, and the statistics say so.  Collected last, like the other tests of this entry point."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64, FP32 = 0, 1


@pytest.mark.parametrize("prec", [FP32, FP64], ids=["fp32", "fp64"])
def test_noalloc_overflow_is_repeated_and_reported(prec):
    """9000 primaries of 40 keV on flat Si (twice the tables' domain) create more secondaries than the scratch holds with either set of
    kernels: CM_EOVERFLOW, with both runs in the statistics (one restart, launches of both sets).  A scan that
    fits follows on the same context, runs once and gives cm_run_device's tallies."""
    import torch
    from cudamonsel_b200 import capi, scenes
    dev = torch.device("cuda", 0)
    e = capi.Engine(0)
    h = scenes.build_engine(scenes.halfspace(), e)

    def at(x, kind):
        return C.cast(C.c_void_p(x.data_ptr()), C.POINTER(kind))

    def call(entry, e_eV, nprim):
        npix, nb = 10, min(1000, int(e_eV / 10))
        t = [torch.tensor(np.tile([0.0, 0.0, -20e-9], npix), dtype=torch.float64, device=dev),
             torch.full((npix,), scenes.eV(e_eV), dtype=torch.float64, device=dev),
             torch.full((npix,), nprim, dtype=torch.int32, device=dev),
             torch.full((npix,), nb, dtype=torch.int32, device=dev),
             torch.arange(5, 5 + npix, dtype=torch.int64, device=dev)]
        back = torch.zeros((npix, nb + 2), dtype=torch.int32, device=dev)
        fwd = torch.zeros_like(back)
        d = capi.RunDesc(h["chamber"], prec, npix, 0.0, at(t[0], C.c_double), at(t[1], C.c_double), at(t[2], C.c_int),
                         at(t[3], C.c_int), 0, nb + 2, 0, 0, at(t[4], C.c_uint64), 0)
        st = capi.RunStats()
        rc = entry(e.h, C.byref(d), C.c_void_p(back.data_ptr()), C.c_void_p(fwd.data_ptr()), C.byref(st), None)
        torch.cuda.synchronize()
        return rc, st, back.cpu().numpy(), fwd.cpu().numpy()

    rc0, s0, b0, f0 = call(e.L.cm_run_device, 1000.0, 100)
    rc1, s1, _, _ = call(e.L.cm_run_noalloc, 40000.0, 900)
    rc2, s2, b2, f2 = call(e.L.cm_run_noalloc, 1000.0, 100)
    e.close()
    print("overflow: restarts %d, resident-steps launches %d, queue launches %d, %.1f ms" % (
        s1.pool_restarts, s1.step_launches, s1.kernel_launches[1], s1.device_ms))
    assert rc0 == 0 and rc1 == capi.EOVERFLOW and rc2 == 0
    assert s1.pool_restarts == 1 and s1.step_launches > 0 and s1.step_units > 0 and s1.kernel_launches[0] > 0
    assert s1.kernel_launches[4] == s1.step_launches + s1.kernel_launches[1]
    assert s1.kernel_launches[0] == 2 * s1.kernel_launches[1]
    assert s2.pool_restarts == 0 and s2.step_launches > 0 and s2.kernel_launches[0] == 0
    assert s2.steps == s0.steps and np.array_equal(b2, b0) and np.array_equal(f2, f0)
