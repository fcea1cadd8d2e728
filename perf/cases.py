"""The work that is timed: whole runs of the transport engine through its public entry points.

Each case is one scan (or one burst of served scan jobs) of a scene this package defines, run through
the call a program makes: Engine.run (host arrays), Engine.run_device or Engine.run_noalloc (arrays on
the GPU) and the job server.  Outputs are the tallies and the event totals, which are whole numbers and
depend only on the scene, the pixels and the random-stream keys.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from cudamonsel_b200 import capi, data, scenes, serving

PREC = {"fp32": capi.PREC_FP32, "fp64": capi.PREC_FP64}


def listed():
    return [
        # One landing point at the lowest count a user asks for: the setting-up of a measurement.  Launches,
        # copies and the longest electron lineage are all there is.
        dict(name="point_si_fp32", kind="scan", scene="halfspace", prec="fp32", entry="host", side_x=1, side_y=1,
             nprim=100, energy_eV=1000.0, beam_nm=0.0),
        # The validation run: a pencil beam on flat silicon in the plain form.
        dict(name="point_si_fp64", kind="scan", scene="halfspace", prec="fp64", entry="host", side_x=1, side_y=1,
             nprim=10000, energy_eV=1000.0, beam_nm=0.0),
        # A quick look at a line profile: few pixels, few trajectories each, host arrays.
        dict(name="quick_lines_fp32", kind="scan", scene="lines", prec="fp32", entry="host", side_x=33, side_y=1,
             nprim=100, energy_eV=500.0, beam_nm=1.0),
        # The line scan of a critical-dimension measurement at its full size, arrays resident on the GPU.
        dict(name="linescan_fp32", kind="scan", scene="lines", prec="fp32", entry="device", side_x=256, side_y=1,
             nprim=2000, energy_eV=500.0, beam_nm=1.0),
        # The same scan in the plain form, as its reference, at a quarter of the trajectories.
        dict(name="linescan_fp64", kind="scan", scene="lines", prec="fp64", entry="device", side_x=256, side_y=1,
             nprim=500, energy_eV=500.0, beam_nm=1.0),
        # An image of rough lines (385 regions), beam energy by row: a quarter-side tile of the batched image.
        dict(name="image_rough_fp32", kind="image", prec="fp32", side=64, nprim=300),
        # A smaller image tile in the plain form.
        dict(name="image_rough_fp64", kind="image", prec="fp64", side=37, nprim=101),
        # Deep penetration: 10 keV over a field of 256 blocks and cylinders.
        dict(name="deep_fp32", kind="scan", scene="deep", prec="fp32", entry="device", side_x=61, side_y=61,
             nprim=50, energy_eV=10000.0, beam_nm=1.0),
        # Rounded lines and cylinders (union trees), with the angle histograms.
        dict(name="rounded_fp32", kind="scan", scene="features", prec="fp32", entry="angles", side_x=101, side_y=1,
             nprim=1000, energy_eV=800.0, beam_nm=2.0),
        # Silicon with its phonon mechanism at a high beam energy.
        dict(name="phonon_fp32", kind="scan", scene="phonon", prec="fp32", entry="host", side_x=17, side_y=1,
             nprim=1500, energy_eV=3000.0, beam_nm=1.0),
        # A caller that owns the device memory: the fixed-scratch entry.
        dict(name="noalloc_fp32", kind="scan", scene="lines", prec="fp32", entry="noalloc", side_x=64, side_y=1,
             nprim=100, energy_eV=500.0, beam_nm=1.0),
        # A burst of scan jobs of different samples sent to the job server at once.
        dict(name="served_fp32", kind="served", prec="fp32", jobs=8, scale=0.04),
    ]


def _log(rng, lo, hi):
    return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "scan", "image", "served"])
    prec = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "served":
        return dict(kind="served", prec="fp32", jobs=rng.randint(2, 8), scale=round(rng.uniform(0.01, 0.03), 4))
    if kind == "image":
        return dict(kind="image", prec=prec, side=_log(rng, 9, 64 if prec == "fp32" else 37),
                    nprim=_log(rng, 20, 250 if prec == "fp32" else 100))
    scene = rng.choice(["halfspace", "lines", "lines", "features", "phonon", "pmma", "deep"])
    energy = {"lines": (300, 1000), "deep": (3000, 10000), "halfspace": (200, 5000)}.get(scene, (300, 3000))
    e = float(_log(rng, *energy))
    entry = rng.choice(["host", "device", "angles", "noalloc"])
    x, y = _log(rng, 1, 400), 1
    if scene == "deep":
        y = x = _log(rng, 4, 48)
    # the trajectories that a drawn scan may have at its beam energy
    top = 1.2e5 * (1000.0 / e) ** 0.8 * (1.0 if prec == "fp32" else 0.4)
    if entry == "noalloc":
        top = min(top, 1.5e4 * 500.0 / e)  # the fixed scratch holds a small pool of secondaries
    n = max(1, min(_log(rng, 20, 5000), int(top / (x * y))))
    return dict(kind="scan", scene=scene, prec=prec, entry=entry, side_x=x, side_y=y, nprim=n, energy_eV=e,
                beam_nm=float(rng.choice([0.0, 1.0, 2.5])))


# the scattering tables and elastic data are parsed once, as a program that builds several scenes does
@functools.lru_cache(maxsize=None)
def _table(path):
    return data.read_nu_table(path)


class _Backend(scenes.EngineBackend):
    def table(self, path):
        return self.e.table(*_table(path))


def _build(scene, engine):
    return scenes.replay(scene.spec, _Backend(engine))[scene.chamber.idx]


def _scene(name, seed):
    """The scene, and the height (m) the beam starts above the substrate."""
    if name == "halfspace":
        return scenes.halfspace(), 20e-9
    if name == "phonon":
        return scenes.halfspace(phonon=True), 20e-9
    if name == "pmma":
        return scenes.halfspace(material="pmma"), 20e-9
    if name == "lines":
        return scenes.lines(), 120e-9
    if name == "features":
        return scenes.features(), 120e-9
    sc, top = scenes.deep_features(seed=seed)
    return sc, top + 20e-9


def _pixels(case, seed):
    """Landing points (m), beam energies (J), primaries and histogram bins of a scan."""
    nx, ny = case["side_x"], case["side_y"]
    step = 16e-9 if case["scene"] == "deep" else 1.5e-9
    x = (np.arange(nx) - (nx - 1) / 2.0) * step
    y = (np.arange(ny) - (ny - 1) / 2.0) * step
    gx, gy = np.meshgrid(x, y)
    centers = np.stack([gx.ravel(), gy.ravel(), np.zeros(nx * ny)], axis=1)
    n = nx * ny
    return (centers, np.full(n, scenes.eV(case["energy_eV"])), np.full(n, case["nprim"], dtype=np.int32),
            np.full(n, min(1024, max(1, int(case["energy_eV"] / 10.0))), dtype=np.int32))


def _keys(n, seed):
    return np.random.default_rng(seed).integers(1, 2**63, n, dtype=np.uint64)


def prepare(case, seed):
    prec = PREC[case["prec"]]
    if case["kind"] == "served":
        return _prepare_served(case, seed, prec)
    eng = capi.Engine(0)
    if case["kind"] == "image":
        chamber = _build(scenes.rough_lines(seed=seed), eng)
        centers, energy, nprim, nbins = scenes.rough_image(seed=seed, side=case["side"], mean_nprim=case["nprim"])
        entry, beam = "host", 1e-9
    else:
        sc, z = _scene(case["scene"], seed)
        chamber = _build(sc, eng)
        centers, energy, nprim, nbins = _pixels(case, seed)
        centers[:, 2] = -z
        entry, beam = case["entry"], case["beam_nm"] * 1e-9
    keys = _keys(len(centers), seed)
    state = dict(entry=entry, engine=eng, prec=prec, chamber=chamber, centers=centers, energy=energy, nprim=nprim,
                 nbins=nbins, keys=keys, beam=beam)
    if entry in ("device", "noalloc"):
        dev = torch.device("cuda", 0)
        stride = int(nbins.max()) + 2
        t = [torch.from_numpy(centers.ravel()).to(dev), torch.from_numpy(energy).to(dev),
             torch.from_numpy(nprim).to(dev), torch.from_numpy(nbins).to(dev),
             torch.from_numpy(keys.astype(np.int64)).to(dev)]
        back = torch.zeros((len(centers), stride), dtype=torch.int32, device=dev)
        fwd = torch.zeros_like(back)

        def at(x, kind):
            return C.cast(C.c_void_p(x.data_ptr()), C.POINTER(kind))

        desc = capi.RunDesc(chamber, prec, len(centers), beam, at(t[0], C.c_double), at(t[1], C.c_double),
                            at(t[2], C.c_int), at(t[3], C.c_int), seed, stride, 0, 0, at(t[4], C.c_uint64), 0)
        state.update(arrays=t, back=back, fwd=fwd, desc=desc)
        if entry == "noalloc":  # this entry wants the scene on the device beforehand
            eng.eval_freepath(0, np.array([[scenes.eV(100.0), 0.5]]), prec)
    torch.cuda.synchronize()
    return state


def _prepare_served(case, seed, prec):
    holder = capi.Engine(0)
    jobs = serving.make_jobs(case["jobs"], seed=seed, scale=case["scale"])
    for k, job in enumerate(jobs):
        # like sizes for every seed: the stream's mix of images and line scans at fixed sizes, its beam
        # energies in fixed steps over their range
        n = max(4, int(3000 * case["scale"]))
        x = (np.arange(n) - (n - 1) / 2.0) * 1e-9
        job["centers"] = np.stack([x, np.zeros(n), np.full(n, -220e-9)], axis=1)
        e = 300.0 * (10.0 ** (k / max(1, case["jobs"] - 1)))
        job.update(energy=scenes.eV(e), nbins=max(1, int(e / 10.0)), nprim=max(1, int(500 * case["scale"] * 4)),
                   keys=_keys(n, seed + 7 * k))
    server = capi.Server(0, case["jobs"], 16.0)
    return dict(entry="served", server=server, holder=holder, jobs=jobs, prec=prec)


def _totals(st):
    return [int(st.primaries), int(st.steps), int(st.scatter_events), int(st.barrier_events), int(st.escapes),
            int(st.secondaries)]


def run(state):
    if state["entry"] == "served":
        return _run_served(state)
    e = state["engine"]
    if state["entry"] in ("device", "noalloc"):
        call = e.run_device if state["entry"] == "device" else e.run_noalloc
        st = call(state["desc"], state["back"].data_ptr(), state["fwd"].data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
        return [state["back"], state["fwd"], _totals(st)]
    out = e.run(state["chamber"], state["centers"], state["energy"], state["nprim"], state["nbins"], state["beam"], 0,
                state["prec"], pixel_keys=state["keys"], angles=state["entry"] == "angles")
    res = [out[0], out[1], _totals(out[2])]
    if state["entry"] == "angles":
        res += [out[3]["elevation"], out[3]["azimuth"]]
    return res


def _run_served(state):
    server, holder = state["server"], state["holder"]
    ids = []
    for job in state["jobs"]:
        holder.reset()
        chamber = scenes.replay(job["spec"], _Backend(holder))[job["chamber"].idx]
        ids.append(server.submit(holder, chamber, job["centers"], job["energy"], job["nprim"], job["nbins"], 1e-9, 0,
                                 state["prec"], pixel_keys=job["keys"]))
    for j in ids:
        server.wait(j)
    out = []
    for j in ids:
        back, fwd, st = server.result(j)
        out += [back, fwd, [int(st.primaries), int(st.steps)]]
    return out


def work(case):
    """Input and output bytes, and about 400 operations per electron-step (cross sections, free path, boundary
    search, event); a primary and its secondaries take about 380 steps at 1 keV and 2100 at 10 keV."""
    if case["kind"] == "served":
        n, jobs = max(4, int(3000 * case["scale"])), case["jobs"]
        nprim = max(1, int(500 * case["scale"] * 4))
        scans = [(n, nprim, 300.0 * (10.0 ** (k / max(1, jobs - 1)))) for k in range(jobs)]
    elif case["kind"] == "image":
        scans = [(case["side"] ** 2, case["nprim"], 600.0)]
    else:
        scans = [(case["side_x"] * case["side_y"], case["nprim"], case["energy_eV"])]
    size = steps = 0.0
    angles = (182 + 362) * 4 if case.get("entry") == "angles" else 0
    for npix, nprim, e in scans:
        size += npix * (48 + 2 * 4 * (e / 10.0 + 2) + angles)
        steps += npix * nprim * 380.0 * (e / 1000.0) ** 0.75
    return {"bytes": size, "flops": 400.0 * steps}


def exact(case, seed):
    return None  # every output is a count
