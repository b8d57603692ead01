"""The routes W3SRCE's kernel takes by a rule, against the general ones: on the CPU the tables derived
from the registered ones and the branch-free libm forms (bit for bit), on the GPU the kernel's forms (36,
24 and other numbers of directions, with and without sheltering, numbers of points around the slots
and CTAs) against the host build of the same source, one point at a time."""

import ctypes
import itertools
import re
import subprocess

import numpy as np
import pytest

from conftest import cuda_available
import st4_common as sc

P = ctypes.c_void_p
_igrid = itertools.count(1000)  # a grid is bound to one VA


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    so = tmp_path_factory.mktemp("routes") / "libroutes.so"
    csrc = sc.ROOT / "ww3-gpu_b200" / "csrc"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O2", "-march=x86-64-v3", "-ffp-contract=off",
                    "-fno-math-errno", "-fPIC", "-shared", f"-I{csrc}", "-I/usr/local/cuda/include",
                    str(sc.ROOT / "tests" / "srce_routes.cpp"), str(csrc / "snl1_tables.cpp"), "-o",
                    str(so)], check=True)
    H = ctypes.CDLL(str(so))
    H.hemu_st4_init.argtypes = [P, sc.I, P, sc.I]
    for f in (H.hemu_st4_set_real, H.hemu_st4_set_int):
        f.argtypes = [sc.I, P, sc.I, P, P]
    H.hemu_snl1_init.argtypes = [sc.I, sc.I] + [sc.F] * 10 + [P]
    H.hemu_srce_init.argtypes = [P, sc.I, P, sc.I, P, P, P, P, P]
    H.hemu_srce_batch.argtypes = [sc.I] * 4 + [sc.F, sc.I] + [P] * 9
    H.routes_libm.argtypes = [ctypes.c_long, ctypes.c_ulonglong, P]
    return H


def config(synth, nk, nth, shelter, ln1=0, seed=0):
    st = synth.st4_setup(nk, nth, variant="analytic")
    st["rpar"][st["R"]["TTAUWSHELTER"]] = shelter
    t = synth.st4_tables_own(st)
    return st, t, synth.srce_setup(st, ln1=ln1, seed=seed), synth.dia_config(nk, nth)


def host_setup(H, synth, st, t, sr, dia, regs=None):
    assert H.hemu_st4_init(sc.p(st["rpar"]), st["rpar"].size, sc.p(st["ipar"]), st["ipar"].size) == 0
    for aid, arr, is_int, lb, ext in regs or synth.st4_registrations(st, t):
        arr = np.ascontiguousarray(arr, np.int32 if is_int else np.float32)
        lb, ext = np.asarray(lb, np.int32), np.asarray(ext, np.int32)
        f = H.hemu_st4_set_int if is_int else H.hemu_st4_set_real
        assert f(aid, sc.p(arr), len(ext), sc.p(lb), sc.p(ext)) == 0
    assert H.hemu_st4_commit() == 0
    cfg, sig = dia
    assert H.hemu_snl1_init(cfg["nk"], cfg["nth"], *[cfg[k] for k in sc.NK_ARGS], sc.p(sig)) == 0
    assert H.hemu_srce_init(sc.p(sr["rpar"]), len(sr["rpar"]), sc.p(sr["ipar"]), len(sr["ipar"]),
                            *[sc.p(sr[k]) for k in ("sig", "dden", "ecos", "esin", "mapwn")]) == 0


def same(a, b):
    return {k: int((np.ascontiguousarray(a[k]).view(np.uint32) != np.ascontiguousarray(b[k]).view(np.uint32)).sum())
            for k in a}


@pytest.mark.parametrize("nk,nth", [(25, 24), (13, 7), (12, 10)])
def test_derived_tables_change_no_bit(routes, synth, nk, nth):
    st, t, sr, dia = config(synth, nk, nth, 0.0)
    host_setup(routes, synth, st, t, sr, dia)
    pts = synth.srce_points(5, seed=nk, nk=nk, nth=nth, depth_range=(2.0, 4000.0))
    pts["pin"][0, 2] = 0.0  # a wind along an axis leaves the stress scan's parallel form
    be = sc.hemu_backend(routes)
    assert routes.routes_derived(0) & 7 == 7
    general = be.srce_batch(pts)
    routes.routes_derived(1)
    assert not any(same(general, be.srce_batch(pts)).values())


def test_derived_tables_are_refused_where_they_do_not_apply(routes, synth):
    st, t, sr, dia = config(synth, 12, 10, 0.0)
    for key, at, value, bit in (("cumulw", 7 * 120 + 13, 0.5, 1), ("cumulw", 3, np.inf, 2)):
        t2 = dict(t, cumulw=t["cumulw"].copy())
        t2[key][at] = value
        host_setup(routes, synth, st, t2, sr, dia)
        assert routes.routes_derived(1) & bit == 0
    regs = [list(r) for r in synth.st4_registrations(st, t)]
    regs[6][1] = np.array(regs[6][1], copy=True)
    regs[6][1][25] += np.float32(1e-3)  # ECOS of another row
    host_setup(routes, synth, st, t, sr, dia, regs)
    assert routes.routes_derived(1) & 4 == 0


def test_branch_free_libm_equals_general(routes):
    bad = np.zeros(7, np.int64)
    routes.routes_libm(3_000_000, 88172645463325252, sc.p(bad))
    assert not bad.any(), bad


def test_working_set_layout_depends_on_the_spectral_grid_only(routes, synth):
    """ww_steps_fuse takes grids whose layouts are equal: ST4's options must not show in them."""
    seen = set()
    for shelter, case, stab3 in ((0.0, 1.0, 0), (0.3, 1.0, 0), (0.0, 3.0, 0), (0.0, 1.0, 1)):
        st, t, sr, dia = config(synth, 12, 10, shelter)
        st["rpar"][st["R"]["SSDSC"]] = case
        st["ipar"][6] = stab3
        host_setup(routes, synth, st, t, sr, dia)
        buf = np.zeros(4096, np.uint8)
        seen.add(bytes(buf[:routes.routes_layout(sc.p(buf), buf.size)]))
    assert len(seen) == 1


def test_named_barriers_do_not_ask_for_a_converged_warp():
    """bar.sync and bar.arrive are the .aligned forms: all lanes have to issue them together, which the
    W3SRCE kernels' code before them does not guarantee."""
    csrc = sc.ROOT / "ww3-gpu_b200" / "csrc"
    text = "".join((csrc / f).read_text() for f in ("srce_point.cuh", "st4_srce_kernel.cu"))
    named = re.findall(r'asm volatile\("(bar[a-z.]*) ', text)
    assert sorted(named) == ["barrier.arrive", "barrier.sync"]


def sheltered(st, sr):
    st["rpar"][st["R"]["TTAUWSHELTER"]] = 0.3


def romero(st, sr):
    R = st["R"]
    for k, v in ((0, 3.0), (1, 5e-5), (7, 1.0), (8, 0.05), (10, 1.0), (12, 1.0), (13, 1.0), (14, 1.0),
                 (15, 1.2), (17, 0.5), (18, 1.0)):
        st["rpar"][R["SSDSC"] + k] = v
    st["rpar"][R["SSDSBT"]] = 1e-3


def filipot(st, sr):
    st["rpar"][st["R"]["SSDSC"]] = 2.0


def isotropic_cumulative(st, sr):
    st["rpar"][st["R"]["SSDSC"] + 2] = 0.4


def all_directions(st, sr):
    st["rpar"][st["R"]["SSDSDTH"]] = 180.0


def stab3(st, sr):
    st["ipar"][6] = 1


def ig1(st, sr):
    st["ipar"][7] = 1
    st["rpar"][st["R"]["IGPARS5"]] = 4.0


def tail_level(st, sr):
    st["rpar"][st["R"]["SINTAILPAR"] + 2] = 1.0


def spr4_twice(st, sr):
    st["rpar"][st["R"]["SINTAILPAR"] + 3] = 0.0


def ice(st, sr):
    sr["rpar"][13:17] = [0.5, 0.7, 0.9, 0.3]


@pytest.mark.parametrize("mods", [(), (sheltered,), (romero,), (romero, sheltered), (filipot,),
                                  (isotropic_cumulative,), (all_directions,), (stab3,),
                                  (stab3, sheltered), (ig1,), (tail_level, sheltered)],
                         ids=lambda m: "+".join(f.__name__ for f in m) or "plain")
@pytest.mark.parametrize("nk,nth", [(25, 24), (12, 10)])
def test_terms_equal_the_point_entries_source(routes, synth, nk, nth, mods):
    """W3SIN4, W3SDS4 and W3SPR4 are written twice: as W3SRCE's phases and for ww_sin4, ww_sds4 and
    ww_spr4. Both give the same bits."""
    st, t, sr, dia = config(synth, nk, nth, 0.0)
    for m in mods:
        m(st, sr)
    host_setup(routes, synth, st, synth.st4_tables_own(st), sr, dia)
    routes.routes_derived(1)
    be = sc.hemu_backend(routes)
    routes.hemu_sds4.argtypes = [sc.I] + [P] * 8 + [sc.I, sc.I] + [P] * 4
    routes.hemu_sin4.argtypes = [sc.I] + [P] * 17
    routes.hemu_spr4.argtypes = [sc.I] + [P] * 20
    routes.routes_terms.argtypes = [P] * 4 + [sc.F] * 6 + [P] * 9
    n, ns = 12, nk * nth
    pts = synth.srce_points(n, seed=3, nk=nk, nth=nth, depth_range=(2.0, 4000.0))
    pts["pin"][:, 3] = np.linspace(-6.0, 2.0, n)
    pts["pin"][0, 2] = 0.0
    x, udir = sc.point_inputs(pts), pts["pin"][:, 2].copy()
    sin4 = be.sin4(x["a"], x["cg"], x["k2"], x["u"], x["ustar"], x["drat"], pts["pin"][:, 3].copy(), udir,
                   x["z0"], x["cd"], x["tauwx"], x["tauwy"])
    sds4 = be.sds4(x["a"], x["k"], x["cg"], x["ustar"], x["usdir"], x["depth"], x["dair"], x["dlw"])
    spr4 = be.spr4(x["a"], x["cg"], x["k"], x["u"], udir, x["tauwx"], x["tauwy"], sin4["llws"], x["ustar"],
                   x["usdir"])
    f = lambda k: np.zeros(k, np.float32)  # noqa: E731
    for j in range(n):
        d, llws, tau, srhs, dd, brl, wc, o = f(ns), np.zeros(ns, np.int32), f(4), f(ns), f(ns), f(ns), f(4), f(12)
        rows = [np.ascontiguousarray(a[j]) for a in (x["a"], x["k"], x["cg"], pts["pin"], sin4["llws"])]
        routes.routes_terms(*[sc.p(r) for r in rows[:4]], x["ustar"][j], x["usdir"][j], x["dlw"][j], x["z0"][j],
                            x["tauwx"][j], x["tauwy"][j], sc.p(rows[4]),
                            *[sc.p(a) for a in (d, llws, tau, srhs, dd, brl, wc, o)])
        got = {"d": d, "tau": tau, "srhs": srhs, "ddiag": dd, "brlambda": brl, "whitecap": wc, "spr4": o}
        want = {"d": sin4["d"][j], "tau": np.array([sin4[k][j] for k in ("tauwx", "tauwy", "tauwnx", "tauwny")]),
                "srhs": sds4["srhs"][j], "ddiag": sds4["ddiag"][j], "brlambda": sds4["brlambda"][j],
                "whitecap": sds4["whitecap"][j],
                "spr4": np.array([spr4[k][j] for k in ("ustar", "usdir", "emean", "fmean", "fmean1", "wnmean",
                                                       "amax", "cd", "z0", "charn", "fmeanws", "dlwmean")])}
        assert not any(same(got, want).values()), (j, same(got, want))
        assert np.array_equal(llws, sin4["llws"][j])


needs_gpu = pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")


@pytest.mark.gpu
@needs_gpu
def test_grids_of_different_st4_options_fuse(pkg, synth):
    """One launch over the points of three grids of one spectral size whose ST4 parameters differ gives
    every grid the spectra of its own recorded step."""
    def record(base):
        grids, vas, steps = [], [], []
        for j, (shelter, n) in enumerate(((0.0, 1300), (0.3, 40), (0.0, 9))):
            st, t, sr, dia = config(synth, 25, 24, shelter)
            if j == 2:
                st["rpar"][st["R"]["SSDSC"] + 2] = 0.4  # the isotropic cumulative term
            g = pkg.SrceGrid(base + j, st["rpar"], st["ipar"], synth.st4_registrations(st, t), *dia, sr)
            p = synth.srce_points(n, seed=7 * j, nk=25, nth=24, depth_range=(5.0, 4000.0))
            va = np.zeros((n + 1, 600), np.float32)
            va[1:] = p["spec"]
            jsea = np.arange(n, 0, -1, dtype=np.int32)
            with pkg.Step(base + j) as step:
                g.batch_va(n, va, jsea, *[p[k] for k in ("wn1", "cg1", "pin", "psc", "whitecap", "taubbl",
                                                         "tauice")], np.zeros(n, np.int32), dtg=300.0)
            grids.append(g), vas.append(va), steps.append(step)
        return vas, steps

    def read(base, vas):
        for j, va in enumerate(vas):
            assert pkg.va_host_read(base + j, va) == 0

    own, steps = record(970)
    for s in steps:
        s.run(2)
    read(970, own)
    before, fsteps = record(980)
    start = [va.copy() for va in before]
    pkg.steps_fuse([980, 981, 982])
    pkg.steps_run([980, 981, 982], 2)
    pkg.steps_fuse([])
    read(980, before)
    for j in range(3):
        assert np.array_equal(own[j].view(np.uint32), before[j].view(np.uint32)), j
        assert not np.array_equal(start[j], before[j])
    for s in steps + fsteps:
        s.free()


@pytest.mark.gpu
@needs_gpu
def test_launches_of_two_threads_do_not_lower_each_others_limits(pkg, synth, capfd):
    """Two grids on two threads and streams, one with one slot per CTA and one with eight: neither call may
    be refused by the shared-memory limit that the other has set."""
    import threading

    import torch

    jobs = []
    for j, n in enumerate((3, 1200)):
        st, t, sr, dia = config(synth, 25, 24, 0.0)
        g = pkg.SrceGrid(990 + j, st["rpar"], st["ipar"], synth.st4_registrations(st, t), *dia, sr)
        p = synth.srce_points(n, seed=j, nk=25, nth=24, depth_range=(5.0, 4000.0))
        dev = [torch.from_numpy(np.ascontiguousarray(p[k])).cuda()
               for k in ("spec", "wn1", "cg1", "pin", "psc", "whitecap", "taubbl", "tauice")]
        jobs.append((g, n, dev + [torch.zeros(n, dtype=torch.int32, device="cuda")], torch.cuda.Stream()))
    torch.cuda.synchronize()
    capfd.readouterr()

    def call(g, n, dev, stream):
        for _ in range(300):
            g.L.ww_srce_batch_device(g.igrid, 1, 0, 1, 1, 10.0, n, *[d.data_ptr() for d in dev],
                                     ctypes.c_void_p(stream.cuda_stream))

    threads = [threading.Thread(target=call, args=job) for job in jobs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert "code" not in capfd.readouterr().err


def device_tables(pkg, synth, st):
    """INSIN4's tables of ``st`` built on the device; the DEL* steps go into st["rpar"]."""
    L = pkg.lib()
    pkg.init()
    mk, mth, mspec = (int(v) for v in st["ipar"][3:6])
    nsat = 2 * (mth // 2 - 1) + 1
    tabs = float(st["rpar"][st["R"]["SINTAILPAR"]]) > 0.5
    f = lambda n, on=True: np.zeros(n, np.float32) if on else None  # noqa: E731
    t = {"satweights": f(nsat * mth), "satindices": np.zeros(nsat * mth, np.int32),
         "iktab": np.zeros(mk * 2000, np.int32), "dcki": f(2000 * 1300), "qbi": f(2000 * 1300),
         "cumulw": f(mspec * mspec), "taut": f(201 * 201, tabs), "tauhft": f(101 * 201, tabs),
         "tauhft2": f(101 * 201 * 51, tabs)}
    dl = f(5)
    L.ww_st4_tables.argtypes = [P, sc.I, P, sc.I, P, P, P, P, sc.I] + [P] * 10
    L.ww_st4_tables.restype = sc.I
    assert L.ww_st4_tables(sc.p(st["rpar"]), st["rpar"].size, sc.p(st["ipar"]), st["ipar"].size,
                           *[sc.p(st[k]) for k in ("sig", "dsip", "th", "ecos")], 1,
                           *[sc.p(v) for v in t.values()], sc.p(dl)) == 0
    for name, v in zip(("DELUST", "DELALP", "DELTAUW", "DELU", "DELTAIL"), dl):
        st["rpar"][st["R"][name]] = v
    return dict(t, nsat=nsat)


@pytest.mark.gpu
@needs_gpu
@pytest.mark.parametrize("nk,nth,variant,mods,call", [
    (25, 24, "default", (), {}), (25, 24, "default", (sheltered, ice), {"inflags24": 1, "f58": 0}),
    (36, 36, "romero", (), {}), (25, 24, "romero", (spr4_twice,), {"f57": 0}),
    (25, 24, "default", (filipot,), {}), (12, 10, "default", (stab3,), {}),
    (25, 24, "analytic", (stab3, sheltered), {"it": 0}), (12, 10, "analytic", (spr4_twice, romero), {}),
    (25, 24, "analytic", (tail_level, spr4_twice), {"f57": 0, "f58": 0}),
    (36, 36, "analytic", (isotropic_cumulative, ice), {"it": 0, "inflags24": 1}),
    (12, 10, "default", (all_directions, ig1), {})],
    ids=lambda v: "+".join(f.__name__ for f in v) or "plain" if isinstance(v, tuple) else None)
def test_st4_forms_equal_host_build(pkg, routes, synth, nk, nth, variant, mods, call):
    """Breaking forms, tails, two-pass stresses, ice, IT = 0 and the whitecap flags, on host arrays and on
    the resident VA, with more points than one CTA has slots."""
    st = synth.st4_setup(nk, nth, variant=variant)
    sr = synth.srce_setup(st, ln1=1, seed=1)
    for m in mods:
        m(st, sr)
    t = device_tables(pkg, synth, st)
    dia = synth.dia_config(nk, nth)
    host_setup(routes, synth, st, t, sr, dia)
    routes.routes_derived(0)
    host = sc.hemu_backend(routes)
    grid = pkg.SrceGrid(next(_igrid), st["rpar"], st["ipar"], synth.st4_registrations(st, t), *dia, sr)
    gpu = sc.Backend(lambda name: (lambda *a: getattr(grid.L, "ww_" + name)(grid.igrid, *a)))
    n = 9 if nk == 36 else 310
    pts = synth.srce_points(n, seed=nk + n, nk=nk, nth=nth, depth_range=(5.0, 4000.0))
    pts["pin"][0, 2] = 0.0
    pts["pin"][:, 3] = np.linspace(-6.0, 2.0, n)  # AS
    pts["pin"][:, 4] = np.linspace(0.0, 0.9, n)   # ICE
    r, g = host.srce_batch(pts, dtg=60.0, **call), gpu.srce_batch(pts, dtg=60.0, **call)
    assert grid.L.ww_srce_last_error() == 0
    assert not any(same(r, g).values()), same(r, g)
    assert not np.array_equal(g["psc"], pts["psc"])
    va = np.zeros((n + 1, nk * nth), np.float32)
    jsea = np.random.default_rng(n).permutation(n).astype(np.int32) + 1
    va[jsea] = pts["spec"]
    v = {k: pts[k].copy() for k in ("psc", "whitecap", "taubbl", "tauice")}
    v["shave"] = np.zeros(n, np.int32)
    kw = {"f57": "flogrd57", "f58": "flogrd58"}
    grid.batch_va(n, va, jsea, pts["wn1"], pts["cg1"], pts["pin"], *v.values(), dtg=60.0,
                  **{kw.get(k, k): x for k, x in call.items()})
    assert pkg.va_host_read(grid.igrid, va) == 0
    assert not any(same(r, dict(v, spec=va[jsea])).values())


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
@pytest.mark.parametrize("nk,nth,shelter,ln1,seed,sizes", [
    (36, 36, 0.0, 0, 0, (1, 9)), (25, 24, 0.0, 1, 1, (1, 8, 150)), (25, 24, 0.3, 0, 0, (7, 300)),
    (36, 36, 0.3, 0, 1, (3,)), (13, 7, 0.0, 0, 0, (1, 1185)), (12, 10, 0.3, 1, 0, (17, 1300))])
def test_kernel_forms_equal_host_build(pkg, routes, synth, nk, nth, shelter, ln1, seed, sizes):
    st, t, sr, dia = config(synth, nk, nth, shelter, ln1, seed)
    host_setup(routes, synth, st, t, sr, dia)
    routes.routes_derived(0)
    host = sc.hemu_backend(routes)
    grid = pkg.SrceGrid(950 + nk, st["rpar"], st["ipar"], synth.st4_registrations(st, t), *dia, sr)
    gpu = sc.Backend(lambda name: (lambda *a: getattr(grid.L, "ww_" + name)(grid.igrid, *a)))
    for n in sizes:
        pts = synth.srce_points(n, seed=n, nk=nk, nth=nth, depth_range=(5.0, 4000.0))
        pts["pin"][0, 2] = 0.0
        # Fewer substeps a point keep the host build's share short.
        r, g = host.srce_batch(pts, dtg=60.0), gpu.srce_batch(pts, dtg=60.0)
        assert grid.L.ww_srce_last_error() == 0
        assert not any(same(r, g).values()), (n, same(r, g))
