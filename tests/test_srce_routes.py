"""The routes W3SRCE's kernel takes by a rule, against the general ones: on the CPU the tables derived
from the registered ones and the branch-free libm forms (bit for bit), on the GPU the kernel's forms (36,
24 and other numbers of directions, with and without sheltering, numbers of points around the slots
and CTAs) against the host build of the same source, one point at a time."""

import ctypes
import re
import subprocess

import numpy as np
import pytest

from conftest import cuda_available
import st4_common as sc

P = ctypes.c_void_p


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
