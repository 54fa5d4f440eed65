"""Host code of the library on the CPU, linked with a stand-in for the CUDA
runtime (fake_cudart.cpp) whose streams run their work as late as the runtime
allows. Each test runs a script in a process of its own."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PRELUDE = """
import ctypes as C
import numpy as np
from pincosimulator_gb300 import twmc
lib = twmc.load()
for f in ("fake_uploads", "fake_changed", "fake_lowered", "fake_queued_most"):
    getattr(lib, f).restype = C.c_long
lib.fake_pinned_peak.restype = C.c_size_t
lib.fake_pinned_limit.argtypes = [C.c_size_t]
lib.fake_fail_launch.argtypes = [C.c_char_p, C.c_long]
lib.fake_log.restype = C.c_char_p
lib.fake_cost.argtypes = [C.c_char_p, C.c_double]
lib.fake_pin.argtypes = [C.c_void_p, C.c_size_t]
def chain(n_traj, n_frames, sites=64):
    s = twmc.System(nx=1, ny=sites, J=1.0, dt=0.01, frame_steps=2, omega=-0.5, U=0.2, F=1.0, beta_init_sigma=0.5)
    t = s.make_tasks(n_traj, t_end=0.02 * (n_frames - 1))
    return s, t, {"frames": np.full((n_traj, n_frames, sites), np.nan + 0j)}
"""


@pytest.fixture(scope="session")
def fake_lib(built_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("fake_cudart")
    obj, lib = str(d / "fake.o"), str(d / "libtwmc_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-I/usr/local/cuda/include", "-c",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", obj], check=True)
    from pincosimulator_gb300 import build_ext

    objs = [os.path.join(build_ext.BUILD, s.replace(".cu", ".o")) for s in build_ext.SOURCES]
    if not all(map(os.path.exists, objs)):
        build_ext.build(force=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined", *objs, obj, "-o", lib], check=True)
    return lib


@pytest.fixture
def script(fake_lib):
    def go(text):
        r = subprocess.run([sys.executable, "-c", PRELUDE + text], capture_output=True, text=True, timeout=120,
                           env=dict(os.environ, TWMC_LIB=fake_lib, PYTHONPATH=ROOT))
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return go


def test_sources_of_uploads_live_until_their_copies_have_run(script):
    """An asynchronous copy from pageable memory may read its source after the
    call: tables, parameters, seeds, given fields and realisations, caller noise
    and the F(t) schedule must still be there when the stream runs it."""
    script("""
rng = np.random.default_rng(1)
c = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
def square(n_traj=5, **kw):
    a = dict(nx=16, ny=16, J=1.0, dt=0.01, frame_steps=2, omega=c(256), U=twmc.Noisy(c(256), 1, c(256)), F=c(256),
             beta_init=c(256), beta_init_sigma=c(256))
    a.update(kw)
    s = twmc.System(**a)
    t = s.make_tasks(n_traj, t_end=0.04, ic=twmc.IC_GIVEN, init_field=c(n_traj, 256),
                     realizations={"U": c(n_traj, 256)})
    return s, t
for prec in (twmc.PREC_F32, twmc.PREC_F64):
    for integ in (twmc.INTEGRATOR_EULER, twmc.INTEGRATOR_SPLIT):
        s, t = square(precision=prec, integrator=integ)
        s.run(t, realizations=True)
        s.run(t, moments=True)
        s.batch_init(t); s.advance(3); s.batch_init(t); s.advance(3); s.reduce(); s.sync()
        for _ in range(40):
            s.batch_init(t); s.advance(1)
        s.sync()
        s.close()
    s, t = square(precision=prec, noise=twmc.NOISE_BUFFER)
    s.set_noise(c(5, 4, 256))
    s.run(t)
    s.close()
    times = np.arange(0, 0.1, 0.01)
    s = twmc.System(lattice=twmc.LATTICE_LIEB, nx=1, ny=8, J_AB=1.0, J_BC=1.0, dt=0.002, frame_steps=5, precision=prec,
                    U=c(24), F_t=(times, c(len(times), 24)))
    s.run(s.make_tasks(3, t_end=0.04))
    s.close()
assert lib.fake_uploads() > 600, lib.fake_uploads()
assert lib.fake_changed() == 0, (lib.fake_changed(), lib.fake_uploads())
""")


@pytest.mark.parametrize("sites", [64, 8192])  # frames collected on the device; frames staged one by one
def test_progress_counts_steps_that_have_run(script, sites):
    """At the k-th step launch of a run of five, at most k of them have run."""
    script(f"sites = {sites}" + """
s, t, bufs = chain(130, 6, sites)
seen = []
def hook(name):
    if b"fft_kernel" in name or b"pair" in name:
        p = C.c_double()
        lib.twmc_progress(s.h, C.byref(p))
        seen.append(p.value)
CB = C.CFUNCTYPE(None, C.c_char_p)
cb = CB(hook)
lib.fake_hook(cb)
s.run(t, final=False, buffers=bufs)
assert len(seen) == 5, seen
assert all(p <= k / 5 + 1e-12 for k, p in enumerate(seen)), seen
p = C.c_double()
lib.twmc_progress(s.h, C.byref(p))
assert p.value == 1.0
lib.fake_hook(CB(0))
s.close()
""")


def test_collected_frames_without_page_locked_memory(script):
    """The buffer that frames go home through is bounded, and a run does
    not need it."""
    script("""
s, t, bufs = chain(500, 80)   # 41 MB of frames
s.run(t, buffers=bufs)
assert not np.isnan(bufs["frames"]).any()
assert 0 < lib.fake_pinned_peak() <= 1 << 24, lib.fake_pinned_peak()
s.close()
for limit in (0, 1 << 20):
    lib.fake_pinned_limit(limit)
    s, t, bufs = chain(500, 8)   # 4 MB
    s.run(t, buffers=bufs)
    assert not np.isnan(bufs["frames"]).any()
    s.close()
""")


def test_partly_page_locked_frames(script):
    """A caller's array of which only a part is page-locked: not one copy, which
    the runtime refuses."""
    script("""
for part in (4096, 100000):
    s, t, bufs = chain(20, 10)
    lib.fake_pin(bufs["frames"].ctypes.data, part)
    s.run(t, buffers=bufs)
    assert not np.isnan(bufs["frames"]).any()
    s.close()
""")


def test_frames_before_an_error_reach_the_caller(script):
    script("""
s, t, bufs = chain(20, 10)
lib.fake_fail_launch(b"square_fft_kernel", 3)   # the fourth launch: frames 0 to 3 are there
try:
    s.run(t, buffers=bufs)
    raise SystemExit("no error")
except twmc.TWMCError:
    pass
lost = np.isnan(bufs["frames"]).any(axis=(0, 2))
assert not lost[:4].any() and lost[4:].all(), lost
s.close()
""")


@pytest.mark.parametrize("n_frames", [1, 3])
def test_step_time_is_that_of_the_step_launches(script, n_frames):
    """twmc_sync's step time after a run whose last steps go in ranges on streams
    of their own, each followed by its widening and its copy home: the step
    launches' time, overlapping ones counted once, and nothing else's."""
    script(f"n_frames = {n_frames}" + """
lib.fake_cost(b"fft_kernel", 1.0)
lib.fake_cost(b"widen_kernel", 10.0)
lib.fake_cost(b"memcpy", 100.0)
s = twmc.System(nx=16, ny=16, J=1.0, dt=0.01, frame_steps=2, omega=-0.5, U=0.2, F=1.0, beta_init_sigma=0.5)
t = s.make_tasks(4096, t_end=0.02 * n_frames, store_initial=False)
for frames in (False, True):
    s.run(t, frames=frames)
    ms = s.sync()
    assert n_frames <= ms <= n_frames + 3, ms   # each stretch once; the four ranges one after the other at most
s.batch_init(t)
s.advance(2); s.advance(2); s.reduce()
assert s.sync() == 2.0
assert s.sync() == 0.0
s.close()
""")


def test_step_kernel_names_the_kernel_launched(script):
    script("""
def last_step():
    names = [n for n in lib.fake_log().decode().split() if "kernel" in n]
    return [n for n in names if any(k in n for k in ("pair", "ell_", "lieb_cell", "fft_kernel"))][-1]
def check(want, **kw):
    a = dict(J=1.0, dt=0.01, frame_steps=2, omega=-0.5, U=0.2, F=1.0, hop=twmc.HOP_STENCIL)
    a.update(kw)
    s = twmc.System(**a)
    assert s.step_kernel == ""
    s.batch_init(s.make_tasks(7))
    s.advance(1)
    got = s.step_kernel
    assert got.split("<")[0] in (want, want + "_wide"), (kw, got)
    assert got.split("<")[0] + "I" in last_step(), (kw, got, last_step())
    s.close()
for nx, ny in [(1, 2), (2, 2), (6, 10), (50, 50), (64, 64), (1, 1000), (2, 2048)]:
    for kw in ({}, dict(U=twmc.Noisy(0.2, 1, 0.1)), dict(omega=twmc.Noisy(0.2, 1, 0.1))):
        check("pair_kernel", nx=nx, ny=ny, **kw)
check("pair_kernel", nx=1, ny=8192)
check("pair_cluster_kernel", nx=128, ny=128)
check("pair_cluster_kernel", nx=80, ny=80)
for nx, ny in [(5, 7), (7, 4), (25, 25), (49, 50)]:
    check("ell_kernel", nx=nx, ny=ny)
check("ell_kernel", nx=64, ny=64, precision=twmc.PREC_F64)
check("ell_cluster_kernel", nx=99, ny=101)
check("ell_cluster_pow2_kernel", nx=4, ny=4096)
check("square_fft_kernel", nx=64, ny=64, hop=twmc.HOP_FFT)
lieb = dict(lattice=twmc.LATTICE_LIEB, nx=1, J_AB=1.0, J_BC=1.0)
check("lieb_pair_kernel", ny=8, **lieb)
check("lieb_pair_kernel", ny=1024, **lieb)
check("lieb_cell_kernel", ny=8, precision=twmc.PREC_F64, **lieb)
check("ell_kernel", ny=7, **lieb)
pts = lambda *shapes: [dict(nx=nx, ny=ny, dt=0.01, n_traj=3) for nx, ny in shapes]
hb = twmc.HBatch(pts((1, 32), (6, 10), (5, 7), (128, 128), (80, 80), (81, 81), (4, 4096), (45, 90)), 10)
kernels = [hb.step_kernel(i).split(" ")[0].rstrip(">") for i in range(8)]
assert kernels == ["hbatch_kernel<fft", "hbatch_kernel<pair", "hbatch_kernel<ell", "hbatch_cluster4_kernel<pair",
                   "hbatch_cluster_kernel<pair", "hbatch_cluster_kernel_ell<ell_cluster",
                   "hbatch_cluster_kernel_ell<ell_cluster_pow2", "hbatch_kernel_512_ell<ell"], kernels
hb.close()
hb = twmc.HBatch(pts((64, 64)), 10, variants=["rowrun"])
assert hb.step_kernel(0) == "hbatch_kernel_512<pair 2,2>", hb.step_kernel(0)
hb.close()
hb = twmc.HBatch(pts((64, 64), (63, 64)), 10, variants=["ell8w", "ell8w"])   # one queue for both
assert [hb.step_kernel(i) for i in range(2)] == ["hbatch_kernel_512<pair 2,2>", "hbatch_kernel_512<ell>"]
hb.close()
""")


def test_tuned_choices_hold_for_the_kernels_they_were_timed_on(script, tmp_path):
    """A cached choice without the revision of the queue kernels is not taken, and
    a new one is kept beside it. (The stand-in times nothing: the first variant
    that a lattice admits wins.)"""
    cache = tmp_path / "tune.json"
    cache.write_text('{\n  "fake|64x64": "ell8w",\n  "fake|0123456789ab|64x64": "rowrun"\n}\n')
    script(f"cache = {str(cache)!r}" + """
import json, os
os.environ["TWMC_TUNE_CACHE"] = cache
from pincosimulator_gb300 import build_ext
pts = [dict(nx=64, ny=64, dt=0.01, n_traj=3)]
hb = twmc.HBatch(pts, 10, tune=True)
assert "<fft " in hb.plan(0), hb.plan(0)
hb.close()
entries = json.load(open(cache))
assert entries == {"fake|64x64": "ell8w", "fake|0123456789ab|64x64": "rowrun",
                   "fake|" + build_ext.queue_revision() + "|64x64": "fft"}, entries
text = open(cache).read().replace('"fft"', '"ell8w"')
open(cache, "w").write(text)
hb = twmc.HBatch(pts, 10, tune=True)
assert "<ell8w " in hb.plan(0), hb.plan(0)
assert open(cache).read() == text
hb.close()
""")


@pytest.mark.parametrize("nx,ny,trials", [
    (64, 64, 2),    # fft; rowrun and ell8w run the same split
    (32, 32, 4),    # fft, ell4, ell8 (one split), rowrun and ell8w (another)
    (128, 128, 1),  # both cluster names run clusters of four
    (4, 4096, 2),   # no packed split: the two unpacked cluster bodies
    (25, 25, 3),    # odd: ell4, ell8, ell8w
])
def test_tuner_times_each_kernel_once(script, tmp_path, nx, ny, trials):
    """Variant names that run the same kernel on a lattice are one trial, and its
    first name is kept, not the one that noise favours."""
    script(f"nx, ny, trials, cache = {nx}, {ny}, {trials}, {str(tmp_path / 'c.json')!r}" + """
import os
os.environ["TWMC_TUNE_CACHE"] = cache
hb = twmc.HBatch([dict(nx=nx, ny=ny, dt=0.01, n_traj=3)], 10, tune=True)
queues = [n for n in lib.fake_log().decode().split() if "hbatch_kernel" in n or "hbatch_cluster" in n]
assert len(queues) == trials + 1, queues   # and the batch itself
hb.close()
""")


def test_shared_memory_limits_are_not_lowered(script):
    """The limit of a kernel's dynamic shared memory is process-wide: a launch that
    needs less must not lower it under another thread's launch that needs more."""
    script("""
def go(n_traj, **kw):
    a = dict(J=1.0, dt=0.01, frame_steps=2, omega=-0.5, U=0.2, F=1.0, hop=twmc.HOP_STENCIL)
    a.update(kw)
    s = twmc.System(**a)
    s.batch_init(s.make_tasks(n_traj))
    s.advance(1)
    s.close()
for n_traj in (4000, 1, 300):
    for nx, ny in [(32, 32), (16, 16), (64, 64), (50, 50), (6, 10), (128, 128), (80, 80), (96, 96), (99, 101), (5, 7),
                   (4, 4096), (128, 4), (1, 4096), (1, 50)]:
        go(n_traj, nx=nx, ny=ny)
        go(n_traj, nx=nx, ny=ny, omega=twmc.Noisy(-0.5, 1, 0.2))
    for cells in (256, 16, 7, 1024):
        for prec in (twmc.PREC_F32, twmc.PREC_F64)[:1 if cells > 256 else 2]:  # 1024 cells fit in FP32 only
            go(n_traj, lattice=twmc.LATTICE_LIEB, nx=1, ny=cells, J_AB=1.0, J_BC=1.0, precision=prec)
    for integ in (twmc.INTEGRATOR_SPLIT, twmc.INTEGRATOR_EULER):
        for prec in (twmc.PREC_F32, twmc.PREC_F64):
            go(n_traj, nx=16, ny=16, hop=twmc.HOP_FFT, integrator=integ, precision=prec, U=twmc.Noisy(0.2, 1, 0.1))
for shapes in ([(64, 64), (128, 128)], [(6, 10), (80, 80), (25, 25)], [(128, 128), (96, 96)], [(50, 50)], [(120, 100)]):
    twmc.HBatch([dict(nx=nx, ny=ny, dt=0.01, n_traj=3) for nx, ny in shapes], 10).close()
assert lib.fake_lowered() == 0, lib.fake_lowered()
""")


def test_kept_sources_are_bounded(script):
    """Batches that nothing waits for: their uploads' sources do not pile up."""
    script("""
rng = np.random.default_rng(2)
s = twmc.System(nx=64, ny=64, J=1.0, dt=0.01, frame_steps=2)
f = rng.normal(size=(100, 4096)) + 1j * rng.normal(size=(100, 4096))   # 6.6 MB
t = s.make_tasks(100, ic=twmc.IC_GIVEN, init_field=f)
for _ in range(40):
    s.batch_init(t)
    s.advance(1)
assert lib.fake_changed() == 0
assert lib.fake_queued_most() < (1 << 26) + (1 << 23), lib.fake_queued_most()
s.close()
""")
