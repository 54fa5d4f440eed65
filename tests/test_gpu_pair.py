"""The packed real-space kernel (site p and p + N/2 in the two lanes of
packed FP32 instructions): FP32 Philox runs against the oracle fed the
device's normals at the FP32 parity tolerance (1e-5), on lattices at the
edges of its splits -- two-site lattices, one row of pairs, rows that no run
length divides, ragged warps, chains of odd halves, one CTA, clusters of 2 and
4 CTAs -- and on odd ones, which it leaves to the unpacked kernels."""
import numpy as np
import pytest

from pincosimulator_gb300 import twmc

from gpu_util import philox_ref, rel_err

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2), (2, 1), (2, 2), (2, 3), (1, 50), (6, 10), (22, 7), (30, 34), (50, 50), (2, 2048), (64, 1),
          (1, 1034), (80, 80), (128, 64), (100, 120), (98, 102), (1, 16384), (5, 7), (7, 4)]


def run(nx, ny, par, n_traj, steps, beta0, seeds, rng):
    n = nx * ny
    kw = dict(omega=-0.5, U=0.2, F=1.5)
    if par != "scalar":
        kw["omega"] = -0.5 + 0.2 * rng.normal(size=n)
    if par == "site":
        kw["omega"] = kw["omega"] + 0.02j * rng.normal(size=n)
        kw["U"] = 0.2 + 0.05 * rng.random(size=n) + 0.01j
        kw["F"] = 1.0 + 0.3 * rng.normal(size=n) + 0.1j
    s = twmc.System(nx=nx, ny=ny, J=1.0, gamma=1.0, dt=0.005, frame_steps=steps, hop=twmc.HOP_STENCIL, **kw)
    tasks = s.make_tasks(n_traj, t_start=0.0, t_end=steps * 0.005, ic=twmc.IC_GIVEN, init_field=beta0[:n_traj],
                         seeds=seeds[:n_traj], id0=9)
    res = s.run(tasks, frames=False)
    s.close()
    assert (res["status"] == 0).all()
    return res["final"], kw


@pytest.mark.parametrize("par", ["scalar", "rsl", "site"])
@pytest.mark.parametrize("shape", SHAPES)
def test_packed_steps_match_oracle(built_lib, oracle, shape, par):
    nx, ny = shape
    n = nx * ny
    steps = 60 if n <= 1024 or n & (n - 1) == 0 else 15  # the oracle's transform of other sides is quadratic
    rng = np.random.default_rng(nx * 1000 + ny)
    beta0 = 0.3 * (rng.normal(size=(2, n)) + 1j * rng.normal(size=(2, n)))
    seeds = [21, 4242]
    final, kw = run(nx, ny, par, 2, steps, beta0, seeds, rng)
    for k in range(2):
        ref = philox_ref(oracle, twmc.PREC_F32, seeds[k], 9 + k, steps, n, nx=nx, ny=ny, J=1.0, gamma=1.0, dt=0.005,
                         t_start=0.0, t_end=steps * 0.005, frame_steps=steps, n_frames=2, store_initial=True,
                         beta0=beta0[k], **kw)
        assert rel_err(final[k], ref["final"]) < 1e-5


@pytest.mark.parametrize("shape", [(16, 16), (6, 10), (50, 50), (64, 64), (1, 1000), (128, 128)])
def test_packed_bits_do_not_depend_on_the_batch(built_lib, shape):
    """The split changes with the number of trajectories, a trajectory's bits
    do not: one alone, a few, and as many as fill the device."""
    nx, ny = shape
    many = 700 if nx * ny < 10000 else 310
    rng = np.random.default_rng(3)
    beta0 = 0.3 * (rng.normal(size=(many, nx * ny)) + 1j * rng.normal(size=(many, nx * ny)))
    seeds = list(range(50, 50 + many))
    out = [run(nx, ny, "rsl", k, 20, beta0, seeds, np.random.default_rng(8))[0] for k in (1, 17, many)]
    assert np.array_equal(out[0], out[2][:1]) and np.array_equal(out[1], out[2][:17])
