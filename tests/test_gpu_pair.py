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


@pytest.mark.parametrize("par,ramp", [("scalar", False), ("im", False), ("im", True), ("site", True), ("site", False)])
@pytest.mark.parametrize("cells,pbc", [(2, True), (2, False), (6, True), (66, False), (256, True), (1024, False)])
def test_packed_lieb_matches_oracle(built_lib, oracle, cells, pbc, par, ramp):
    """The packed Lieb kernel (cells c and c + Nc/2 in the lanes): rings and
    open chains, one slot to the most a CTA holds, F(t) over several table
    segments, J_AB != J_BC so that each coupling lands on its bond."""
    n, steps, dt = 3 * cells, 60, 0.002
    rng = np.random.default_rng(cells)
    beta0 = 0.4 * (rng.normal(size=(2, n)) + 1j * rng.normal(size=(2, n)))
    E, U, F, F_t = 0.1, 0.27, 0.3, None
    if par != "scalar":
        E, U = 0.1 * rng.normal(size=n), 0.27 + 0.06 * rng.random(size=n)
    if par == "site":
        E, U, F = E + 0.02j * rng.normal(size=n), U + 0.01j * rng.normal(size=n), 0.3 + 0.1j * rng.normal(size=n)
    if ramp:
        times = np.round(np.arange(0, 0.09, 0.01), 10)
        F_t = (times, np.outer(times / 0.05, 1.0 + 0.2 * rng.random(n)) * (1 + 0.3j))
    s = twmc.System(lattice=twmc.LATTICE_LIEB, nx=1, ny=cells, pbc=pbc, J_AB=0.8, J_BC=1.3, gamma=1.0, detuning=0.5,
                    dt=dt, frame_steps=steps, omega=E, U=U, F=F, F_t=F_t)
    seeds = [7, 123]
    tasks = s.make_tasks(2, t_end=steps * dt, ic=twmc.IC_GIVEN, init_field=beta0, seeds=seeds, id0=4)
    res = s.run(tasks, frames=False)
    assert s.kernel_name == "lieb_cell_kernel"
    s.close()
    for k in range(2):
        xi = twmc.debug_wiener(twmc.PREC_F32, seeds[k], 4 + k, steps, n)
        ref = oracle.lieb_run(cells, pbc, 0.8, 1.3, 0.5, 1.0, dt, 0.0, steps * dt, steps, 2, True, E, U, F, beta0[k],
                              xi=xi, F_t=F_t)
        assert rel_err(res["final"][k], ref["final"]) < 1e-5
