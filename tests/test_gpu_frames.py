"""Saved frames of small runs (collected on the device, then copied home): the
state after as many steps, for page-locked and pageable arrays, in more pieces
than one with trajectories across their ends, and for two task groups whose
frames lie in longer rows than their own."""
import numpy as np
import pytest

from pincosimulator_gb300 import twmc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("groups", [1, 2])
def test_frames_are_the_states_between_steps(built_lib, pinned, groups):
    n_traj, frames, sites, fs = 300, 70, 64, 3   # 21.5 MB, pieces of 16 MB
    dt = 0.002
    s = twmc.System(nx=1, ny=sites, J=1.0, gamma=1.0, dt=dt, frame_steps=fs, omega=twmc.Noisy(-0.5, 1, 0.2), U=0.2,
                    F=1.5, beta_init_sigma=0.5)
    t = s.make_tasks(n_traj, t_end=(frames - 1) * fs * dt, seed0=5, id0=11)
    count = np.full(n_traj, frames)
    if groups == 2:
        count[170:] = 61
        for k in range(170, n_traj):
            t[k].t_end = 60 * fs * dt
    buf = torch.full((n_traj, frames, sites), float("nan"), dtype=torch.complex128, pin_memory=pinned).numpy()
    res = s.run(t, buffers={"frames": buf})
    assert np.array_equal(res["frames_written"], count)
    s.batch_init(t)
    for f in range(frames):
        state, _ = s.download()
        rows = count > f
        assert np.array_equal(buf[rows, f], state[rows]), f
        assert np.isnan(buf[~rows, f]).all(), f
        s.advance(fs)
    s.close()
