"""Which step body a batch point runs, and that each is right. Lattices that pair
up run the packed body, as single systems do: bit for bit, whatever the
variant. Those that do not (an odd number of sites or of rows, rows too wide for
a split) run the unpacked bodies of their variant's queue and agree with
the same point run alone, on whichever unpacked kernel it takes, to the FP32
parity tolerance (1e-5)."""
import numpy as np
import pytest

from pincosimulator_gb300 import twmc

pytestmark = pytest.mark.gpu

DT, FS, FRAMES = 0.002, 50, 2
PACKED = [(1, 2), (2, 2), (1, 50), (6, 10), (16, 16), (1, 256), (32, 32), (2, 512), (50, 50), (64, 64), (80, 80),
          (96, 128), (128, 128)]
UNPACKED = [(5, 7), (7, 4), (5, 8), (1, 51), (25, 25), (33, 32), (49, 50), (45, 90), (63, 64), (81, 81), (99, 101),
            (4, 4096)]


def points(shapes):
    return [dict(nx=nx, ny=ny, U=0.2, omega=-0.5, F=1.5, dt=DT, n_traj=3 + i % 5 + (40 if nx * ny < 300 else 0),
                 seed0=100 * i + 3, id0=7 * i + 1) for i, (nx, ny) in enumerate(shapes)]


def single(p):
    s = twmc.System(nx=p["nx"], ny=p["ny"], J=1.0, gamma=1.0, dt=DT, frame_steps=FS, omega=p["omega"], U=p["U"],
                    F=p["F"], beta_init_sigma=0.5, hop=twmc.HOP_STENCIL)
    s.batch_init(s.make_tasks(p["n_traj"], seed0=p["seed0"], id0=p["id0"]))
    for _ in range(FRAMES):
        s.advance(FS)
    f, _ = s.download()
    kernel = s.step_kernel
    s.close()
    return f, kernel


def admitted(shapes, variant):
    out = []
    for p in points(shapes):
        try:
            twmc.HBatch([p], FS, variants=[variant]).close()
            out.append(p)
        except twmc.TWMCError as e:
            assert e.code == twmc.ERR_INVALID
    return out


REAL_SPACE = [v for v in twmc.HBatch.VARIANTS if v != "fft"]


@pytest.mark.parametrize("variant", REAL_SPACE)
def test_packed_points_equal_single_runs_bit_for_bit(built_lib, variant):
    pts = admitted(PACKED, variant)
    assert pts
    hb = twmc.HBatch(pts, FS, variants=[variant] * len(pts))
    hb.run(FRAMES)
    hb.sync()
    for i, p in enumerate(pts):
        assert "<pair " in hb.step_kernel(i), (p, hb.step_kernel(i))
        f, kernel = single(p)
        assert kernel.startswith("pair_"), (p, kernel)
        assert np.array_equal(hb.state(i), f), (p, hb.step_kernel(i), kernel)
    hb.close()


@pytest.mark.parametrize("variant", REAL_SPACE)
def test_unpacked_points_match_single_runs(built_lib, variant):
    pts = admitted(UNPACKED, variant)
    assert pts
    hb = twmc.HBatch(pts, FS, variants=[variant] * len(pts))
    hb.run(FRAMES)
    hb.sync()
    for i, p in enumerate(pts):
        assert "<ell" in hb.step_kernel(i), (p, hb.step_kernel(i))
        f, kernel = single(p)
        assert kernel.startswith("ell_"), (p, kernel)
        e = np.abs(hb.state(i) - f).max() / np.abs(f).max()
        assert e < 1e-5, (p, hb.step_kernel(i), kernel, e)
    hb.close()


def test_packed_and_unpacked_points_in_one_batch(built_lib):
    """Every queue at once, and 512-thread points of both kinds in one."""
    pts = points([(64, 64), (63, 64), (45, 90), (50, 50), (128, 128), (81, 81), (4, 4096), (80, 80), (5, 7), (6, 10)])
    variants = ["ell8w", "ell8w", "ell8w", "ell8w", "cluster", "cluster", "cluster_pow2", "cluster", "ell2", "ell2"]
    hb = twmc.HBatch(pts, FS, variants=variants)
    hb.run(FRAMES)
    hb.sync()
    for i, p in enumerate(pts):
        f, kernel = single(p)
        packed = "<pair " in hb.step_kernel(i)
        assert packed == kernel.startswith("pair_"), (p, hb.step_kernel(i), kernel)
        e = np.abs(hb.state(i) - f).max() / np.abs(f).max()
        assert e == 0 if packed else e < 1e-5, (p, hb.step_kernel(i), kernel, e)
    hb.close()
