"""GPU tests of the force-coupling transforms on the used rows (csrc/fcm_fft.cuh) against the FP64 oracle: every
radix, short and long stages, box shapes with different axes, axes that fall back to the general transforms, and
particles in one corner (most rows unused, supports across the periodic boundary) or spread over the box.
Tolerance 1e-4 relative L2, as for the other FP32 grids of test_gpu_fcm.py."""
import numpy as np
import pytest

import oracle
from oracle import fcm as ofcm
from cufcm_fil_b200.fcm import FcmSolver

pytestmark = pytest.mark.gpu


# Grids large enough for these transforms: fixed lengths 128 to 1024 on each axis, every runtime radix, two-stage
# lengths; the last two fall back to the general transforms (a prime factor 11, an axis above 1024).
SHAPES = [(512, 96, 128, "corner"), (200, 180, 162, "everywhere"), (256, 128, 192, "corner"), (30, 500, 375, "corner"),
          (2048, 54, 50, "everywhere"), (24, 512, 512, "corner"), (64, 1024, 90, "corner"), (80, 72, 1024, "everywhere"),
          (1024, 64, 90, "everywhere"), (128, 256, 256, "corner"), (352, 132, 132, "corner"), (32, 1080, 162, "corner")]


@pytest.mark.parametrize("nx,ny,nz,where", SHAPES)
def test_matches_fp64_oracle(cuda, nx, ny, nz, where):
    dx, n = 2.0, 60
    kw = dict(rh=1.0, alpha=1.0, beta=8.0, eta=5.0, nx=nx, ny=ny, nz=nz, boxsize=nx * dx)
    rng = np.random.default_rng(nx + ny + nz)
    box = dx * np.array([nx, ny, nz])
    m = 4 if where == "corner" else None
    if m:  # a 4 x 4 x 4 cluster of spacing 2.6 around the origin, wrapped into the box
        cells = np.stack(np.unravel_index(rng.permutation(m ** 3)[:n], (m, m, m)), 1)
        Y = np.mod(2.6 * (cells - 1.5) + rng.uniform(-0.1, 0.1, (n, 3)), box)
    else:  # a lattice over the whole box, at least 2.6 apart
        k = np.maximum(1, np.floor(box / 2.6)).astype(int)
        idx = rng.choice(int(np.prod(k)), min(n, int(np.prod(k))), replace=False)
        Y = np.stack(np.unravel_index(idx, k), 1) * (box / k) + 0.3
    F = rng.standard_normal(Y.shape)
    Y, F = Y.astype(np.float32), F.astype(np.float32)
    with FcmSolver(len(Y), **kw) as s:
        first = s.hydrodynamic_solver(Y, F)
        s.hydrodynamic_solver(np.mod(Y + 0.37 * box, box).astype(np.float32), F)  # other rows of the same grid
        again = s.hydrodynamic_solver(Y, F)
    v64 = ofcm.fcm_apply(Y.astype(np.float64), F.astype(np.float64), ofcm.FcmParams(**kw))
    assert oracle.rel_l2(first, v64) <= 1e-4
    assert oracle.rel_l2(again, first) <= 1e-5  # nothing of the other rows is left (atomic order aside)
