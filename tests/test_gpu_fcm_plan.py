"""GPU tests of the force-coupling transforms (csrc/fcm_fft.cuh) at the lengths that its rule admits: against the FP64
oracle (tolerance 1e-4 relative L2, as test_gpu_fcm_fft.py), and, for the longest, three axis orders of one grid against
each other (1e-5: the same sums but for the order of the stages)."""
import numpy as np
import pytest
import torch

import oracle
from oracle import fcm as ofcm
from cufcm_fil_b200.fcm import FcmSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(486, 100, 125), (160, 250, 250), (320, 160, 135), (640, 128, 128), (512, 256, 128),
                                      (162, 180, 200)])
def test_lengths(cuda, nx, ny, nz):
    dx, n = 2.0, 60
    kw = dict(rh=1.0, alpha=1.0, beta=8.0, eta=5.0, nx=nx, ny=ny, nz=nz, boxsize=nx * dx)
    rng = np.random.default_rng(nx + ny + nz)
    Y = rng.uniform(0, 1, (n, 3)) * dx * np.array([nx, ny, nz])
    Y, F = Y.astype(np.float32), rng.standard_normal((n, 3)).astype(np.float32)
    with FcmSolver(n, **kw) as s:
        v = s.hydrodynamic_solver(Y, F)
    v64 = ofcm.fcm_apply(Y.astype(np.float64), F.astype(np.float64), ofcm.FcmParams(**kw))
    assert oracle.rel_l2(v, v64) <= 1e-4


def test_longest_axes_agree(cuda):
    n, dx, shape = 2000, 2.0, (1024, 256, 256)
    rng = np.random.default_rng(8)
    Y = rng.uniform(0, 1, (n, 3)) * dx * np.array(shape)
    F = rng.standard_normal((n, 3))
    out = []
    for turn in range(3):
        roll = lambda a: torch.as_tensor(np.roll(a, turn, axis=1).astype(np.float32).ravel(), device="cuda")
        nx, ny, nz = np.roll(shape, turn)
        V = torch.zeros(3 * n, device="cuda")
        with FcmSolver(n, rh=1.0, alpha=1.0, beta=8.0, eta=5.0, nx=nx, ny=ny, nz=nz, boxsize=nx * dx) as s:
            s.apply_device(roll(Y), roll(F), V)
            torch.cuda.synchronize()
        out.append(np.roll(V.cpu().numpy().reshape(n, 3), -turn, axis=1))
    assert oracle.rel_l2(out[1], out[0]) <= 1e-5
    assert oracle.rel_l2(out[2], out[0]) <= 1e-5
