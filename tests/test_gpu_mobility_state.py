"""What a mobility handle holds after a one-call product: cf_apply_mobility stages positions and forces as the single
copy calls do, so an evaluation after it, with or without new forces, works on the call's own particles.  Below and
above the size at which one launch serves the whole call.  Tolerance: the mobility contract's 1e-5 relative L2."""
import numpy as np
import pytest
import torch

import oracle
from cufcm_fil_b200 import RpyMobilitySolver

from .test_gpu_rpy_sets import TOL, particles

pytestmark = pytest.mark.gpu


def reference(xs, fs, xb, fb, wall):
    w = lambda a: a.astype(np.float64)
    blobs = (w(xb), w(fb)) if len(xb) else ()
    return oracle.mobility_full(w(xs), w(fs), *blobs, wall=wall, seg_dof=3)


@pytest.mark.parametrize("device_call", [False, True])
@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("n_seg,n_blob", [(64, 0), (40, 24), (1280, 0), (1281, 0), (2000, 30)])
def test_evaluations_after_apply_see_its_particles(cuda, n_seg, n_blob, wall, device_call):
    dev = lambda a: torch.as_tensor(a.ravel(), device="cuda")
    zeros = lambda k: torch.zeros(k, device="cuda")
    with RpyMobilitySolver(n_seg, n_blob, wall=wall, seg_dof=3) as mob:
        for seed in (11, 12):  # a new handle, then one that has seen other positions
            xs, fs, xb, fb = particles(n_seg, n_blob, 3, wall, seed)
            if device_call:
                mob.apply_device(dev(xs), dev(fs), zeros(6 * n_seg), dev(xb), dev(fb), zeros(3 * n_blob))
                torch.cuda.synchronize()
            else:
                mob.apply(xs, fs, *((xb, fb) if n_blob else ()))
            for new_forces in (False, True):
                if new_forces:  # positions once, forces again: an iteration of a solver
                    fs = particles(n_seg, n_blob, 3, wall, seed + 50)[1]
                    mob.f_segs_host[:] = fs.ravel()
                    mob.copy_segment_forces_to_device()
                mob.evaluate_full_mobility()
                mob.copy_segment_velocities_to_host()
                mob.copy_blob_velocities_to_host()
                vs64, vb64 = reference(xs, fs, xb, fb, wall)
                assert oracle.rel_l2(mob.v_segs_host, vs64) <= TOL
                if n_blob:
                    assert oracle.rel_l2(mob.v_blobs_host, vb64) <= TOL
