"""Creation of a mobility handle while little device memory is free: where the partials of the symmetric product do not
fit, the handle is made with the tile kernel's and its products are right."""
import numpy as np
import pytest
import torch

import oracle
from cufcm_fil_b200 import RpyMobilitySolver

from .test_gpu_rpy_sets import TOL, particles

pytestmark = pytest.mark.gpu

FREE = 300 << 20  # what is left: the symmetric product of 20,480 particles with torques has 420 MB of partials


@pytest.mark.parametrize("n_seg,n_blob", [(20480, 0), (14336, 6144)])
def test_creation_with_little_memory(cuda, n_seg, n_blob):
    xs, fs, xb, fb = particles(n_seg, n_blob, 6, False, seed=3)
    targets = np.random.default_rng(2).permutation(n_seg)[:200]
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(max(0, free - FREE), dtype=torch.uint8, device="cuda")
    try:
        with RpyMobilitySolver(n_seg, n_blob, wall=False, seg_dof=6) as mob:
            vs, vb = mob.apply(xs, fs, *((xb, fb) if n_blob else ()))
    finally:
        del hold
        torch.cuda.empty_cache()
    w = lambda a: a.astype(np.float64)
    blobs = (w(xb), w(fb)) if n_blob else ()
    vs64, vb64 = oracle.mobility_full(w(xs), w(fs), *blobs, wall=False, seg_dof=6, seg_targets=targets)
    assert oracle.rel_l2(np.asarray(vs).reshape(-1, 6)[targets], vs64) <= TOL
    if n_blob:
        assert oracle.rel_l2(vb, vb64) <= TOL
