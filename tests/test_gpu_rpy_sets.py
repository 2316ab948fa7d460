"""GPU tests of the product of one particle set on itself, every kernel and layout that a size can take, against the
FP64 oracle: the one-launch kernel of small sets (up to 1280 force-only particles), the symmetric kernel over pairs of
32-particle tiles (with torques from 512 particles), tiles that are partly filled or hold both segments and blobs, and
the tile kernel for unequal radii.  Tolerance: the mobility contract's 1e-5 relative L2."""
import numpy as np
import pytest
import torch

import oracle
from cufcm_fil_b200 import RpyMobilitySolver

pytestmark = pytest.mark.gpu
TOL = 1e-5


def particles(n_seg, n_blob, dof, wall, seed):
    """Particles on a shaken cubic lattice (some neighbours overlap), above the wall where there is one."""
    rng = np.random.default_rng(seed)
    n = n_seg + n_blob
    m = int(np.ceil(n ** (1 / 3)))
    cells = rng.permutation(m ** 3)[:n]
    x = 2.6 * np.stack([cells % m, cells // m % m, cells // m ** 2], 1) + rng.uniform(-0.5, 0.5, (n, 3))
    x[:, 2] += 2.0 if wall else 0.0
    f = np.zeros((n_seg, 6))
    f[:, :dof] = rng.standard_normal((n_seg, dof))
    as32 = lambda a: a.astype(np.float32)
    return as32(x[:n_seg]), as32(f), as32(x[n_seg:]), as32(rng.standard_normal((n_blob, 3)))


def check(n_seg, n_blob, dof, wall, **radii):
    xs, fs, xb, fb = particles(n_seg, n_blob, dof, wall, seed=7 * n_seg + n_blob)
    kw = dict(wall=wall, seg_dof=dof, **radii)
    w = lambda a: a.astype(np.float64)
    blobs = (xb, fb) if n_blob else ()
    with RpyMobilitySolver(n_seg, n_blob, **kw) as mob:
        vs, vb = mob.apply(xs, fs, *blobs)
    vs64, vb64 = oracle.mobility_full(w(xs), w(fs), *map(w, blobs), **kw)
    assert oracle.rel_l2(vs, vs64) <= TOL
    if n_blob:
        assert oracle.rel_l2(vb, vb64) <= TOL
    if dof == 3:
        assert (np.asarray(vs).reshape(-1, 6)[:, 3:] == 0).all()


@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 256, 1279, 1280, 1281, 2080])
def test_force_only_sets(cuda, n, wall):
    check(n, 0, 3, wall)


@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("n", [1, 33, 511, 512, 1041])
def test_sets_with_torques(cuda, n, wall):
    check(n, 0, 6, wall)


@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("dof,n_seg,n_blob", [(3, 5, 40), (3, 1000, 280), (3, 1000, 281), (6, 20, 30), (6, 480, 31), (6, 480, 32),
                                              (6, 1056, 70), (6, 31, 1100)])
def test_segments_and_blobs(cuda, dof, n_seg, n_blob, wall):
    check(n_seg, n_blob, dof, wall)


def test_unequal_radii_keep_their_blocks(cuda):
    check(700, 500, 6, False, seg_radius=1.0, blob_radius=0.7)


@pytest.mark.parametrize("n", [64, 2000])
def test_velocities_may_overwrite_the_forces(cuda, n):
    xs, fs, _, _ = particles(n, 0, 3, True, seed=1)
    dev = lambda a: torch.as_tensor(a.ravel(), device="cuda")
    with RpyMobilitySolver(n, 0, wall=True, seg_dof=3) as mob:
        x, f, v = dev(xs), dev(fs), torch.zeros(6 * n, device="cuda")
        mob.apply_device(x, f, v)
        torch.cuda.synchronize()
        want = v.cpu().numpy()
        mob.apply_device(x, f, f)
        torch.cuda.synchronize()
    assert oracle.rel_l2(f.cpu().numpy(), want) <= TOL
