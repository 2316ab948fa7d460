"""Products of one set of equal particles at the limits of single precision: particles at the places of the inert ones
that fill a tile, and spheres of a few nanometres in SI units, where fifth powers of a distance leave the range.
Against the FP64 oracle; tolerance 1e-5 relative L2 (the mobility contract), velocities and spins apart where their
units differ."""
import numpy as np
import pytest

import oracle
from cufcm_fil_b200 import RpyMobilitySolver

from .test_gpu_rpy_sets import TOL, particles

pytestmark = pytest.mark.gpu


def product(xs, fs, xb, fb, **kw):
    w = lambda a: a.astype(np.float64)
    blobs = (xb, fb) if len(xb) else ()
    with RpyMobilitySolver(len(xs), len(xb), **kw) as mob:
        vs, vb = mob.apply(xs, fs, *blobs)
    vs64, vb64 = oracle.mobility_full(w(xs), w(fs), *map(w, blobs), **kw)
    return np.asarray(vs).reshape(-1, 6), vb, vs64.reshape(-1, 6), vb64


@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("dof,n_seg,n_blob", [(3, 1300, 0), (3, 1290, 20), (6, 1041, 0), (6, 520, 20)])
def test_far_places_are_not_special(cuda, dof, n_seg, n_blob, wall):
    xs, fs, xb, fb = particles(n_seg, n_blob, dof, wall, seed=5)
    for k, y in enumerate((0.0, 1e5, 2e5)):
        for lane in (0, 5, 20, 31):
            xs[32 * k + lane] = (1e5 * (lane + 1), y, 1e4)
    for lane in (3, 17):  # where a particle's own place in the tile used to be taken by an inert one
        xs[320 + lane, 0] = -1e5 * (lane + 1)
    vs, vb, vs64, vb64 = product(xs, fs, xb, fb, wall=wall, seg_dof=dof)
    assert oracle.rel_l2(vs, vs64) <= TOL
    if n_blob:
        assert oracle.rel_l2(vb, vb64) <= TOL


@pytest.mark.parametrize("a", [1e-9, 1e-8, 1e-6, 1.0, 1e4])
@pytest.mark.parametrize("n_seg,n_blob", [(600, 0), (500, 70)])
def test_sets_with_torques_in_other_units(cuda, n_seg, n_blob, a):
    xs, fs, xb, fb = particles(n_seg, n_blob, 6, False, seed=9)
    xs, xb = (xs * a).astype(np.float32), (xb * a).astype(np.float32)
    fs[:, 3:] *= np.float32(a)  # torques in units of force times radius
    kw = dict(wall=False, seg_dof=6, seg_radius=a, blob_radius=a, mu=1e-3)
    vs, vb, vs64, vb64 = product(xs, fs, xb, fb, **kw)
    assert oracle.rel_l2(vs[:, :3], vs64[:, :3]) <= TOL
    assert oracle.rel_l2(vs[:, 3:], vs64[:, 3:]) <= TOL
    if n_blob:
        assert oracle.rel_l2(vb, vb64) <= TOL
