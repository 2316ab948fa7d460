"""The symmetric product of force-only sets in its two kinds of work units (csrc/rpy_kernels.cuh, rpy_sym_packed): pairs of
tiles for launches too small to fill the SMs, packed units above.  Against the FP64 oracle around the sizes of tiles and of
the rule (1,952 particles), tolerance 1e-5 relative L2; and bit for bit the same: an array of a batch that takes packed
units against its own run, which takes pairs."""
import numpy as np
import pytest

import oracle
from cufcm_fil_b200 import RpyMobilitySolver, _lib
from cufcm_fil_b200.sim import WallCiliaBatch

from .test_gpu_batch import SHARED, array_spec, run_single
from .test_gpu_rpy_sets import TOL, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wall", [True, False])
@pytest.mark.parametrize("dof,n_seg,n_blob", [(3, 1, 33), (3, 32, 64), (3, 65, 2), (3, 1000, 31), (6, 20, 1281), (3, 1300, 652),
                                              (3, 1952, 1), (3, 1953, 95)])
def test_evaluations(cuda, dof, n_seg, n_blob, wall):
    xs, fs, xb, fb = particles(n_seg, n_blob, dof, wall, 21)
    w = lambda a: a.astype(np.float64)
    with RpyMobilitySolver(n_seg, n_blob, wall=wall, seg_dof=dof) as mob:
        mob.x_segs_host[:], mob.f_segs_host[:] = xs.ravel(), fs.ravel()
        mob.x_blobs_host[:], mob.f_blobs_host[:] = xb.ravel(), fb.ravel()
        for what in ("segment", "blob"):
            getattr(mob, f"copy_{what}_positions_to_device")()
            getattr(mob, f"copy_{what}_forces_to_device")()

        def results():
            mob.copy_segment_velocities_to_host()
            mob.copy_blob_velocities_to_host()
            return mob.v_segs_host.copy(), mob.v_blobs_host.copy()

        mob.evaluate_segment_segment_mobility()
        mob.evaluate_blob_blob_mobility()
        vs, vb = results()
        mob.evaluate_full_mobility()
        full = results()
    vs64, _ = oracle.mobility_full(w(xs), w(fs), wall=wall, seg_dof=dof)
    vb64, _ = oracle.mobility_full(w(xb), np.concatenate([w(fb), np.zeros((n_blob, 3))], 1), wall=wall, seg_dof=3)
    assert oracle.rel_l2(vs, vs64) <= TOL
    assert oracle.rel_l2(vb.reshape(-1, 3), vb64.reshape(-1, 6)[:, :3]) <= TOL
    for v, v64 in zip(full, oracle.mobility_full(w(xs), w(fs), w(xb), w(fb), wall=wall, seg_dof=dof)):
        assert oracle.rel_l2(v, v64) <= TOL


def test_batch_of_packed_units_matches_runs_of_pairs():
    # 20 segments a filament: 40, 39, 3 and 1 tiles (odd and even), partly filled; 3,900 pairs of tiles in all
    specs = [array_spec(n, 12.0, seed) for seed, n in enumerate((64, 63, 61, 64, 4, 1, 62))]
    single = [run_single(sp, 2) for sp in specs]
    with WallCiliaBatch(specs, **SHARED) as batch:
        for nt in range(2):
            it, _, rc = batch.step(nt)
            assert rc == _lib.CF_OK
            st = batch.state()
            for b in range(len(specs)):
                assert it[b] == single[b][0][nt]
                for key in ("phase", "angle", "phase_dot", "angle_dot"):
                    np.testing.assert_array_equal(st[b][key], single[b][1][nt][key])
