"""Flow points next to a blob's centre or a body's (distances down to 1e-17, as between cos(pi/2) and 0) and very far from
them: the cube of such a distance leaves the range of FP32, the velocity does not.  Against the FP64 oracle, tolerance
1e-5 relative for each point."""
import numpy as np
import pytest

from oracle import flow as oflow
from cufcm_fil_b200.flow import FlowFieldEvaluator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("net", [False, True])
@pytest.mark.parametrize("r", [6.1e-17, 1e-14, 1e13])
def test_points_at_extreme_distances(cuda, r, net):
    f32 = lambda a: np.asarray(a, np.float32).astype(np.float64)
    rng = np.random.default_rng(4)
    d = np.array([[1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.6, -0.7, 0.0]])
    blobs = f32([[0.0, 0.0, 3.0]])
    body = f32([[0.0, 0.0, 2.0]])
    xf = f32(np.concatenate([d * r + [0, 0, 3], d * r + [0, 0, 2]]))
    fb = f32(rng.standard_normal((1, 3)))
    none = np.zeros((0, 3)), np.zeros((0, 6))
    kw = dict(n_seg_per_body=1, n_blob_per_body=1)
    with FlowFieldEvaluator(len(xf), 0, 1, 1, remove_net_force=net) as ev:
        v = np.asarray(ev.velocities(xf, *none, x_blobs=blobs, f_blobs=fb, x_bodies=body, **kw)).reshape(-1, 3)
    want = oflow.flow_velocities(xf, *none, blobs, fb, body, remove_net_force=net, **kw)
    if r > 1 and net:  # the Stokeslet at the body cancels the blob's
        assert np.abs(v).max() <= 1e-5 / r
    else:
        assert (np.linalg.norm(v - want, axis=1) <= 1e-5 * np.linalg.norm(want, axis=1)).all(), (v, want)
