"""GPU tests of the flow-field kernel at the edges of its tiles (64 sources, 128 or 256 flow points a block), for every
number of source splits that its plan can choose there, and of host calls on both sides of the staging limit (4 MB),
against the FP64 oracle; tolerance 1e-5 relative L2, the mobility contract."""
import numpy as np
import pytest

import oracle
from oracle import flow as oflow
from cufcm_fil_b200.flow import FlowFieldEvaluator

pytestmark = pytest.mark.gpu
TOL = 1e-5


def check(n_seg, n_blob, nf, net, sample=None):
    rng = np.random.default_rng(n_seg + 3 * n_blob + nf)
    f32 = lambda a: np.asarray(a, np.float32).astype(np.float64)
    box = lambda n: f32(rng.uniform([-40, -40, 1.5], [40, 40, 60], (n, 3)))
    xs, xb, xf, body = box(n_seg), box(n_blob), box(nf), box(1)
    xf[:, 2] -= 1.0
    xf = f32(xf)
    fs, fb = f32(rng.standard_normal((n_seg, 6))), f32(rng.standard_normal((n_blob, 3)))
    kw = dict(n_seg_per_body=max(n_seg, 1), n_blob_per_body=n_blob)
    blobs = dict(x_blobs=xb, f_blobs=fb) if n_blob else {}
    with FlowFieldEvaluator(nf, n_seg, n_blob, 1, remove_net_force=net) as ev:
        v = ev.velocities(xf, xs, fs, x_bodies=body, **blobs, **kw)
    ids = np.arange(nf) if sample is None else rng.permutation(nf)[:sample]
    want = oflow.flow_velocities(xf[ids], xs, fs, *((xb, fb) if n_blob else (None, None)), body, remove_net_force=net, **kw)
    assert oracle.rel_l2(np.asarray(v).reshape(-1, 3)[ids], want) <= TOL


@pytest.mark.parametrize("net", [False, True])
@pytest.mark.parametrize("n_seg,n_blob", [(1, 0), (63, 1), (64, 0), (65, 64), (700, 333)])
@pytest.mark.parametrize("nf", [1, 127, 129, 257])
def test_tile_edges(cuda, n_seg, n_blob, nf, net):
    check(n_seg, n_blob, nf, net)


@pytest.mark.parametrize("nf", [40000, 180000])
def test_many_points(cuda, nf):
    check(200, 40, nf, False, sample=300)
