"""Residual of the line patches' inverses: the preconditioner applied to A_pp x gives x back, A_pp being the oracle's FP64
block of the same patch, so what is left over is the device inverse's own error (FP32 assembly and elimination, its
64 x 64 pivot blocks by Gauss-Jordan with one Newton step).  Bound: sixteen FP32 roundings (1e-6) times the largest
condition number of the patches."""
from pathlib import Path

import numpy as np
import pytest

from oracle import implicit
from cufcm_fil_b200 import _lib, workloads
from cufcm_fil_b200.sim import WallCiliaSimulation

from .test_gpu_precond import GOLD, rel

pytestmark = pytest.mark.gpu

S_TABLE = np.load(Path(__file__).resolve().parent / "golden" / "ref_tips_16x16_80a.npz")["s_table"]


@pytest.mark.parametrize("spacing", [80.0, 20.0])
@pytest.mark.parametrize("n_fil,nx,line", [(24, 4, 4), (32, 2, 16), (18, 2, 9), (3, 1, 1)])
def test_inverse_times_block(n_fil, nx, line, spacing):
    bases = workloads.lattice_bases(n_fil, nx, spacing, 1.3)
    rng = np.random.default_rng(7)
    args = dict(nseg=20, seg_sep=2.6, dt=1 / 300, phase0=rng.uniform(0, 2 * np.pi, n_fil),
                angle0=rng.normal(0, 0.05, n_fil), spring_factor=0.01, phase_refs=GOLD["fb_phase"],
                angle_refs=GOLD["fb_angle"], s_table=S_TABLE)
    cpu = implicit.WallCilia(bases=bases, shape_sequence=1, **args)
    with WallCiliaSimulation(bases=bases, precond=_lib.CF_PRECOND_LINE, line_patch=line, **args) as gpu:
        gpu.initial_guess(0)
        cpu.initial_guess(0)
        x = rng.standard_normal(gpu.size)
        v = np.zeros_like(x)
        cond = 1.0
        for fils in implicit.line_patches(cpu.bases, line):
            rows, block = cpu.patch_rows(fils), cpu.patch_block(fils)
            v[rows] = block @ x[rows]
            cond = max(cond, np.linalg.cond(block))
        err = rel(gpu.apply_preconditioner_new(v), x)
    print(f"{n_fil} filaments in lines of {line}, {spacing}a apart: {err:.1e}, condition number {cond:.0f}")
    assert err <= 1e-6 * cond
