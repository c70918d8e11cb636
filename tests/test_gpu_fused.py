"""GPU: the plain form's one-launch stages (plain_fused.cu) against the CPU oracle, bit for bit,
at the sizes where their split matters: fewer targets than a warp, a ragged last warp, a
target's sums shared by several lanes (small problems) and by one lane (large ones), with
the list constants of walls, CSPM moments, artificial viscosity, several stress-points a cell
and nodes without stress-points in reach."""
import numpy as np
import pytest

import cases
import orc
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu

CASES = {
    # 15 + 8 particles
    "tiny": (lambda: cases.bui_like(width=0.2, height=0.1, dx=0.05, dt=2e-5), 6),
    "ragged": (lambda: sps_gb300.Problem.column(dx=0.0043), 12),
    # h = 0.3 dx: no partner in reach, every interpolation keeps its cleared value
    "isolated": (lambda: cases.bui_like(width=1.0, height=0.5, dx=0.1, sml=0.3), 4),
    "cspm_viscosity": (lambda: cases.bui_like(width=1.0, height=0.5, dx=0.05, cspm=True,
                                              dt=5e-5), 8),
    "three_points": (lambda: cases.bui_like(width=1.0, height=0.5, dx=0.05, npoints=3,
                                            dt=5e-5), 8),
    "one_lane": (lambda: sps_gb300.Problem.slope(dx=0.066), 3),
    "one_lane_viscosity": (lambda: sps_gb300.Problem.slope(dx=0.066, xsph=True, alpha=0.1,
                                                           beta=0.1), 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fused_stages_equal_oracle(built_gpu, name):
    make, nsteps = CASES[name]
    p = make()
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP64_PLAIN))
    ref = orc.context(p.params_copy())
    tg, to = cases.run_pair(p, nsteps, [gpu, ref], chunks=[1, nsteps - 1])
    assert tg == to
    cases.assert_bitwise(gpu.download(), ref.download(), p.ntotal)
    gpu.close()


FAST = {
    "tiny": (lambda: cases.bui_like(width=0.2, height=0.1, dx=0.05, dt=2e-5), 6),
    "isolated": (lambda: cases.bui_like(width=1.0, height=0.5, dx=0.1, sml=0.3), 4),
    "cspm_viscosity": (lambda: cases.bui_like(width=1.0, height=0.5, dx=0.05, cspm=True,
                                              dt=5e-5), 6),
    "cspm_bcs": (lambda: cases.bc_case(), 6),
    "ragged": (lambda: cases.bui_like(width=1.15, height=0.45, dx=0.05, dt=5e-5), 6),
    "large": (lambda: sps_gb300.Problem.slope(dx=0.066), 3),
}


@pytest.mark.parametrize("name", sorted(FAST))
def test_fused_fp32_stages_against_oracle(built_gpu, name):
    # the FP32 form's one-launch stages against the oracle's FP64: each sum is compensated
    # FP32 over FP32 records (relative 2^-24 a term), so a step's rates carry a few 1e-7
    # relative; velocities start from zero and accumulate `nsteps` of those rates, stresses
    # change by dt times them
    make, nsteps = FAST[name]
    p = make()
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP32_FAST))
    ref = orc.context(p.params_copy())
    cases.run_pair(p, nsteps, [gpu, ref])
    a, b = gpu.download(), ref.download()
    for k, n in (("x", 2 * p.ntotal), ("vel", 2 * p.ntotal), ("stress", 4 * p.ntotal)):
        u, v = a[k][:n], b[k][:n]
        assert np.linalg.norm(u - v) <= 1e-5 * np.linalg.norm(v), k
    gpu.close()
