"""GPU: the plain form's one-launch stages (plain_fused.cu) against the CPU oracle, bit for bit,
at the sizes where their split matters: fewer targets than a warp, a ragged last warp, a
target's sums shared by several lanes (below 60,000 particles) and by one lane (above), with
the list constants of walls, CSPM moments, artificial viscosity, several stress-points a cell
and nodes without stress-points in reach."""
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
