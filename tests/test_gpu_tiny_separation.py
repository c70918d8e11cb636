"""GPU: pairs whose separation has a component of 1e-47 to 1e-31, down to where FP32 holds no low
part of it (2^-149) and no part at all: the plain form's stored kernel values, formed in
double-float arithmetic with a rounding certificate, equal the CPU oracle's FP64 evaluation
rounded to FP32, bit for bit."""
import numpy as np
import pytest

import cases
import orc
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1])
def test_pairs_on_one_line(built_gpu, axis):
    # h = 4.8e-4, so that the gradient's factor (1e12) lifts such a component to ordinary floats
    p = cases.bui_like(width=0.008, height=0.004, dx=4e-4, floor_to=0.01, dt=1e-7, xsph=False,
                       alpha=0.0, beta=0.0)
    s, nt = p.state(), p.ntotal
    x = s["x"].reshape(-1, 2)
    line = np.unique(np.round(x[:nt, axis], 9))
    x[:, axis] -= line[len(line) // 2]
    on = np.flatnonzero(np.abs(x[:nt, axis]) < 1e-8)
    assert len(on) >= 10
    rng = np.random.default_rng(7)
    x[on, axis] = rng.choice([-1.0, 1.0], len(on)) * 10.0 ** rng.uniform(-47, -31, len(on))
    x[on[::5], axis] = 0.0
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP64_PLAIN))
    ref = orc.context(p.params_copy())
    for c in (gpu, ref):
        c.upload(**s)
        c.upload_bcs(p.bc_or_not, p.bc_info)
        c.step(1, 0.0)
    a, b = gpu.dump_pairs(), ref.dump_pairs()
    for k in ("pair_i", "pair_j"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for k in ("w", "dwdx", "dwdy"):
        np.testing.assert_array_equal(a[k].view(np.int32), b[k].view(np.int32), err_msg=k)
    cases.assert_bitwise(gpu.download(), ref.download(), nt)
    gpu.close()
