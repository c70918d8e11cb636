"""GPU: the autotuner times the L2 prefetch only where a kernel takes it, and leaves the flags as
they were where none does."""
import pytest

import cases
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu


def test_autotune_leaves_a_prefetch_that_nothing_reads(built_gpu):
    p = cases.bui_like()
    ctx = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP32_FAST))
    sps_gb300.set_prefetch(ctx, True, False)
    ctx.upload_problem(p)
    sps_gb300.autotune(ctx, 2)
    assert sps_gb300.prefetch(ctx) == {"interp": True, "derivs": False}
    la = sps_gb300.lookahead(ctx)
    assert (la["interp"], la["derivs"]) in ((2, 1), (2, 2), (4, 2), (8, 4))
    ctx.close()
