"""GPU: the device memory that a context takes."""
import pytest

import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu

SLOTS = 48  # a list's slots where max_neighbours is left to the library (h = 1.2 dx)


def used(make):
    """The bytes a context and its first upload take, and the particles."""
    torch = pytest.importorskip("torch")
    p = sps_gb300.Problem.slope(dx=0.02)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    torch.zeros(1, device="cuda")
    a = free()
    ctx = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps", p.params_copy(precision=make))
    b = free()
    ctx.upload_problem(p)
    c = free()
    ctx.close()
    return a - b, b - c, len(p.mass)


@pytest.mark.parametrize("precision", [_abi.SPS_PREC_FP64_PLAIN, _abi.SPS_PREC_FP32_FAST],
                         ids=["plain", "fp32"])
def test_an_upload_takes_its_lists_and_cells(built_gpu, precision):
    # 76 bytes a list slot and particle at most, 32 a cell of about 0.7 a particle, and 32 MB of
    # the allocator's own pages: not a second block of a context's size
    _, upload, n = used(precision)
    assert n > 700000
    assert upload <= n * (76 * SLOTS + 32) + (32 << 20), upload / n
