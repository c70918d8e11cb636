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


@pytest.mark.parametrize("precision,slot,most", [(_abi.SPS_PREC_FP64_PLAIN, 56, 1230),
                                                 (_abi.SPS_PREC_FP32_FAST, 64, 1230)],
                         ids=["plain", "fp32"])
def test_list_constants_take_no_slots_of_their_own(built_gpu, precision, slot, most):
    # 16 bytes a slot for each of the half, cross and same-kind lists, 8 for their keys, 8 for the
    # FP32 form's compact entries; the list constants share the half lists' place
    create, upload, n = used(precision)
    assert upload <= n * (slot * SLOTS + 32) + (32 << 20), upload / n
    assert create <= n * most + (32 << 20), create / n


@pytest.mark.parametrize("max_neighbours", [0, 400], ids=["gathered", "from_half_lists"])
def test_pairs_and_detection_after_steps(built_gpu, max_neighbours):
    # with 200 slots a list does not fit the gather's shared memory, so the step builds the
    # half lists, which its constants overwrite: the pairs and the detection's lists are
    # rebuilt from the step's own positions, every step anew
    import numpy as np

    import cases
    import orc

    p = cases.bui_like(width=1.0, height=0.5, dx=0.05, dt=5e-5, xsph=False, alpha=0.0, beta=0.0)
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP64_PLAIN,
                                              max_neighbours=max_neighbours))
    fast = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                 p.params_copy(precision=_abi.SPS_PREC_FP32_FAST,
                                               max_neighbours=max_neighbours))
    ref = orc.context(p.params_copy())
    for c in (gpu, fast, ref):
        c.upload_problem(p)
    for n in (1, 1, 4, 1):
        for c in (gpu, fast, ref):
            c.step(n, 0.0)
        a, b, f = gpu.dump_pairs(), ref.dump_pairs(), fast.dump_pairs()
        for k in ("pair_i", "pair_j"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
            np.testing.assert_array_equal(np.sort(f[k]), np.sort(b[k]), err_msg=k)
        for k in ("w", "dwdx", "dwdy"):
            np.testing.assert_array_equal(a[k].view(np.int32), b[k].view(np.int32), err_msg=k)
        x, y = gpu.download(), ref.download()
        cases.assert_bitwise(x, y, p.ntotal)
        np.testing.assert_array_equal(x["bc_or_not"], y["bc_or_not"])
        assert (fast.download()["bc_or_not"] == y["bc_or_not"]).mean() > 0.99
        (na, sa), (nb, sb) = gpu.download_surface(), ref.download_surface()
        np.testing.assert_array_equal(sa, sb)
        np.testing.assert_array_equal(na.view(np.int64), nb.view(np.int64))
    for c in (gpu, fast):
        c.close()


def test_a_batch_takes_its_cells_once(built_gpu):
    # 64 uploads one after the other: the cells' arrays (40 bytes a cell, four times the cells of
    # the uploaded realisations) grow by doubling, so what they left behind is no more than what
    # they are
    torch = pytest.importorskip("torch")
    probs = [sps_gb300.Problem.column(dx=0.004 + 1e-5 * i) for i in range(64)]
    torch.zeros(1, device="cuda")
    b = sps_gb300.Batch(probs, precision=_abi.SPS_PREC_FP32_FAST)
    torch.cuda.synchronize()
    a = torch.cuda.mem_get_info()[0]
    b.upload_all()
    torch.cuda.synchronize()
    took = a - torch.cuda.mem_get_info()[0]
    n = sum(len(p.mass) for p in probs)
    b.close()
    assert took <= n * 64 * SLOTS + (32 << 20), took / n


@pytest.mark.parametrize("precision", [_abi.SPS_PREC_FP64_PLAIN, _abi.SPS_PREC_FP32_FAST],
                         ids=["plain", "fp32"])
def test_a_context_has_one_form_of_stages(built_gpu, precision):
    # its arrays come to 700 bytes a particle (plain) and 760 (FP32) where a stage is one
    # launch; the separate kernels' would be 184 more
    create, _, n = used(precision)
    assert create <= n * 850 + (32 << 20), create / n
