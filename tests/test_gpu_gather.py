"""GPU: the lists gathered straight from the cell stencil (neighbours.cu) at both sides of each
size where the number of lanes a target changes (16,000, 100,000 and 400,000 targets), with and
without same-kind lists, on jittered positions (every pair at its own distance).

Plain form: a step and the free-surface detection after it equal the CPU oracle's bit for bit,
which needs every list entry, its kernel value and gradient, and the order of each list.  FP32
form: the kernel values are FP32 and the sums compensated (relative 2^-24 a term), so that a
step's change agrees to a few 1e-7; 1e-5 as in the other comparisons of that form."""
import numpy as np
import pytest

import cases
import orc
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu

OPTIONS = dict(xsph=True, alpha=0.1, beta=0.1)  # the steps that read same-kind lists
# spacing, options, number of targets at least / at most
SIZES = {
    "column": (lambda **o: sps_gb300.Problem.column(dx=0.0043, **o), 0, 16000),
    "eight": (lambda **o: sps_gb300.Problem.slope(dx=0.15, **o), 10000, 16000),
    "four": (lambda **o: sps_gb300.Problem.slope(dx=0.125, **o), 16001, 30000),
    "four_most": (lambda **o: sps_gb300.Problem.slope(dx=0.055, **o), 80000, 100000),
    "two": (lambda **o: sps_gb300.Problem.slope(dx=0.05, **o), 100001, 130000),
    "one": (lambda **o: sps_gb300.Problem.slope(dx=0.026, **o), 400001, 500000),
}


def upload(p, contexts, seed=3):
    s = p.state()
    rng = np.random.default_rng(seed)
    x = np.array(s["x"], dtype=np.float64)
    n = p.ntotal
    jitter = rng.uniform(-1.0, 1.0, 2 * n) * 0.02 * np.repeat(s["hsml"][:n], 2)
    x[:2 * n] += jitter
    for c in contexts:
        c.upload(**dict(s, x=x))
        c.upload_bcs(p.bc_or_not, p.bc_info)


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("name", sorted(SIZES))
def test_gathered_lists_equal_oracle(built_gpu, name, same):
    make, least, most = SIZES[name]
    p = make(**(OPTIONS if same else {}))
    assert least <= p.ntotal <= most
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP64_PLAIN))
    ref = orc.context(p.params_copy())
    upload(p, [gpu, ref])
    assert gpu.step(1, 0.0) == ref.step(1, 0.0)
    a, b = gpu.download(), ref.download()
    cases.assert_bitwise(a, b, p.ntotal)
    np.testing.assert_array_equal(a["bc_or_not"], b["bc_or_not"])
    (ng, sg), (nr, sr) = gpu.download_surface(), ref.download_surface()
    np.testing.assert_array_equal(sg, sr)
    np.testing.assert_array_equal(ng.view(np.int64), nr.view(np.int64))
    gpu.close()


@pytest.mark.parametrize("name", ["eight", "four", "two", "one"])
def test_gathered_lists_fp32(built_gpu, name):
    p = SIZES[name][0]()
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                p.params_copy(precision=_abi.SPS_PREC_FP32_FAST))
    ref = orc.context(p.params_copy())
    upload(p, [gpu, ref])
    gpu.step(1, 0.0)
    ref.step(1, 0.0)
    a, b = gpu.download(), ref.download()
    for k, n in (("x", 2 * p.ntotal), ("vel", 2 * p.ntotal), ("stress", 4 * p.ntotal)):
        u, v = a[k][:n], b[k][:n]
        assert np.linalg.norm(u - v) <= 1e-5 * np.linalg.norm(v), k
    gpu.close()


def test_batch_of_unequal_problems(built_gpu):
    # realisations of 2,000 to 140,000 particles, so that the bounding boxes' stretches of
    # consecutive particles (64 and more a warp at this total) lie in one realisation or
    # span two; each equals its own run bit for bit
    probs = [sps_gb300.Problem.slope(dx=0.045), sps_gb300.Problem.column(dx=0.0043),
             sps_gb300.Problem.slope(dx=0.046), sps_gb300.Problem.column(dx=0.004),
             sps_gb300.Problem.slope(dx=0.05)]
    assert sum(p.ntotal for p in probs) > 320000
    batch = sps_gb300.Batch(probs, precision=_abi.SPS_PREC_FP64_PLAIN)
    batch.upload_all()
    batch.step(2)
    for r, p in enumerate(probs):
        one = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                    p.params_copy(precision=_abi.SPS_PREC_FP64_PLAIN))
        one.upload_problem(p)
        one.step(2, 0.0)
        cases.assert_bitwise(batch.download(r), one.download(), p.ntotal)
        one.close()
    batch.close()
