"""GPU: the exact free-surface detection of the FP32 form reads same-kind kernel gradients of the
lists' accuracy, whether or not a step kernel reads those lists too."""
import numpy as np
import pytest

import cases
import orc
import sps_gb300
from sps_gb300 import _abi
from sps_gb300.context import set_surface_detection

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [[1], [1, 1, 1]], ids=["rebuilt", "in_step"])
def test_exact_detection_does_not_depend_on_the_list_readers(built_gpu, chunks):
    # two runs that differ in nothing but who reads the same-kind lists: a viscosity factor of
    # 1e-300, zero in the FP32 sums, makes the steps' kernels read them.  A neighbour u of a
    # surface particle t is lifted past the point where t counts as inside (bisected with the
    # oracle), in steps of 1e-8 dx: the decision is one of gradients' last bits.
    def make(alpha):
        return cases.bui_like(width=1.0, height=0.5, dx=0.05, sle=2, xsph=False, alpha=alpha,
                              beta=0.0, dt=1e-12)

    probs = [make(0.0), make(1e-300)]
    p = probs[0]
    nn, nt, s = p.nnode, p.ntotal, p.state()
    x = s["x"].reshape(-1, 2)
    top = np.flatnonzero(x[:nn, 1] > x[:nn, 1].max() - 1e-6)
    x[:nt] += np.random.default_rng(11).uniform(-1e-3, 1e-3, (nt, 2))
    top = top[np.argsort(x[top, 0])]
    ref = orc.context(p.params_copy())
    gpu = [sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                 q.params_copy(precision=_abi.SPS_PREC_FP32_FAST)) for q in probs]
    for c in gpu:
        set_surface_detection(c, True)

    def subset(c, u, lift):
        y = x.copy()
        y[u, 1] += lift
        c.upload(**dict(s, x=y.ravel()))
        c.upload_bcs(p.bc_or_not, p.bc_info)
        for n in chunks:
            c.step(n, 0.0)
            c.download()
        return c.download_surface()[1]

    for k in (3, 5, 9, 13):
        t, u = top[k], top[k + 1]
        lo, hi = 0.0, 0.06
        assert subset(ref, u, lo)[t] == 1 and subset(ref, u, hi)[t] == 2
        while lo < 0.5 * (lo + hi) < hi:
            m = 0.5 * (lo + hi)
            lo, hi = (m, hi) if subset(ref, u, m)[t] == 1 else (lo, m)
        for lift in lo + np.linspace(-3e-8, 3e-8, 121):
            a, b = (subset(c, u, lift) for c in gpu)
            np.testing.assert_array_equal(a, b, err_msg="%d %r" % (k, lift))
    for c in gpu:
        c.close()


def test_fp32_detection_does_not_depend_on_the_list_readers(built_gpu):
    # the same of the FP32 detection, where the lists are in walk order (sle 2): the threshold is
    # its own, within a few 1e-7 dx of the oracle's
    def make(alpha):
        return cases.bui_like(width=1.0, height=0.5, dx=0.05, sle=2, xsph=False, alpha=alpha,
                              beta=0.0, dt=1e-12)

    probs = [make(0.0), make(1e-300)]
    p = probs[0]
    nn, nt, s = p.nnode, p.ntotal, p.state()
    x = s["x"].reshape(-1, 2)
    top = np.flatnonzero(x[:nn, 1] > x[:nn, 1].max() - 1e-6)
    x[:nt] += np.random.default_rng(11).uniform(-1e-3, 1e-3, (nt, 2))
    top = top[np.argsort(x[top, 0])]
    gpu = [sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps",
                                 q.params_copy(precision=_abi.SPS_PREC_FP32_FAST)) for q in probs]

    def subset(c, u, lift):
        y = x.copy()
        y[u, 1] += lift
        c.upload(**dict(s, x=y.ravel()))
        c.upload_bcs(p.bc_or_not, p.bc_info)
        c.step(1, 0.0)
        c.download()
        return c.download_surface()

    for k in range(3, 15):
        t, u = top[k], top[k + 1]
        lo, hi = 0.0, 0.06
        while lo < 0.5 * (lo + hi) < hi:  # the second run's threshold
            m = 0.5 * (lo + hi)
            # (both runs: the order of the sums depends on the largest pair count so far)
            f = [subset(c, u, m)[1][t] for c in gpu]
            lo, hi = (m, hi) if f[1] == 1 else (lo, m)
        for lift in lo + np.linspace(-3e-8, 3e-8, 61):
            (na, a), (nb, b) = (subset(c, u, lift) for c in gpu)
            np.testing.assert_array_equal(a, b, err_msg="%d %r" % (k, lift))
            np.testing.assert_array_equal(na.view(np.int64), nb.view(np.int64))
    for c in gpu:
        c.close()
