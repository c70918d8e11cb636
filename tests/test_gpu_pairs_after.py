"""GPU: sps_dump_pairs reports the last step's pairs also after calls that replace what their
rebuild reads: an upload of other smoothing lengths, which may move the list and cell capacities,
and the autotuner's steps, which also leave the free surface as it was."""
import numpy as np
import pytest

import cases
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu

FORMS = {"plain": _abi.SPS_PREC_FP64_PLAIN, "fp32": _abi.SPS_PREC_FP32_FAST}
# one-launch stages; separate kernels; separate kernels whose half lists cannot be built again
OPTIONS = {"fused": {}, "separate": dict(art_stress=True), "kept": dict(cont_density=True, sle=2)}


def _ctx(p, form):
    c = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps", p.params_copy(precision=FORMS[form]))
    c.upload_problem(p)
    return c


def _same(a, b):
    assert len(a["pair_i"]) > 0
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("option", OPTIONS)
@pytest.mark.parametrize("factors", [(1.25,), (0.8,), (1.0, 0.7, 1.3)])
def test_pairs_after_an_upload(built_gpu, form, option, factors):
    # 1.25 raises the list capacity (48 -> 65 entries), 0.8 the number of cells
    p = cases.bui_like(width=1.0, height=0.5, dx=0.05, **OPTIONS[option])
    ref, ctx = _ctx(p, form), _ctx(p, form)
    assert len(ctx.dump_pairs()["pair_i"]) == 0
    for c in (ref, ctx):
        c.step(3, 0.0)
    want = ref.dump_pairs()
    for f in factors:
        s = p.state()
        s["hsml"] *= f
        ctx.upload(**s)
    ctx.upload_bcs(p.bc_or_not, p.bc_info)
    _same(want, ctx.dump_pairs())
    # (the list of pairs carries over to the next step's order, as it does in the reference)
    ref.upload(**s)
    ref.upload_bcs(p.bc_or_not, p.bc_info)
    for c in (ref, ctx):
        c.step(2, 0.0)
    cases.assert_bitwise(ctx.download(), ref.download(), p.ntotal)
    _same(ref.dump_pairs(), ctx.dump_pairs())
    ref.close()
    ctx.close()


@pytest.mark.parametrize("form", FORMS)
def test_pairs_of_a_batch_after_one_upload(built_gpu, form):
    ps = [cases.bui_like(width=1.0, height=0.5, dx=0.05), cases.bui_like(width=0.8, height=0.6, dx=0.05)]
    ref, b = [sps_gb300.Batch(ps, precision=FORMS[form]) for _ in range(2)]
    for c in (ref, b):
        c.upload_all()
        c.step(3)
    s = ps[0].state()
    s["hsml"] *= 0.8
    fn = b._lib.sps_upload_real
    a = [s[k] for k in ("x", "vel", "stress", "mass", "rho", "hsml")]
    dp, ip = sps_gb300.context._dp, sps_gb300.context._ip
    assert fn(b._h, 0, *[dp(v) for v in a], ip(s["itype"]), dp(s["intvars1"]), dp(s["f_drucker"]),
              dp(s["x00"])) == 0
    for r in (0, 1):
        _same(ref.dump_pairs(r), b.dump_pairs(r))
    ref.close()
    b.close()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("option", OPTIONS)
@pytest.mark.parametrize("upload", [False, True])
def test_pairs_and_surface_after_tuning(built_gpu, form, option, upload):
    # the block falls apart at 20 m/s: the autotuner's steps meet other pairs than the last one
    p = cases.bui_like(width=1.0, height=0.5, dx=0.05, coh=1e9, dt=6e-4, **OPTIONS[option])
    s = p.state()
    x, v = s["x"].reshape(-1, 2), s["vel"].reshape(-1, 2)
    v[:p.ntotal] = 20.0 * (x[:p.ntotal] + 0.1)
    ref, ctx = _ctx(p, form), _ctx(p, form)
    for c in (ref, ctx):
        c.upload(**s)
        c.step(3, 0.0)
        if upload:
            s2 = p.state()
            s2["hsml"] *= 0.9
            c.upload(**s2)
    sps_gb300.autotune(ctx, 4)
    a, b = ctx.download(), ref.download()
    cases.assert_bitwise(a, b, p.ntotal)
    assert np.array_equal(a["bc_or_not"], b["bc_or_not"])
    for u, w in zip(ctx.download_surface(0), ref.download_surface(0)):
        assert np.array_equal(u, w, equal_nan=True)
    _same(ref.dump_pairs(), ctx.dump_pairs())
    ref.close()
    ctx.close()
