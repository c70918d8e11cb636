"""GPU: the outside approach's re-interpolation at the start of a step (SPH_shift, every
shift_update steps) in steps whose pair build moves particles between cells or meets more pairs
than any step before: its sums have to walk the lists of that step."""
import numpy as np
import pytest

import cases
import orc
import sps_gb300
from sps_gb300 import _abi

pytestmark = pytest.mark.gpu

OUTSIDE = dict(sph_shift=True, vel_vector=False, shift_update=2, rx=1 / 3, ry=1 / 3,
               disp_tol=0.125)


def pair(p, state, precision):
    """A GPU context and the oracle, both with this state."""
    gpu = sps_gb300.StepContext(sps_gb300.gpu_lib(), "sps", p.params_copy(precision=precision))
    ref = orc.context(p.params_copy())
    for c in (gpu, ref):
        c.upload(**state)
        c.upload_bcs(p.bc_or_not, p.bc_info)
    return gpu, ref


def test_reinterpolation_with_moving_particles_fp32(built_gpu):
    # an elastic block pushed against its wall at up to 3 m/s: the particles' order by cell
    # changes between most steps, and the pair count passes its maximum in the
    # re-interpolating steps 5 and 7
    p = cases.bui_like(width=1.0, height=0.5, dx=0.05, outside=OUTSIDE, npoints=2, dt=6e-4, coh=1e9)
    nt, nsteps = p.ntotal, 8
    s = p.state()
    x, v = s["x"].reshape(-1, 2)[:nt], s["vel"].reshape(-1, 2)[:nt]
    v[:, 0] = 1.0 - 4.0 * (x[:, 0] - 0.5)
    v[:, 1] = -3.0 * (x[:, 1] - 0.1) * np.sin(3.0 * x[:, 0])
    s["intvars1"][:nt] = 1e-3 * (1.0 + x[:, 0] * x[:, 1])
    x0 = x.copy()
    gpu, ref = pair(p, s, _abi.SPS_PREC_FP32_FAST)
    order, grew, moved, most = None, [], [], 0
    for it in range(1, nsteps + 1):
        ref.step(1, 0.0)
        d = ref.dump_pairs()
        # (the pairs in walk order; the particles in the order of their first pair)
        o = list(dict.fromkeys(np.minimum(d["pair_i"], d["pair_j"]).tolist()))
        if it % 2 == 1 and it > 1:
            grew.append(len(d["pair_i"]) > most)
            moved.append(o != order)
        order, most = o, max(most, len(d["pair_i"]))
    assert sum(grew) >= 2 and sum(moved) >= 3
    gpu.step(nsteps, 0.0)
    a, b = gpu.download(), ref.download()
    # a velocity is a compensated FP32 mean over FP32 records, relative 2^-24 a term, and its
    # rates carry a few 1e-7; 8 steps leave well below 1e-5 of the largest displacement,
    # velocity, stress and internal variable, in every particle
    da, db = a["x"][:2 * nt] - x0.ravel(), b["x"][:2 * nt] - x0.ravel()
    for k, u, w in (("displacement", da, db), ("vel", a["vel"][:2 * nt], b["vel"][:2 * nt]),
                    ("stress", a["stress"][:4 * nt], b["stress"][:4 * nt]),
                    ("intvars1", a["intvars1"][:nt], b["intvars1"][:nt])):
        assert np.abs(u - w).max() <= 1e-5 * np.abs(w).max(), (k, np.abs(u - w).max())
    gpu.close()


def test_reinterpolation_in_a_step_that_grows_the_list(built_gpu):
    # Plain form, bit for bit.  The stress-points start 1.5 times as far apart as their nodes;
    # the shift at the end of step 2 puts them at their nodes, so the re-interpolating step 3
    # meets 8% more pairs than any step before and takes the new ones first.  The nodes' large
    # velocities, antisymmetric about the diagonal, cancel in the sums of the stress-points on
    # it: what is left shows the order.  One of those lies at the origin, so that its position
    # shows the last bits of its velocity.
    dx = 0.05
    p = cases.bui_like(width=0.5, height=0.5, dx=dx, outside=OUTSIDE, npoints=1, dt=1e-13,
                       coh=1e9, alpha=0.0, beta=0.0, xsph=False)
    s, nn = p.state(), p.nnode
    x, v = s["x"].reshape(-1, 2), s["vel"].reshape(-1, 2)
    i, j = np.rint((x[:nn] - x[:nn].min(axis=0)) / dx).T
    x -= x[np.flatnonzero((i == 8) & (j == 8))[0]] + dx / 3
    x[nn:2 * nn] = 1.5 * (x[:nn] - x[:nn].mean(axis=0)) + x[:nn].mean(axis=0)
    v[:nn] = np.random.default_rng(5).uniform(0.5e-3, 1.5e-3, (nn, 2))
    v[:nn] += 1e8 * np.sign(i - j)[:, None] * [1.0, -1.0]
    v[nn:2 * nn] = v[:nn]
    gpu, ref = pair(p, s, _abi.SPS_PREC_FP64_PLAIN)
    n = []
    for _ in range(3):
        gpu.step(1, 0.0)
        ref.step(1, 0.0)
        n.append(len(ref.dump_pairs()["pair_i"]))
    assert n[2] > 1.05 * max(n[:2])
    cases.assert_bitwise(gpu.download(), ref.download(), p.ntotal)
    gpu.close()
