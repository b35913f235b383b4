"""The chain rule from the accumulated (M, mu, rho) sums to the gradient of
the chosen parameters (sfd_get_gradient), against FP64 numpy on the raw sums.

Both sides are FP32 roundings of FP64 values: the raw sums lose 2^-24 of
each term, and the terms of the density gradient may partly cancel, so the
bound is 4 x 2^-24 of the sum of the absolute terms."""
import dataclasses

import numpy as np
import pytest

from tests._cases import engine_config, make_case


def _chain(raw, model, pt):
    """transf_grad in FP64: the gradient and the size of its terms."""
    vp, vs, rho = (model[k].astype(np.float64) for k in ("vp", "vs", "rho"))
    M, mu = vp ** 2 * rho, vs ** 2 * rho
    gM, gmu, gr = (raw[k].astype(np.float64) / np.float64(np.float32(1e-3)) for k in ("M", "mu", "rho"))
    if pt == 1:
        return [gM, gmu, gr], [abs(gM), abs(gmu), abs(gr)]
    f = (lambda m: 2 * np.sqrt(rho * m)) if pt == 0 else (lambda m: 2 * np.sqrt(m / rho))
    terms = [gr, M / rho * gM, mu / rho * gmu]
    return ([f(M) * gM, f(mu) * gmu, sum(terms)],
            [abs(f(M) * gM), abs(f(mu) * gmu), sum(abs(t) for t in terms)])


@pytest.mark.gpu
@pytest.mark.parametrize("kw,pt,batch", [
    (dict(nd=2, nz=38, nx=45, nt=60, freesurf=0, nab=8), 0, 1),
    (dict(nd=2, nz=38, nx=45, nt=60, freesurf=0, nab=8), 2, 3),
    (dict(nd=3, nz=30, ny=31, nx=33, nt=40, nab=6), 1, 1),
    # more cells than one staging chunk holds
    (dict(nd=2, nz=2306, nx=3701, nt=4, freesurf=0, nab=8), 0, 1),
])
def test_gradient_transform(kw, pt, batch, cuda_device):
    from seiscl_b200.engine import Plan

    cfg, model, acq = make_case(**kw)
    plan = Plan(dataclasses.replace(engine_config(cfg), param_type=pt, batch=batch))
    vp, vs, rho = (model[k].astype(np.float64) for k in ("vp", "vs", "rho"))
    given = {0: (vp, vs), 1: (vp ** 2 * rho, vs ** 2 * rho), 2: (vp * rho, vs * rho)}[pt]
    plan.set_model(*[p.astype(np.float32) for p in given], model["rho"])
    shots = [(acq["src_pos"], acq["src"] * (1 + b), acq["rec_pos"]) for b in range(batch)]
    outs = ["vx", "vz"]
    d = plan.forward_batch(shots, outs, save_boundaries=True)
    plan.zero_gradient()
    plan.adjoint_batch(shots, d)
    raw, got = plan.gradient(transform=False), plan.gradient()
    assert np.abs(raw["M"]).max() > 0
    want, size = _chain(raw, model, pt)
    for g, w, s in zip(got.values(), want, size):
        # M, mu and rho reach the device in FP32 as well: 2^-24 each, squared or rooted
        assert np.all(np.abs(g - w) <= 12 * 2.0 ** -24 * s + 1e-45)
