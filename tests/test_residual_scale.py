"""Residual scaling (sfd_residual_scale) needs a few values of the model, not
its arrays: its result after every new model, from several threads, and the
host memory it may touch."""
import dataclasses
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from tests._cases import engine_config, make_case


def _want(cfg, par, rec, res):
    """The scaling in the engine's precisions, from the host's parameters."""
    dh, dt = np.float32(cfg["dh"]), np.float32(cfg["dt"])
    shape = [cfg["nx"]] + ([cfg["ny"]] if cfg["nd"] == 3 else []) + [cfg["nz"]]
    out = {}
    for n, r in res.items():
        x = (rec[:, 0] / dh).astype(np.int64)
        if n == "p":
            at = [x] + [(rec[:, 1] / dh).astype(np.int64)] * (cfg["nd"] == 3) + [(rec[:, 2] / dh).astype(np.int64)]
        else:
            at = [x] * len(shape)
        pos = at[0]
        for a, m in zip(at[1:], shape[1:]):
            pos = pos * m + a
        if n == "p":
            d = (par["M"].ravel()[pos] - par["mu"].ravel()[pos]).astype(np.float64)
            s = (-2.0 * d * dh / dt).astype(np.float32)
            f = (s * dt)[:, None]
            out[n] = (r * f).astype(np.float32)
        else:
            s = (1.0 / par["r%sp" % {"vx": "i", "vy": "j", "vz": "k"}[n]].ravel()[pos].astype(np.float64) * dh / dt).astype(np.float32)
            out[n] = (r * (1.0 / s.astype(np.float64) * dt)[:, None]).astype(np.float32)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kw,how", [
    (dict(nd=2, nz=62, nx=57), {}),
    (dict(nd=3, nz=38, ny=40, nx=41, L=1), {}),
    (dict(nd=3, nz=36, ny=40, nx=41), dict(field_precision="fp16")),
    (dict(nd=2, nz=60, nx=64, fdorder=6), dict(kernels="general")),
])
def test_scaling_after_each_model(kw, how, cuda_device):
    from seiscl_b200 import engine

    cfg, model, acq = make_case(nt=40, nab=6, **kw)
    c = dataclasses.replace(engine_config(cfg), **how)
    p = engine.Plan(c)
    outs = ["vx", "vz", "p"] + ["vy"] * (kw["nd"] == 3)
    rng = np.random.default_rng(3)
    for scale in (1.0, 1.1):
        m = [model[k] if k != "rho" or model[k] is None else model[k] * np.float32(scale) for k in ("vp", "vs", "rho", "taup", "taus")]
        p.set_model(*m)
        par = engine.host_transform(c, *m)
        res = {n: rng.standard_normal((len(acq["rec_pos"]), 40)).astype(np.float32) for n in outs}
        want = _want(cfg, par, acq["rec_pos"], res)
        with ThreadPoolExecutor(4) as pool:   # the same plan from several threads
            for got in pool.map(lambda _: p.residual_scale(acq["rec_pos"], res), range(8)):
                for n in outs:
                    # the row factor is rounded once, the product once more
                    assert np.abs(got[n] - want[n]).max() <= 2.0 ** -22 * np.abs(want[n]).max(), n
    far = acq["rec_pos"].copy()
    far[1, 0] = 1e7
    with pytest.raises(engine.SeisCLEngineError, match="outside the model"):
        p.residual_scale(far, res)


def _resident():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


@pytest.mark.gpu
def test_scaling_copies_no_whole_arrays(cuda_device):
    from seiscl_b200.engine import Plan

    # 120 MB a parameter
    cfg, model, acq = make_case(nd=2, nz=5000, nx=6000, nt=4, nab=8)
    p = Plan(engine_config(cfg))
    p.set_model(model["vp"], model["vs"], model["rho"])
    res = {n: np.ones((len(acq["rec_pos"]), 4), np.float32) for n in ("vx", "vz", "p")}
    before = _resident()
    p.residual_scale(acq["rec_pos"], res)
    assert _resident() - before < 60e6   # half of one array
