"""Material parameters prepared on the device (sfd_model.cu) against the host
transforms (sfd_host_transform), bit for bit: every physics, parametrisation
and a model of several slabs; models that are refused leave the old one."""
import dataclasses

import numpy as np
import pytest

from tests._cases import engine_config, make_case

CASES = [
    (dict(nd=2, nz=38, nx=45), 0, {}),
    (dict(nd=2, nz=42, nx=33, L=2), 1, {}),
    (dict(nd=2, nz=40, nx=31, L=1), 2, dict(kernels="general")),
    (dict(nd=3, nz=26, ny=24, nx=23, L=3), 0, {}),
    (dict(nd=3, nz=28, ny=25, nx=21), 2, dict(fdorder=4)),
    (dict(nd=2, nz=2306, nx=2411, L=1), 0, {}),       # two slabs
    (dict(nd=3, nz=1602, ny=1650, nx=3), 0, {}),      # slabs of two planes
    (dict(nd=21, nz=38, nx=45), 0, {}),               # SH
    (dict(nd=21, nz=40, nx=31), 2, {}),
    (dict(nd=22, nz=42, nx=33), 1, {}),               # acoustic
    (dict(nd=22, nz=42, nx=33, L=1), 0, {}),
]


def _given(model, pt):
    vp, vs, rho = (model[k].astype(np.float64) for k in ("vp", "vs", "rho"))
    a, b = {0: (vp, vs), 1: (vp ** 2 * rho, vs ** 2 * rho), 2: (vp * rho, vs * rho)}[pt]
    return [a.astype(np.float32), b.astype(np.float32), model["rho"], model["taup"], model["taus"]]


@pytest.mark.gpu
@pytest.mark.parametrize("kw,pt,how", CASES, ids=lambda v: str(v).replace(" ", "")[:40])
def test_parameters(kw, pt, how, cuda_device):
    from seiscl_b200 import engine

    cfg, model, _ = make_case(nt=5, nab=4, freesurf=0, fdorder=how.pop("fdorder", 8), **kw)
    c = dataclasses.replace(engine_config(cfg), param_type=pt, **how)
    given = _given(model, pt)
    given[1].flat[:cfg["nz"] * 2] = 0.0      # a fluid corner: harmonic means of zero
    want = engine.host_transform(c, *given)
    p = engine.Plan(c)
    p.set_model(*given)
    for i, n in enumerate(engine.PARAM_NAMES):
        got = p.debug_array(3, i, want[n].size)
        assert np.array_equal(got, want[n].ravel(), equal_nan=True), (n, np.nanmax(np.abs(got - want[n].ravel())))


@pytest.mark.gpu
def test_refused_models_leave_the_old_one(cuda_device):
    from seiscl_b200 import engine

    cfg, model, acq = make_case(nd=2, nz=40, nx=50, nt=60)
    p = engine.Plan(engine_config(cfg))
    p.set_model(model["vp"], model["vs"], model["rho"])
    want = p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx"])["vx"]
    rho = model["rho"].copy()
    rho[20, 20] = 0.0
    for bad, code in (([model["vp"], model["vs"], rho], -1), ([model["vp"] * 5, model["vs"], model["rho"]], -3),
                      ([model["vp"], model["vs"], rho * np.nan], -1)):
        with pytest.raises(engine.SeisCLEngineError) as e:
            p.set_model(*bad)
        assert e.value.code == code
    assert np.array_equal(p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx"])["vx"], want)
