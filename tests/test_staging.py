"""What a call allocates beside the plan's arrays (sfd_set_model,
sfd_get_gradient) makes do with less where the plan fills the device: with
failed allocations, counted on the host, the same bits."""
import dataclasses

import numpy as np
import pytest

from tests._cases import engine_config, make_case

CASES = [
    dict(nd=3, nz=38, ny=30, nx=90, L=1),
    dict(nd=3, nz=40, ny=30, nx=34, fdorder=4, freesurf=0),
    dict(nd=2, nz=62, nx=700),
]


def _run(p, acq):
    outs = ["vx", "vz"]
    d = p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], outs, save_boundaries=True)
    p.zero_gradient()
    p.adjoint(acq["src_pos"], acq["src"], acq["rec_pos"], d)
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["fp32", "fp16"])
@pytest.mark.parametrize("fails", [1, 3, 40])
@pytest.mark.parametrize("kw", CASES, ids=lambda k: "%dD-%d" % (k["nd"], k["nz"]))
def test_model_and_gradient_with_little_room(kw, fails, fields, cuda_device):
    """One or three failures halve the staging or use up its sizes; then, as
    with 40, a new model goes through the plan's own fields, and a gradient is
    refused."""
    from seiscl_b200.engine import Plan, SeisCLEngineError

    cfg, model, acq = make_case(nt=40, nab=8, **kw)
    how = dict(field_precision=fields, checkpoint=13) if fields == "fp16" else {}
    args = [model[k] for k in ("vp", "vs", "rho", "taup", "taus")]
    got = []
    for n in (0, fails):
        p = Plan(dataclasses.replace(engine_config(cfg), **how))
        if 0 < n < 40 and kw["nx"] == 90:   # room to halve
            p.debug_launch(16 + n)
        p.set_model(*args)
        _run(p, acq)
        if n:
            p.debug_launch(16 + n)
        p.set_model(args[0], args[1], args[2] * np.float32(1.01), *args[3:])
        p.debug_launch(16)
        out = {"p%d" % i: p.debug_array(3, i, model["vp"].size) for i in (0, 1, 5, 7, 8)}
        out.update(_run(p, acq))
        if n:
            p.debug_launch(16 + (40 if n == 40 else 1))
            if n == 40:
                with pytest.raises(SeisCLEngineError, match="staging"):
                    p.gradient()
                p.debug_launch(16)
        out.update(p.gradient())
        got.append(out)
        p.close()
    for k in got[0]:
        assert np.abs(got[0][k]).max() > 0 and np.array_equal(got[0][k], got[1][k]), k


@pytest.mark.gpu
def test_refused_model_through_borrowed_fields(cuda_device):
    """A model staged over the wave fields and then refused leaves no state
    an adjoint could start from; the old model stays."""
    from seiscl_b200.engine import Plan, SeisCLEngineError

    cfg, model, acq = make_case(nd=2, nz=62, nx=700, nt=40, nab=8)
    p = Plan(engine_config(cfg))
    p.set_model(model["vp"], model["vs"], model["rho"])
    d = _run(p, acq)
    p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx", "vz"], save_boundaries=True)
    p.debug_launch(16 + 40)
    with pytest.raises(SeisCLEngineError):
        p.set_model(model["vp"] * 9, model["vs"], model["rho"])
    p.debug_launch(16)
    with pytest.raises(SeisCLEngineError, match="preceding"):
        p.adjoint(acq["src_pos"], acq["src"], acq["rec_pos"], d)
    again = _run(p, acq)
    assert all(np.array_equal(again[k], d[k]) for k in d)
