"""The 4-cell 2D P-SV kernels (sfd_quad2d.cu) against the one-cell kernels
(kernels "general"), bit for bit: both use the cell arithmetic of
sfd_device.cuh.  A receiver in the padding keeps the runs off the resident
loop (sfd_resident2d.cu).  Rows with and without dummy cells, slab edges
inside quads, touching and overlapping slabs, tapers, batches, boundary
shells in every storage type, checkpoints, DFT and Hessian."""
import dataclasses

import numpy as np
import pytest

from tests._cases import engine_config, make_case

CASES = [
    dict(nz=60, nx=45, nt=80, nab=8, fdorder=8, L=0),
    dict(nz=62, nx=47, nt=80, nab=8, fdorder=4, L=1),
    dict(nz=58, nx=51, nt=80, nab=7, fdorder=8, L=2, freesurf=0),
    dict(nz=64, nx=39, nt=60, nab=6, fdorder=4, L=3, freesurf=0, src_type=2),
    dict(nz=34, nx=35, nt=60, nab=16, fdorder=4, L=0, freesurf=0),   # slabs nearly touching
    dict(nz=26, nx=29, nt=60, nab=16, fdorder=8, L=0, freesurf=0),   # overlapping
    dict(nz=50, nx=41, nt=60, nab=9, fdorder=8, L=1, abs_type=2, src_type=0),
    dict(nz=702, nx=23, nt=40, nab=4, fdorder=4, L=0),
]
IDS = ["%dx%d-o%d-L%d" % (k["nz"], k["nx"], k["fdorder"], k["L"]) for k in CASES]


def _case(kw):
    cfg, model, acq = make_case(nd=2, **kw)
    nz, nx = kw["nz"], kw["nx"]
    acq["src_pos"][0, [0, 2]] = [nx // 2 * 10.0, nz // 2 * 10.0]
    rec = np.zeros((2 * nx - 8, 8), np.float32)
    rec[:, 0] = np.tile(np.arange(2, nx - 2), 2) * 10.0
    rec[:, 2] = np.repeat([nz // 2 - 6, nz - 2], nx - 4) * 10.0
    rec[0, 2] = -20.0
    rec[:, 4] = np.arange(1, len(rec) + 1)
    acq["rec_pos"] = rec
    return cfg, model, acq


def _plans(cfg, model, **kw):
    from seiscl_b200.engine import Plan

    out = []
    for kernels in ("fast", "general"):
        p = Plan(dataclasses.replace(engine_config(cfg), kernels=kernels, **kw))
        p.set_model(model["vp"], model["vs"], model["rho"], model["taup"], model["taus"])
        out.append(p)
    return out


def _same(a, b):
    for k in b:
        assert np.array_equal(a[k], b[k]), (k, float(np.abs(a[k] - b[k]).max()), float(np.abs(b[k]).max()))


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("kw", CASES, ids=IDS)
def test_forward(kw, batch, cuda_device):
    cfg, model, acq = _case(kw)
    shots = [(acq["src_pos"], acq["src"] * (1 + b), acq["rec_pos"]) for b in range(batch)]
    got = []
    for p in _plans(cfg, model, batch=batch):
        d = p.forward_batch(shots, ["vx", "vz", "p"])
        d = {"%s%d" % (k, b): v for b, s in enumerate(d) for k, v in s.items()}
        d.update({"f%d" % i: p.debug_array(0, i, p.nvol) for i in (0, 2, 3, 5, 8)})
        if cfg["abs_type"] == 1:
            d["psi"] = p.debug_array(5, 9, 2 * cfg["nab"] * cfg["nz"])
        got.append(d)
    assert np.abs(got[1]["vz0"]).max() > 0
    _same(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [k for k in CASES if not k["L"]] + CASES[1:2], ids=lambda k: "%dx%d-L%d" % (k["nz"], k["nx"], k["L"]))
@pytest.mark.parametrize("how", [dict(), dict(precision="fp16"), dict(precision="bf16", batch=2), dict(checkpoint=13),
                                 dict(back_prop_type=2, gradfreqs=(40.0, 60.0)), dict(hout=1), dict(restype=1)],
                         ids=["bnd", "fp16", "bf16-batch", "ckpt", "dft", "hessian", "restype1"])
def test_gradient(kw, how, cuda_device):
    cfg, model, acq = _case(kw)
    if kw["nz"] < 2 * kw["nab"] + 2 * (kw["fdorder"] // 2) and not (how.get("checkpoint") or how.get("back_prop_type")):
        pytest.skip("no cells inside the absorbing layers to save")
    shots = [(acq["src_pos"], acq["src"] * (1 + b), acq["rec_pos"]) for b in range(how.get("batch", 1))]
    got = []
    for p in _plans(cfg, model, **how):
        d = p.forward_batch(shots, ["vx", "vz"], save_boundaries=True)
        p.zero_gradient()
        p.adjoint_batch(shots, d)
        g = p.gradient(transform=False)
        if how.get("hout"):
            g.update({"h" + k: v for k, v in p.hessian(transform=False).items()})
        got.append(g)
    assert all(np.isfinite(v).all() for v in got[1].values()) and np.abs(list(got[1].values())[0]).max() > 0
    _same(*got)
