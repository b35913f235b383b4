"""2D P-SV modelling with the wave fields resident on chip
(sfd_resident2d.cu) against the one-launch-per-kernel loop (kernels
"general"), bit for bit: seismograms, final wave fields and memory
variables, the gradient from the boundary shells it saves, and the adjoint
loop of elastic media without a free surface.  Grids from
one tile to the whole chip, ragged tiles, every order, more points in a tile
than its list holds, several sources in one cell, points in the padding."""
import dataclasses

import numpy as np
import pytest

from tests._cases import engine_config, make_case

CASES = [
    dict(nz=20, nx=33, nt=60, nab=4, fdorder=4),                               # one CTA's worth of cells
    dict(nz=100, nx=150, nt=90, nab=16, fdorder=4, L=3),
    dict(nz=38, nx=301, nt=300, nab=8, fdorder=8, L=2),                        # two segments
    dict(nz=302, nx=395, nt=70, nab=20, fdorder=8),                            # two cells a thread
    dict(nz=250, nx=611, nt=40, nab=10, fdorder=4, L=1, freesurf=0),           # four
    dict(nz=402, nx=577, nt=40, nab=16, fdorder=8, freesurf=0, src_type=2),
    dict(nz=120, nx=90, nt=600, nab=0, fdorder=8, L=1, src_type=0),            # no absorbing layer, three segments
    # what the resident steps leave to the ordinary loop
    dict(nz=120, nx=90, nt=80, nab=9, fdorder=6, L=3, abs_type=2),
    dict(nz=36, nx=30, nt=80, nab=16, fdorder=8),                              # overlapping slabs
    dict(nz=602, nx=1203, nt=24, nab=16, fdorder=4, freesurf=0),
]


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


def _states(p, cfg):
    out = {n: p.debug_array(0, i, p.nvol) for n, i in (("vx", 0), ("vz", 2), ("sxx", 3), ("szz", 5), ("sxz", 8))}
    if cfg["L"]:
        out.update({n: p.debug_array(2, i, p.nvol * cfg["L"]) for n, i in (("rxx", 0), ("rzz", 2), ("rxz", 5))})
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kw", CASES, ids=lambda k: "%dx%d-o%d" % (k["nz"], k["nx"], k["fdorder"]))
def test_resident_steps_match_general(kw, cuda_device):
    cfg, model, acq = make_case(nd=2, **kw)
    got = []
    for p in _plans(cfg, model):
        d = p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx", "vz", "p", "sxz"])
        got.append({**d, **_states(p, cfg)})
    assert np.abs(got[1]["vx"]).max() > 0
    _same(*got)


@pytest.mark.gpu
def test_resident_points(cuda_device):
    """2800 receivers on a grid of few tiles, some in the padding above the
    surface, two explosive and one force source in shared cells."""
    cfg, model, acq = make_case(nd=2, nz=40, nx=70, nt=60, nab=6)
    x, z = np.meshgrid(np.arange(70), np.arange(40), indexing="ij")
    rec = np.zeros((2800, 8), np.float32)
    rec[:, 0], rec[:, 2] = x.ravel() * 10.0, z.ravel() * 10.0
    rec[:3, 2] = -30.0
    src_pos = np.repeat(acq["src_pos"], 3, 0)
    src_pos[2, 2] = -10.0
    src = np.repeat(acq["src"], 3, 0) * np.array([[1.0], [0.5], [2.0]], np.float32)
    got = [p.forward(src_pos, src, rec, ["vx", "vz", "p"]) for p in _plans(cfg, model)]
    assert np.abs(got[1]["vx"]).max() > 0
    _same(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("nz,nx,nb,prec", [(60, 71, 3, "fp32"), (102, 95, 5, "fp16"), (60, 71, 2, "bf16")])
def test_resident_batch_and_shells(nz, nx, nb, prec, cuda_device):
    """Batched shots with saved boundaries: the adjoint reads what the
    resident run left."""
    cfg, model, acq = make_case(nd=2, nz=nz, nx=nx, nt=100, nab=8)
    shots = []
    for b in range(nb):
        sp = acq["src_pos"].copy()
        sp[0, 0] += 30.0 * b
        shots.append((sp, acq["src"] * (1 + b), acq["rec_pos"][b:]))
    got = []
    for p in _plans(cfg, model, batch=nb, precision=prec):
        d = p.forward_batch(shots, ["vx", "vz"], save_boundaries=True)
        p.zero_gradient()
        p.adjoint_batch(shots, d)
        got.append({**{"%s%d" % (k, i): v for i, s in enumerate(d) for k, v in s.items()}, **p.gradient(transform=False)})
    assert np.abs(got[1]["M"]).max() > 0
    _same(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("kw,nb,prec,sel", [
    (dict(nz=20, nx=33, nt=60, nab=4, fdorder=4), 1, "fp32", ["vx", "vz"]),
    (dict(nz=100, nx=150, nt=90, nab=16, fdorder=4, src_type=2), 1, "fp32", ["p"]),
    (dict(nz=38, nx=301, nt=300, nab=8, fdorder=8), 1, "bf16", ["vx", "vz", "p", "sxz"]),     # two segments
    (dict(nz=302, nx=391, nt=70, nab=20, fdorder=8), 1, "fp32", ["vx", "vz"]),                # two cells a thread
    (dict(nz=102, nx=95, nt=80, nab=9, fdorder=8, src_type=0), 5, "fp16", ["vx", "p"]),
    (dict(nz=120, nx=90, nt=70, nab=12, fdorder=4), 16, "fp32", ["vx", "vz"]),                # groups of shots
    (dict(nz=60, nx=70, nt=60, nab=6, fdorder=8, tmin=10, tmax=50), 1, "fp32", ["vx", "vz"]),
    (dict(nz=96, nx=90, nt=60, nab=9, fdorder=8, abs_type=2), 2, "fp32", ["vx", "vz"]),       # left to the ordinary loop
], ids=lambda k: "%dx%d-o%d" % (k["nz"], k["nx"], k["fdorder"]) if isinstance(k, dict) else None)
def test_resident_adjoint_matches_general(kw, nb, prec, sel, cuda_device):
    """The resident adjoint loop: gradient sums, reconstructed fields and
    memory variables left by the last step, bit for bit.  Two sources, the
    second in the cell of a receiver."""
    steps = {k: kw[k] for k in ("tmin", "tmax") if k in kw}
    cfg, model, acq = make_case(nd=2, freesurf=0, **{k: v for k, v in kw.items() if k not in steps})
    shots = []
    for b in range(nb):
        sp = np.repeat(acq["src_pos"], 2, 0)
        sp[0, 0] += 10.0 * (b % 5)
        sp[1, :3] = acq["rec_pos"][0, :3]
        shots.append((sp, np.repeat(acq["src"], 2, 0) * (1 + b), acq["rec_pos"]))
    got = []
    for p in _plans(cfg, model, batch=nb, precision=prec, **steps):
        d = p.forward_batch(shots, sel, save_boundaries=True)
        p.zero_gradient()
        p.adjoint_batch(shots, d)
        got.append({**p.gradient(transform=False), **_states(p, cfg)})
    assert np.abs(got[1]["M"]).max() > 0
    _same(*got)


@pytest.mark.gpu
def test_resident_unstable_run_is_reported(cuda_device, monkeypatch):
    from seiscl_b200.engine import SeisCLEngineError

    monkeypatch.setenv("SEISCL_B200_UNCHECKED_CFL", "1")
    cfg, model, acq = make_case(nd=2, nz=60, nx=71, nt=200, nab=8, dt=5e-3)
    for p in _plans(cfg, model):
        with pytest.raises(SeisCLEngineError, match="unstable"):
            p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx"])


def _fwi(p, shots):
    d = p.forward_batch(shots, ["vx", "vz"], save_boundaries=True)
    p.zero_gradient()
    p.adjoint_batch(shots, d)
    return {**{"%s%d" % (k, i): v for i, s in enumerate(d) for k, v in s.items()}, **p.gradient(transform=False)}


@pytest.mark.gpu
def test_refused_launches_take_the_ordinary_loop(cuda_device):
    """A cooperative launch that the driver refuses (an error code made on
    the host): the call runs on the ordinary loop, and so do the plan's later
    ones, with the same bits."""
    cfg, model, acq = make_case(nd=2, nz=60, nx=71, nt=300, nab=8, freesurf=0)
    shots = [(acq["src_pos"], acq["src"], acq["rec_pos"])] * 2
    want, got = [], []
    for refuse in ("none", "forward", "adjoint"):
        p = _plans(cfg, model, batch=2)[0]
        if refuse == "forward":
            p.debug_launch(4)
        d = p.forward_batch(shots, ["vx", "vz"], save_boundaries=True)
        p.zero_gradient()
        if refuse == "adjoint":
            p.debug_launch(4)
        p.adjoint_batch(shots, d)
        got.append({**{k: v for k, v in d[1].items()}, **p.gradient(transform=False)})
        want.append(_fwi(p, shots))
    for g, w in zip(got[1:], want[1:]):
        _same(g, got[0])
        _same(w, want[0])


@pytest.mark.gpu
@pytest.mark.parametrize("sms", [0, 5, 60, 1000])
def test_fewer_sms(sms, cuda_device, monkeypatch):
    """What a process with part of the device plans: fewer tiles, or none."""
    cfg, model, acq = make_case(nd=2, nz=100, nx=150, nt=80, nab=16, fdorder=4, freesurf=0)
    shots = [(acq["src_pos"], acq["src"] * (1 + b), acq["rec_pos"]) for b in range(2)]
    want = _fwi(_plans(cfg, model, batch=2)[1], shots)
    monkeypatch.setenv("SEISCL_B200_RESIDENT_SMS", str(sms))
    _same(_fwi(_plans(cfg, model, batch=2)[0], shots), want)


@pytest.mark.gpu
def test_wait_that_runs_out(cuda_device):
    """A tile whose neighbour never sends gives up after its bound, the host
    reads it, and the plan goes on working."""
    from seiscl_b200.engine import SeisCLEngineError

    cfg, model, acq = make_case(nd=2, nz=100, nx=90, nt=60, nab=8)
    p = _plans(cfg, model)[0]
    want = p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx"])
    with pytest.raises(SeisCLEngineError, match="time bound"):
        p.debug_launch(5)
    _same(p.forward(acq["src_pos"], acq["src"], acq["rec_pos"], ["vx"]), want)


@pytest.mark.gpu
def test_plans_on_threads(cuda_device):
    """Resident loops of several plans on threads of their own, forward and
    adjoint, small grids and one of the whole chip: the bits of each alone."""
    from concurrent.futures import ThreadPoolExecutor

    cases = [make_case(nd=2, nz=60, nx=71, nt=300, nab=8, freesurf=0, seed=1),
             make_case(nd=2, nz=302, nx=391, nt=120, nab=20, freesurf=0, seed=2),
             make_case(nd=2, nz=100, nx=150, nt=400, nab=16, fdorder=4, freesurf=0, seed=3)]
    jobs = [(_plans(cfg, model)[0], [(acq["src_pos"], acq["src"], acq["rec_pos"])]) for cfg, model, acq in cases]
    want = [_fwi(*j) for j in jobs]
    with ThreadPoolExecutor(len(jobs)) as pool:
        for _ in range(3):
            for g, w in zip(pool.map(lambda j: _fwi(*j), jobs), want):
                _same(g, w)
