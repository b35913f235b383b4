"""Outputs of small runs, kept to the bit in tests/golden/bits.npz
(tests/test_bits.py).  Recorded once from the engine on a B200 (with the
one-cell kernels on rows that are no whole quads, the launches per kernel in
2D, and the free surface of FP16 fields, batches and boundary-saving runs in a
launch of its own) and not to be recorded again to make a change pass: a new
kernel gives the same roundings.

    python tests/golden/make_bits.py tests/golden/bits.npz
"""
import dataclasses
import sys

import numpy as np

from tests._cases import engine_config, make_case

BASE = dict(nz=48, ny=30, nx=34, nt=160, nab=8, fdorder=8, freesurf=1, L=0, f0=25.0)
CASES = {
    # FP16 fields: one rounding a step, of FP32 values that must not change
    "3d_fp16": dict(nd=3, how="model", L=2, plan=dict(field_precision="fp16")),
    "3d_fp16_filled": dict(nd=3, how="model", nz=50, L=1, plan=dict(field_precision="fp16")),
    "3d_fp16_o4": dict(nd=3, how="model", fdorder=4, freesurf=0, plan=dict(field_precision="fp16")),
    "2d_fp16": dict(nd=2, how="model", L=1, plan=dict(field_precision="fp16")),
    # boundary saving: the adjoint's free surface amplifies a changed rounding
    "3d_bnd": dict(nd=3, how="bnd"),
    "3d_bnd_filled": dict(nd=3, how="bnd", nz=50),
    "3d_bnd_o4": dict(nd=3, how="bnd", fdorder=4),
    "3d_bnd_batch": dict(nd=3, how="bnd", nz=50, plan=dict(batch=2)),
    "2d_bnd": dict(nd=2, how="bnd", nz=58, nx=60),
    "2d_bnd_resident": dict(nd=2, how="bnd", nz=58, nx=60, freesurf=0),
    "2d_bnd_bf16": dict(nd=2, how="bnd", nz=60, nx=61, fdorder=4, plan=dict(batch=2, precision="bf16")),
    # the free surface with relaxation: folded, apart, recomputed, and slab edges inside quads
    "3d_visco": dict(nd=3, how="model", L=2),
    "3d_visco_filled": dict(nd=3, how="model", nz=50, L=1),
    "3d_visco_o4": dict(nd=3, how="model", fdorder=4, L=2),
    "3d_visco_batch": dict(nd=3, how="model", L=1, plan=dict(batch=2)),
    "3d_visco_ckpt": dict(nd=3, how="ckpt", L=1, plan=dict(checkpoint=17)),
    "3d_cut": dict(nd=3, how="model", nab=6, freesurf=0, L=1),
    "3d_cut_filled": dict(nd=3, how="model", nz=50, nab=7, L=2),
    "3d_general": dict(nd=3, how="model", L=1, plan=dict(kernels="general")),
    "2d_resident": dict(nd=2, how="model", nz=100, nx=90, L=2),
    "2d_resident_o4": dict(nd=2, how="model", nz=70, nx=90, fdorder=4),
    "2d_quads": dict(nd=2, how="model", nz=58, nx=60, L=1, off=True),
    "2d_quads_o4": dict(nd=2, how="model", nz=60, nx=60, fdorder=4, freesurf=0, off=True),
    "2d_order6": dict(nd=2, how="model", nz=60, nx=60, fdorder=6, L=1),
}


def run(name):
    """{output: array}: traces of every third receiver in the second half of
    the steps, and every seventh gradient sum.  3D mu sums of rows that are no
    whole quads are left out: the one-cell adjoint kernel adds their terms in
    another order."""
    from seiscl_b200.engine import Plan

    kw = {**BASE, **CASES[name]}
    how, off, plan = kw.pop("how"), kw.pop("off", False), kw.pop("plan", {})
    cfg, model, acq = make_case(**kw)
    nz, nx, ny = kw["nz"], kw["nx"], kw["ny"]
    three = kw["nd"] == 3
    acq["src_pos"][0, [0, 2]] = [nx // 2 * 10.0, (3 if kw["freesurf"] else nz // 2) * 10.0]
    x = np.arange(2, nx - 2, 3)
    rec = np.zeros((2 * len(x), 8), np.float32)
    rec[:, 0] = np.tile(x, 2) * 10.0
    rec[:, 1] = (ny // 2 + 1) * 10.0 if three else 0.0
    rec[:, 2] = np.repeat([0, nz // 2 + 2], len(x)) * 10.0
    if off:
        rec[0, 2] = -20.0   # in the padding: keeps the run off the resident loop
    rec[:, 4] = np.arange(1, len(rec) + 1)
    p = Plan(dataclasses.replace(engine_config(cfg), **plan))
    p.set_model(model["vp"], model["vs"], model["rho"], model["taup"], model["taus"])
    outs = ["vx", "vy", "vz"] if three else ["vx", "vz"]
    shots = [(acq["src_pos"], acq["src"] * (1 + b), rec) for b in range(plan.get("batch", 1))]
    data = p.forward_batch(shots, outs, save_boundaries=how != "model")
    out = {"%s%d" % (k, b): v[1::3, kw["nt"] // 2::4] for b, d in enumerate(data) for k, v in d.items()}
    if how != "model":
        p.zero_gradient()
        p.adjoint_batch(shots, data)
        g = p.gradient(transform=False)
        quads = kw["fdorder"] == 8 and nz % 4 == 0
        out.update({k: v.ravel()[::23] for k, v in g.items() if k != "mu" or quads or not three})
    return out


def main():
    np.savez_compressed(sys.argv[1], **{"%s/%s" % (n, k): v for n in CASES for k, v in run(n).items()})


if __name__ == "__main__":
    main()
