"""Autotuner of the step's launch settings, by measurement on the caller's workload.

* Chemistry (hf_set_chem_tuning): the blocks of 64 lanes per SM the batched queue kernel
  is built for (its per-lane register budget) and the cooperative threshold (cells that
  took at least 2^b - 1 step attempts in the previous call are integrated by groups of 8
  lanes, 4 cells per warp; 16: never, and the kernel without that phase; 17, what the library
  starts with: its own choice of cells from their costs).
  Each candidate runs the batched chemistry three times on the same sample call (the
  chemistry input of a Strang step of the workload): the first two build the per-cell
  history (cost order, warm-started step sizes) as consecutive steps do, the third is
  timed with CUDA events.  The fastest is taken when it is more than MARGIN faster than
  the setting without groups: one call stands for the steps that follow, and a
  cooperative setting whose queue stays empty on the sample can still engage, and cost,
  in later steps.  Otherwise the setting in force stays (unless it is more than MARGIN
  slower than the fastest): a sample that gains little from the library's own choice of
  cells says nothing about the batches that gain 3 to 5 times from it.  The other register
  budgets are timed without groups: where a sample runs wholly in groups all budgets are
  alike, and one of them would win by chance.
* Stepper chemistry (tune_stepper): the same settings timed over a few whole graph
  steps of the caller's stepper from one start state, each candidate from a fresh
  stepper (its history builds up over the steps as it does in a run, so a cooperative
  setting shows whether its queue engages and pays).  The setting in force stays unless one
  is more than MARGIN faster.  Small, tail-bound problems gain most
  (a 1D detonation of 4,000 cells: 15.4 to 5.6 ms a step); the 2048 x 512 detonation's first
  steps gain 8%.
* Flux form: one Euler stage of the workload's state with the plain per-face kernels and
  with the fused TMA-tile kernel (32 x 7 cells per CTA), each timed after a warm-up; the
  faster form is returned for the caller's stepper.

Settings change launch shapes only: results agree to rounding across candidates and are
reproducible for a fixed setting.
"""
import ctypes

import torch

from . import _lib as L
from . import solver as S

# the setting without groups, which the others are measured against; the library starts at (4, 17)
CHEM_DEFAULT = (4, 16)
CHEM_CANDIDATES = [CHEM_DEFAULT, (4, 17), (5, 16), (6, 16), (8, 16), (4, 3), (4, 5), (4, 7)]
MARGIN = 0.03
STEP_CANDIDATES = [CHEM_DEFAULT, (4, 17), (4, 3), (4, 5), (4, 7)]


def pick(sweep, key, default=CHEM_DEFAULT, margin=MARGIN, in_force=None):
    """The sweep entry to apply: that of the setting `in_force` when the sweep has one and the
    fastest by `key` is not more than `margin` faster; else likewise that of the `default`
    setting; else the fastest."""
    best = min(sweep, key=lambda r: r[key])
    for setting in (in_force, default):
        for r in sweep:
            if (r["blocks_per_sm"], r["coop_min_bucket"]) == setting and best[key] >= (1.0 - margin) * r[key]:
                return r
    return best


def get_chem_tuning(ctx):
    m, c = ctypes.c_int32(0), ctypes.c_int32(0)
    ctx.lib.hf_get_chem_tuning(ctypes.byref(m), ctypes.byref(c))
    return int(m.value), int(c.value)


def set_chem_tuning(ctx, blocks_per_sm=0, coop_min_bucket=0):
    ctx.check(ctx.lib.hf_set_chem_tuning(int(blocks_per_sm), int(coop_min_bucket)), "set_chem_tuning")


def _events():
    return torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)


def tune_chemistry(ctx, X, dt, candidates=CHEM_CANDIDATES, apply=True):
    """X: (NV, n) float64 CUDA tensor, the input of one chemistry call over dt (not
    modified).  Returns {"best": (blocks_per_sm, coop_min_bucket), "sweep": [...]} and, with
    apply, leaves the best setting in force."""
    before = get_chem_tuning(ctx)
    sweep = []
    try:
        for minb, coop in candidates:
            set_chem_tuning(ctx, minb, coop)
            cb = S.ChemistryBatch(ctx, "batched")
            for _ in range(2):
                cb.advance(X.clone(), dt)
            field = X.clone()
            c0 = ctx.counters()
            torch.cuda.synchronize()
            e0, e1 = _events()
            e0.record()
            cb.advance(field, dt)
            e1.record()
            torch.cuda.synchronize()
            c1 = ctx.counters()
            sweep.append({"blocks_per_sm": minb, "coop_min_bucket": coop, "ms": e0.elapsed_time(e1),
                          "coop_cells": c1["chem_coop_cells"] - c0["chem_coop_cells"],
                          "attempts": c1["chem_steps"] - c0["chem_steps"]})
            del field
    finally:
        set_chem_tuning(ctx, *before)
    best = pick(sweep, "ms")
    if (best["blocks_per_sm"], best["coop_min_bucket"]) == CHEM_DEFAULT:
        best = pick(sweep, "ms", in_force=before)
    if apply:
        set_chem_tuning(ctx, best["blocks_per_sm"], best["coop_min_bucket"])
    return {"best": (best["blocks_per_sm"], best["coop_min_bucket"]), "sweep": sweep}


def tune_flux(ctx, level, U, dt, repeats=3):
    """U: (NV, ny, nx) state of a one-patch level; dt: a step of it (stages of dt/2 are
    timed).  Returns {"best": "plain"|"fused", "ms": {form: ms per stage}}."""
    nv, ny, nx = U.shape
    pa = S.PatchArray(nv, nx, ny)
    pa.interior().copy_(U)
    S.fill(ctx, level, pa)
    out = pa.like()
    ms = {}
    for name, form in (("plain", L.HF_FLUX_PLAIN), ("fused", L.HF_FLUX_FUSED)):
        S.euler_stage(ctx, level, pa, out, 0.5 * dt, form=form)
        torch.cuda.synchronize()
        e0, e1 = _events()
        e0.record()
        for _ in range(repeats):
            S.euler_stage(ctx, level, pa, out, 0.5 * dt, form=form)
        e1.record()
        torch.cuda.synchronize()
        ms[name] = e0.elapsed_time(e1) / repeats
    return {"best": min(ms, key=ms.get), "ms": ms}


def tune_stepper(ctx, level, U, cfl, flux="plain", warm=2, steps=6, candidates=STEP_CANDIDATES, apply=True):
    """U: (NV, ny, nx) state; the batched chemistry settings timed over `steps` graph steps
    (after `warm` steps) of a fresh stepper per candidate.  Returns {"best": (...),
    "sweep": [{"blocks_per_sm", "coop_min_bucket", "ms_per_step", "coop_cells"}]} and, with
    apply, leaves the best setting in force (as pick() chooses it)."""
    before = get_chem_tuning(ctx)
    sweep = []
    try:
        for minb, coop in candidates:
            set_chem_tuning(ctx, minb, coop)
            st = S.Stepper(ctx, level, U, flux=flux, chem="batched")
            try:
                for _ in range(warm):
                    st.step(cfl=cfl)
                c0 = ctx.counters()
                torch.cuda.synchronize()
                e0, e1 = _events()
                e0.record()
                st.run(steps, cfl=cfl)
                e1.record()
                torch.cuda.synchronize()
                c1 = ctx.counters()
            finally:
                st.close()
            sweep.append({"blocks_per_sm": minb, "coop_min_bucket": coop, "ms_per_step": e0.elapsed_time(e1) / steps,
                          "coop_cells": c1["chem_coop_cells"] - c0["chem_coop_cells"]})
    finally:
        set_chem_tuning(ctx, *before)
    best = pick(sweep, "ms_per_step", in_force=before)
    if apply:
        set_chem_tuning(ctx, best["blocks_per_sm"], best["coop_min_bucket"])
    return {"best": (best["blocks_per_sm"], best["coop_min_bucket"]), "sweep": sweep}
