"""Autotuner of the tensor-core SR matvec tiling.

The tcgen05 O^H u has two tilings (``qes_sr_tc_plan``): one 128-row M tile per sample chunk (small
problems) or an M/N-tiled kernel whose CTAs fold several sample chunks into TMEM (N chunks of NC
hidden units, a target CTA count); ``qes_sr_set_ohu_pairs`` runs the single-tile kernel as pairs
of CTAs that add their split-K partials through distributed shared memory, and
``qes_sr_set_fused_sv`` runs the single-tile matvec as one cooperative S v kernel (O v, the mean of
O v over a grid barrier and O^H u in the same CTAs); ``qes_sr_set_ov_split`` and ``qes_sr_set_ovz`` choose
the O v product (split-complex over the hidden axis, or through z = Sigma V).  ``tune_sr_tiling`` times
CG iterations on a given batch for every candidate (``qes_sr_solve_cg`` with the tolerance at zero, so
that it runs exactly the iterations asked for; the time of K iterations subtracted from that of 2K
removes the once-per-solve work: operand preparation, force, set-up), keeps the fastest, applies it
process-wide and persists it in a JSON cache keyed by device, dtype and shape (``$QES_B200_AUTOTUNE``
or ``~/.cache/pyqusolver_b200/autotune.json``).  Candidates that the shapes do not admit
(QES_ERR_SIZE / QES_ERR_ARG) are skipped.  Every candidate computes the same operator; the choice
changes only the order of the float32 partial sums.

The tilings are those of the kernel chain (warm starts, preconditioned solves, single products, and
shapes that the one-launch CG does not fit), and it is the chain that is timed.  Where the one-launch
CG fits, it solves whatever tiling has been applied (``apply_tiling``), unless it was switched off with
``qes_sr_set_one_launch(0)``.
"""

from __future__ import annotations

import ctypes as C
import json
import os

import torch

from . import _lib
from . import device as dv


def _cache_path(cache=None):
    return cache or os.environ.get("QES_B200_AUTOTUNE", os.path.join(os.path.expanduser("~"), ".cache",
                                                                      "pyqusolver_b200", "autotune.json"))


def _candidates(ns, nh, cplx):
    # (mode, nc, ctas, pairs, fused S v, split-complex O v, O v through z = Sigma V): automatic with
    # the z-form O v, the same with O^H u in CTA pairs, the product over the hidden axis (T as A), its
    # split-complex variant, the fused kernel, then the M/N-tiled O^H u with the z-form O v; the
    # split flag matters for complex networks only
    splits = (0, 1) if cplx else (0,)
    out = [(0, 0, 0, 0, 0, 0, 1), (0, 0, 0, 1, 0, 0, 1)]
    out += [(0, 0, 0, 0, 0, sp, 0) for sp in splits] + [(0, 0, 0, 0, 1, 0, 0)]
    for nc in (256, 208, 128, 96, 64, 32):
        if nc > ((nh + 15) // 16) * 16:
            continue
        for ctas in (148, 296, 592):
            out.append((2, nc, ctas, 0, 0, 0, 1))
    return out


def tune_sr_tiling(net, bits, tanh_theta, *, repeats=3, iters=24, cache=None, candidates=None):
    """Time a CG iteration on (net, bits, tanh_theta) under each tiling candidate (mode, nc, ctas, pairs,
    sv, split, ovz); apply and return the fastest as a dict with the per-iteration times in ms.  A cached choice for
    the same device and shapes is applied without timing."""
    dc = dv.dtype_code(net.flat)
    n = int(bits.shape[0])
    dev = torch.cuda.get_device_name(bits.device)
    key = f"sr_cg_iter8|{dev}|{dc}|{net.ns}|{net.nh}|{n}"
    path = _cache_path(cache)
    table = {}
    try:
        with open(path) as f:
            table = json.load(f)
    except (OSError, ValueError):
        table = {}
    if key in table and candidates is None:
        apply_tiling(*table[key]["choice"])
        return dict(table[key], cached=True)
    cands = candidates or _candidates(net.ns, net.nh, net.is_complex)
    eloc = torch.randn(n, dtype=torch.complex64, device=bits.device)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    timings = {}
    best, best_t = None, float("inf")

    def solve(ws, k):
        dv.sr_solve_cg(net.flat, net.ns, net.nh, bits, tanh_theta, eloc, shift=1e-3, rtol=0.0, atol=0.0,
                       maxiter=k, check_every=k, workspace=ws, allow_not_converged=True)

    def timed(ws, k):
        ts = []
        for _ in range(repeats):
            ev0.record()
            solve(ws, k)
            ev1.record()
            torch.cuda.synchronize()
            ts.append(ev0.elapsed_time(ev1))
        return sorted(ts)[len(ts) // 2]

    one_launch = _one_launch(0)                                         # time the chain
    try:
        for cand in cands:
            apply_tiling(*cand)
            if not _lib.sr_uses_tensor_cores(dc, net.ns, net.nh, n):
                continue
            try:
                ws = dv.sr_workspace(dc, net.ns, net.nh, n, bits.device)
                solve(ws, iters)                                        # warm-up, graph capture
                solve(ws, 2 * iters)
                torch.cuda.synchronize()
                t = (timed(ws, 2 * iters) - timed(ws, iters)) / iters
            except _lib.QESError as e:
                if e.code not in (_lib.QES_ERR_SIZE, _lib.QES_ERR_ARG):
                    raise
                continue
            timings[str(cand)] = t
            if t < best_t:
                best, best_t = cand, t
    finally:
        _one_launch(one_launch)
        apply_tiling(*(best or DEFAULT_TILING))
    if best is None:
        return {"choice": DEFAULT_TILING, "ms": None, "timings": timings, "cached": False}
    entry = {"choice": list(best), "ms": best_t, "timings": timings}
    table[key] = entry
    try:
        os.makedirs(os.path.dirname(path), exist_ok=True)
        tmp = path + ".tmp"
        with open(tmp, "w") as f:
            json.dump(table, f, indent=1)
        os.replace(tmp, path)
    except OSError:
        pass
    return dict(entry, cached=False)


DEFAULT_TILING = (0, 0, 0, 0, 0, 0, 1)


def _one_launch(mode):
    old = C.c_int(0)
    _lib.call("qes_sr_set_one_launch", mode, C.byref(old))
    return old.value


def apply_tiling(mode, nc, ctas, pairs, sv=0, split=0, ovz=1):
    """Tiling of the tensor-core kernel chain in this process; the one-launch CG keeps the shapes that fit it."""
    if _one_launch(-1):
        _one_launch(1 if (mode, nc, ctas, pairs, sv, split, ovz) == DEFAULT_TILING else 2)
    _lib.call("qes_sr_set_tiling", int(mode), int(nc), int(ctas))
    _lib.call("qes_sr_set_ohu_pairs", int(pairs))
    _lib.call("qes_sr_set_fused_sv", int(sv))
    _lib.call("qes_sr_set_ov_split", int(split))
    _lib.call("qes_sr_set_ovz", int(ovz))
