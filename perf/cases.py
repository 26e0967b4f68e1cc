"""The work that this package is timed on: whole VMC epochs, and the calls that programs make on their own.

Kinds of case (every one through the public API):

* ``epoch``   ``NQS.set_params`` + ``NQS.train_step``: one VMC epoch (sampling, local energy, SR solve,
  update) from parameters that an outer program owns; returns the updated weights and the batch drawn.
* ``batch``   ``NQSBatch.set_params`` + ``NQSBatch.train_step``: the same for many problems at once.
* ``update``  ``TDVP.solve`` + ``param_update`` on a batch in hand (configurations, tanh(theta), local
  energies), with or without sample weights; returns the updated weights.
* ``dense``   ``TDVP(sr_form_matrix=True).solve`` on a batch in hand: S formed, float64 Cholesky; returns x.
* ``energy``  ``NQS(states)`` + ``NQS.local_energy(states)``: log psi and E_loc of given configurations.
* ``step``    ``NQS.step(configs)``: local energies and the rows of log-derivatives.
* ``grad``    ``RBM.log_psi_autograd`` + ``backward``: the gradient of a weighted sum of log psi.

Parameters, configurations and start states are drawn from the seed.  Models: ``tfim`` (transverse-field
Ising, single flips, real RBM), ``xxz`` and ``j1j2`` (exchange moves at fixed S^z, complex RBM).
"""

from __future__ import annotations

import numpy as np
import torch

RATE = 1e-2
COUPLINGS = {"tfim": dict(j=1.0, hx=1.0, hz=0.0), "xxz": dict(jxy=-1.0, jz=-1.0), "j1j2": dict(J1=-1.0, J2=-0.5)}


def listed():
    return [
        # the smallest step: a 16-site chain, 16 chains x 64 samples, real RBM with 16 hidden units
        dict(name="epoch_tfim_16", kind="epoch", model="tfim", lx=16, ly=1, nh=16, chains=16, samples=64, scale=0.05,
             shift=1e-3),
        # a chain of odd length with a small, ragged batch
        dict(name="epoch_tfim_63", kind="epoch", model="tfim", lx=63, ly=1, nh=126, chains=100, samples=10, scale=0.05,
             shift=1e-2),
        # frustrated 6x6 magnet, complex RBM with alpha = 4, 8,192 samples
        dict(name="epoch_j1j2_6x6", kind="epoch", model="j1j2", lx=6, ly=6, nh=144, chains=2048, samples=4, scale=0.02,
             shift=1e-3),
        # odd sides, odd hidden layer, ragged batch
        dict(name="epoch_xxz_9x7", kind="epoch", model="xxz", lx=9, ly=7, nh=189, chains=1000, samples=5, scale=0.02,
             shift=1e-3),
        # the flagship step: 10x10 Heisenberg, complex RBM with alpha = 2, 16,384 samples
        dict(name="epoch_xxz_10x10", kind="epoch", model="xxz", lx=10, ly=10, nh=200, chains=4096, samples=4,
             scale=0.02, shift=1e-3),
        # the largest single problem: 20x20, 1,600 hidden units, 642,000 parameters
        dict(name="epoch_tfim_20x20", kind="epoch", model="tfim", lx=20, ly=20, nh=1600, chains=4096, samples=4,
             scale=0.01, shift=1e-4),
        # 64 chains of uneven length advanced together
        dict(name="batch_tfim_64", kind="batch", problems=64, lo=12, hi=64, alpha=2, chains=256, samples=8, scale=0.05,
             shift=1e-2),
        # the optimisation half of a step on a reweighted batch that another sampler drew
        dict(name="update_xxz_10x10", kind="update", model="xxz", lx=10, ly=10, nh=200, rows=10000, weighted=True,
             scale=0.02, shift=1e-2),
        # the formed-matrix solve of the 6x6 magnet (5,364 complex parameters)
        dict(name="dense_j1j2_6x6", kind="dense", model="j1j2", lx=6, ly=6, nh=144, rows=8192, scale=0.02, shift=1e-3),
        # log-derivative rows for an external optimiser
        dict(name="step_xxz_10x10", kind="step", model="xxz", lx=10, ly=10, nh=200, rows=4096, scale=0.05),
        # backward of log psi through autograd
        dict(name="grad_xxz_10x10", kind="grad", model="xxz", lx=10, ly=10, nh=200, rows=16384, scale=0.05),
        # energies of a large evaluation batch, no optimisation
        dict(name="energy_tfim_20x20", kind="energy", model="tfim", lx=20, ly=20, nh=1600, rows=16384, scale=0.01),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["epoch", "epoch", "epoch", "update", "energy", "step", "grad", "dense", "batch"])
    if kind == "batch":
        lo = rng.randint(6, 24)
        return dict(kind=kind, problems=_log_int(rng, 2, 64), lo=lo, hi=lo + rng.randint(1, 40), alpha=rng.randint(1, 2),
                    chains=_log_int(rng, 16, 256), samples=rng.randint(2, 8), scale=0.05, shift=1e-2)
    model = rng.choice(["tfim", "xxz", "j1j2"])
    if model == "tfim" and rng.random() < 0.5:
        lx, ly = _log_int(rng, 10, 120), 1
    else:
        lx, ly = rng.randint(3, 11), rng.randint(3, 11)
    lx += lx * ly % 32 == 0                      # odd words of spins rather than exactly full ones
    ns = lx * ly
    nh = max(4, min(_log_int(rng, max(4, ns // 2), 4 * ns), 480 if model == "tfim" else 250))
    c = dict(kind=kind, model=model, lx=lx, ly=ly, nh=nh, scale=rng.choice([0.01, 0.02, 0.05]))
    if kind in ("epoch", "update", "dense"):
        c["shift"] = 1e-3 if kind == "dense" else 1e-2
    if kind == "epoch":
        samples = rng.randint(2, 16)
        c.update(chains=max(8, _log_int(rng, 256, 16384) // samples), samples=samples)
    elif kind == "dense":
        c["nh"] = max(4, min(nh, 4000 // (ns + 1)))
        c.update(rows=_log_int(rng, 200, 8192))
    else:
        c.update(rows=_log_int(rng, 200, 4096 if kind == "step" else 16384))
        if kind == "update":
            c.update(weighted=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------------------------------ inputs
def _is_complex(case):
    return case["model"] != "tfim"


def _n_params(ns, nh):
    return ns + nh + ns * nh


def _model(case):
    import pyqusolver_b200 as qb
    dim = 2 if case["ly"] > 1 else 1
    lat = qb.SquareLattice(dim, case["lx"], case["ly"], bc="pbc")
    cls = {"tfim": qb.TransverseFieldIsing, "xxz": qb.XXZ, "j1j2": qb.J1J2Model}[case["model"]]
    return cls(lat, **COUPLINGS[case["model"]])


def _params(case, seed, dtype=np.float64):
    """Flat [a, b, W], float64 or complex128."""
    rng = np.random.default_rng([seed, 11])
    P = _n_params(case["lx"] * case["ly"], case["nh"])
    x = rng.normal(0.0, case["scale"], size=P)
    if _is_complex(case):
        x = x + 1j * rng.normal(0.0, case["scale"], size=P)
    return torch.as_tensor(x, device="cuda")


def _spins(case, seed):
    """(rows, sites) of +-1 in float64: any configuration, or exactly half up where S^z is conserved."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 3)
    rows, ns = case["rows"], case["lx"] * case["ly"]
    r = torch.rand((rows, ns), generator=g, device="cuda")
    if case["model"] == "tfim":
        return torch.where(r < 0.5, -1.0, 1.0).to(torch.float64)
    s = torch.full((rows, ns), -1.0, dtype=torch.float64, device="cuda")
    return s.scatter_(1, r.argsort(dim=1)[:, :ns // 2], 1.0)


def _pack(spins):
    """Bit i & 31 of word i >> 5 is set for spin up."""
    rows, ns = spins.shape
    nw = (ns + 31) // 32
    up = torch.zeros((rows, nw * 32), dtype=torch.int64, device=spins.device)
    up[:, :ns] = (spins > 0).to(torch.int64)
    words = (up.view(rows, nw, 32) << torch.arange(32, device=spins.device)).sum(dim=2)
    return torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32).contiguous()


def _bonds(case):
    """(i, j, coupling) of every bond: forward neighbours and, for J1-J2, forward diagonals."""
    lx, ly = case["lx"], case["ly"]
    kinds = [((1, 0), (0, 1)) if ly > 1 else ((1, 0),)]
    couplings = [1.0 if case["model"] == "tfim" else -1.0]
    if case["model"] == "j1j2":
        kinds.append(((1, 1), (-1, 1)))
        couplings.append(-0.5)
    out = []
    for shifts, c in zip(kinds, couplings):
        for y in range(ly):
            for x in range(lx):
                for dx, dy in shifts:
                    out.append((x + lx * y, (x + dx) % lx + lx * ((y + dy) % ly), c))
    return out


def _split(flat, ns, nh):
    return flat[:ns], flat[ns:ns + nh], flat[ns + nh:].view(ns, nh)


def _theta(flat, spins, nh):
    _, b, W = _split(flat, spins.shape[1], nh)
    return spins.to(flat.dtype) @ W + b


def _log_psi(flat, spins, nh):
    a = flat[:spins.shape[1]]
    th = _theta(flat, spins, nh)
    z = torch.where(th.real < 0, -th, th) if th.is_complex() else th.abs()
    return spins.to(flat.dtype) @ a + (z + torch.log1p(torch.exp(-2 * z)) - np.log(2.0)).sum(dim=1)


def _local_energy(case, flat, spins):
    """E_loc in 64 bits: the psi ratio of a move is exp(2 g A) prod_m (cosh 2D_m + g tanh(theta_m) sinh 2D_m)."""
    ns, nh = spins.shape[1], case["nh"]
    a, _, W = _split(flat, ns, nh)
    t = torch.tanh(_theta(flat, spins, nh))
    e = torch.zeros(spins.shape[0], dtype=torch.complex128, device=spins.device)

    def ratio(g, A, D):
        f = torch.cosh(2 * D) + (g[:, None] * t) * torch.sinh(2 * D)
        return torch.exp(2 * g * A) * f.prod(dim=1)

    bonds = _bonds(case)
    for i, j, c in bonds:
        e += -0.25 * c * spins[:, i] * spins[:, j]
    if case["model"] == "tfim":
        for i in range(ns):
            e += -0.5 * COUPLINGS["tfim"]["hx"] * ratio(-spins[:, i], a[i], W[i])
        return e
    for i, j, c in bonds:
        e += -0.5 * c * ratio(-spins[:, i], a[i] - a[j], W[i] - W[j]) * (spins[:, i] != spins[:, j])
    return e


def _weights(case, seed):
    """Reweighting factors that sum to the number of rows (all ones when the case has none)."""
    g = torch.Generator(device="cuda").manual_seed(seed * 5 + 1)
    p = torch.exp(0.3 * torch.randn(case["rows"], generator=g, device="cuda", dtype=torch.float64))
    return (p / p.sum() * case["rows"]).to(torch.float32)


def _batch_models(case, seed):
    import pyqusolver_b200 as qb
    rng = np.random.default_rng([case["lo"], case["hi"], case["problems"]])
    L = rng.integers(case["lo"], case["hi"] + 1, size=case["problems"])
    hx = np.random.default_rng([seed, 13]).uniform(0.5, 1.5, size=case["problems"])
    return [qb.TransverseFieldIsing(qb.SquareLattice(1, int(n), 1, bc="pbc"), j=1.0, hx=float(h), hz=0.0)
            for n, h in zip(L, hx)]


def prepare(case, seed):
    import pyqusolver_b200 as qb
    from pyqusolver_b200.batch import NQSBatch
    from pyqusolver_b200.tdvp import TDVP
    torch.cuda.set_device(0)
    kind = case["kind"]
    if kind == "batch":
        B = NQSBatch(_batch_models(case, seed), alpha=case["alpha"], dtype="float32", s_numchains=case["chains"],
                     seeds=[(seed % 100000) * 1000 + b for b in range(case["problems"])], s_numsamples=case["samples"],
                     init_scale=case["scale"], warps_per_block=4, blocks_per_sm=8)
        B.sample()                                                           # burn-in
        return {"kind": kind, "batch": B, "shift": case["shift"],
                "params": [B.params(b).clone() for b in range(B.n_inst)]}
    ns, nh = case["lx"] * case["ly"], case["nh"]
    dtype = "complex64" if _is_complex(case) else "float32"
    kw = dict(dtype=dtype, seed=seed % 100000, alpha_rbm=nh / ns, s_upd_fun="LOCAL" if case["model"] == "tfim" else "EXCHANGE",
              s_initstate="RND" if case["model"] == "tfim" else "RND_FIXED", nparticles=ns // 2)
    if kind == "epoch":
        kw.update(s_numchains=case["chains"], s_numsamples=case["samples"], s_sweep_steps=ns)
    nqs = qb.NQS("rbm", _model(case), **kw)
    assert nqs.net.nh == nh
    params = _params(case, seed)
    nqs.set_params(params)
    st = {"kind": kind, "nqs": nqs, "params": params}
    st["tdvp"] = TDVP(rhs_prefactor=-1.0, sr_diag_shift=case.get("shift", 1e-3), sr_maxiter=1000,
                      sr_form_matrix=kind == "dense")
    if kind == "epoch":
        nqs.sampler.sample_bits(num_therm=0)                                 # chains that have already run
        return st
    spins = _spins(case, seed)
    st["bits"] = _pack(spins)
    if kind in ("update", "dense"):
        flat64 = nqs.net.flat.to(nqs.net.master_dtype)
        st["tanh"] = torch.tanh(_theta(flat64, spins, nh)).to(nqs.net.dtype).contiguous()
        st["eloc"] = _local_energy(case, flat64, spins).to(torch.complex64).contiguous()
        st["probs"] = _weights(case, seed) if case.get("weighted") else None
    if kind == "grad":
        g = torch.Generator(device="cuda").manual_seed(seed + 17)
        st["cot"] = torch.randn(case["rows"], generator=g, device="cuda", dtype=nqs.net.dtype)
    return st


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    from pyqusolver_b200 import device as dv
    kind = state["kind"]
    if kind == "batch":
        B = state["batch"]
        for b, p in enumerate(state["params"]):
            B.set_params(b, p)
        B.train_step(lr=RATE, diag_shift=state["shift"])
        return {"weights": B.flat, "eloc": B.eloc, "bits": B.sample_bits}
    nqs = state["nqs"]
    if kind == "epoch":
        nqs.set_params(state["params"])
        nqs.train_step(lr=RATE, tdvp=state["tdvp"])
        return {"weights": nqs.net.flat, "bits": nqs.sampler.last_sample_bits, "logpsi": nqs.sampler.last_sample_logpsi}
    if kind == "update":
        net = nqs.net
        x = state["tdvp"].solve(net, state["bits"], state["tanh"], state["eloc"], probs=state["probs"])
        flat, master = net.flat.clone(), net.master.clone()                  # the trial weights of a line search
        dv.param_update(flat, master, x, RATE)
        return {"weights": flat}
    if kind == "dense":
        return {"x": state["tdvp"].solve(nqs.net, state["bits"], state["tanh"], state["eloc"], probs=state["probs"])}
    if kind == "energy":
        return {"logpsi": nqs(state["bits"]), "eloc": nqs.local_energy(state["bits"])}
    if kind == "step":
        r = nqs.step(configs=state["bits"])
        return {"eloc": r.loss, "rows": r.grad_flat}
    lp, p = nqs.net.log_psi_autograd(state["bits"])
    lp.backward(state["cot"])
    return {"logpsi": lp.detach(), "grad": p.grad}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _sr_direction(case, flat, spins, t, eloc, wts):
    """Conjugate gradients on (O_c^H p O_c / n + shift) x = O_c^H p E_c / n in 64 bits, to 1e-13."""
    ns, nh, n = spins.shape[1], case["nh"], spins.shape[0]
    sg = spins.to(flat.dtype)
    p = torch.ones(n, dtype=torch.float64, device=spins.device) if wts is None else wts / wts.sum() * n

    def O(v):
        a, b, W = _split(v, ns, nh)
        return sg @ a + (t * (sg @ W + b)).sum(dim=1)

    def OH(u):
        q = t.conj() * u[:, None]
        return torch.cat([sg.T @ u, q.sum(dim=0), (sg.T @ q).reshape(-1)])

    def S(v):
        w = O(v)
        return OH(p * (w - (p * w).sum() / n)) / n + case["shift"] * v

    e = eloc if flat.is_complex() else eloc.real
    F = OH((p * (e - (p * e).sum() / n)).to(flat.dtype)) / n
    x, r = torch.zeros_like(F), F.clone()
    d, rr = r.clone(), torch.vdot(r, r).real
    stop = 1e-26 * rr
    for k in range(4000):
        Sd = S(d)
        al = rr / torch.vdot(d, Sd).real
        x += al * d
        r -= al * Sd
        new = torch.vdot(r, r).real
        d = r + (new / rr) * d
        rr = new
        if k % 16 == 15 and bool(rr <= stop):
            break
    return -x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("epoch", "batch"):
        return None                                                          # follows its own random chains
    ns, nh = case["lx"] * case["ly"], case["nh"]
    master = _params(case, seed)
    flat = master.to(torch.complex64 if _is_complex(case) else torch.float32).to(master.dtype)
    spins = _spins(case, seed)
    if kind == "energy":
        return {"logpsi": _log_psi(flat, spins, nh), "eloc": _local_energy(case, flat, spins)}
    if kind == "step":
        t = torch.tanh(_theta(flat, spins, nh))
        rows = torch.cat([spins.to(flat.dtype), t, (spins[:, :, None] * t[:, None, :]).reshape(spins.shape[0], -1)], dim=1)
        return {"eloc": _local_energy(case, flat, spins), "rows": rows}
    if kind == "grad":
        g = torch.Generator(device="cuda").manual_seed(seed + 17)
        u = torch.randn(case["rows"], generator=g, device="cuda",
                        dtype=torch.complex64 if _is_complex(case) else torch.float32).to(flat.dtype)
        q = torch.tanh(_theta(flat, spins, nh)).conj() * u[:, None]
        sg = spins.to(flat.dtype)
        return {"logpsi": _log_psi(flat, spins, nh),
                "grad": torch.cat([sg.T @ u, q.sum(dim=0), (sg.T @ q).reshape(-1)])}
    t = torch.tanh(_theta(flat, spins, nh))
    t = t.to(torch.complex64 if _is_complex(case) else torch.float32).to(flat.dtype)
    eloc = _local_energy(case, flat, spins).to(torch.complex64).to(torch.complex128)
    wts = _weights(case, seed).to(torch.float64) if case.get("weighted") else None
    x = _sr_direction(case, flat, spins, t, eloc, wts)
    return {"x": x} if kind == "dense" else {"weights": master + RATE * x}


# ------------------------------------------------------------------------------------------ what a pass cannot do without
ITERATIONS = 100          # CG iterations counted per solve: what a well-conditioned batch takes


def work(case):
    """Inputs read once and results written once; multiply-adds of the contractions and the psi ratios."""
    kind = case["kind"]
    if kind == "batch":
        ns = np.random.default_rng([case["lo"], case["hi"], case["problems"]]).integers(case["lo"], case["hi"] + 1,
                                                                                    size=case["problems"])
        nh, rows = case["alpha"] * ns, case["chains"] * case["samples"]
        P = ns + nh + ns * nh
        flops = rows * (ns * nh * 4.0 + ns * nh * 4.0 + ITERATIONS * 4.0 * ns * nh)
        return {"bytes": float((P * 16 + rows * (ns / 8 + 8 + nh * 4)).sum()), "flops": float(flops.sum())}
    ns, nh = case["lx"] * case["ly"], case["nh"]
    rows = case["chains"] * case["samples"] if kind == "epoch" else case["rows"]
    P, e, f = _n_params(ns, nh), (8 if _is_complex(case) else 4), (4 if _is_complex(case) else 1)
    moves = ns if case["model"] == "tfim" else len(_bonds(case))
    forward, ratios = 2.0 * ns * nh * (2 if _is_complex(case) else 1), 4.0 * f * moves * nh
    matvec = 4.0 * ns * nh * (2 if _is_complex(case) else 1) + 4.0 * f * nh
    if kind == "epoch":
        return {"bytes": rows * (ns / 8 + 8.0 + nh * e) + 3.0 * P * e,
                "flops": rows * (forward + ratios + ns * 4.0 * f * nh + ITERATIONS * matvec)}
    if kind == "update":
        return {"bytes": rows * (ns / 8 + 8.0 + nh * e) + 3.0 * P * e, "flops": rows * ITERATIONS * matvec}
    if kind == "dense":
        return {"bytes": rows * (ns / 8 + 8.0 + nh * e) + 2.0 * P * e,
                "flops": f * rows * float(P) ** 2 + f * float(P) ** 3 / 3}
    if kind == "energy":
        return {"bytes": rows * (ns / 8 + 8.0 + e) + float(P) * e, "flops": rows * (forward + ratios)}
    if kind == "step":
        return {"bytes": rows * (ns / 8 + 8.0 + float(P) * e), "flops": rows * (forward + ratios)}
    return {"bytes": rows * (ns / 8 + 2.0 * e) + 2.0 * P * e, "flops": rows * (forward + matvec / 2)}
