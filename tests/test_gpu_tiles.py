"""Register-tiled kernels at the edges of their tiles, against float64 (the float32 bar: 1e-5)."""

import numpy as np
import pytest
import torch

from oracle import lattice as olat, hamiltonian as oH, rbm as orbm, estimator as oest
import pyqusolver_b200 as qb
from pyqusolver_b200 import _lib, device as dv
from pyqusolver_b200.rbm import RBM
from pyqusolver_b200.tdvp import TDVP

pytestmark = pytest.mark.gpu


def _problem(cplx, ns, nh, n, scale, seed=3):
    net = RBM((ns,), n_hidden=nh, dtype="complex64" if cplx else "float32", seed=seed, init_scale=scale)
    rng = np.random.default_rng(seed)
    st = np.where(rng.random((n, ns)) < 0.5, 0.5, -0.5)
    p = orbm.RBMParams.from_flat(net.flat.cpu().numpy().astype(np.complex128 if cplx else np.float64), ns, nh)
    return net, st, dv.pack_states(st), p


# sites per staged slice (32), hidden units per pass (128) and per thread (4), samples per thread (1, 2, 4, 8) and
# per block; 1,184 and 9,500 rows reach the two- and eight-sample tiles of the real form
@pytest.mark.parametrize("cplx,ns,nh,n", [(False, 5, 3, 1), (True, 33, 129, 9), (False, 32, 128, 1185), (True, 31, 130, 2400),
                                           (False, 64, 5, 9500), (True, 3, 4, 4800), (False, 70, 260, 4750)])
def test_forward_tiles(cplx, ns, nh, n):
    net, st, bits, p = _problem(cplx, ns, nh, n, 0.05)
    th, tn, lp = dv.rbm_forward(net.flat, ns, nh, bits, theta=True)
    sg = np.where(st > 0, 1.0, -1.0)
    ref = orbm.theta(p, sg)
    tol = lambda x: 1e-5 * max(1.0, np.max(np.abs(x)))
    assert np.max(np.abs(th.cpu().numpy() - ref)) <= tol(ref)
    # tanh of a complex theta near a pole amplifies theta's rounding: checked at the path's own theta
    own = np.tanh(th.cpu().numpy().astype(ref.dtype))
    assert np.max(np.abs(tn.cpu().numpy() - own)) <= tol(own)
    d = lp.cpu().numpy() - orbm.log_psi(p, sg)
    assert np.max(np.abs(d.real)) <= tol(ref) * 10
    if cplx:
        assert np.max(np.abs(np.angle(np.exp(1j * d.imag)))) <= tol(ref) * 10
    _, t2, none = dv.rbm_forward(net.flat, ns, nh, bits, logpsi=False)
    assert none is None and torch.equal(t2, tn)


# units 32 apart and in a row, slices of 8 to 32 sites, two samples per thread and four, more than 256 sites
@pytest.mark.parametrize("cplx,ns,nh,n", [
    (False, 96, 64, 2400), (False, 97, 64, 1200), (False, 96, 65, 4800), (False, 8, 33, 1), (False, 48, 300, 2400),
    (False, 49, 140, 4800), (True, 41, 300, 2400), (False, 600, 40, 2400), (True, 523, 33, 1200), (False, 1, 1, 5000)])
def test_forward_of_few_sites_and_units(cplx, ns, nh, n):
    test_forward_tiles(cplx, ns, nh, n)


# moves per thread (4) and per block (32), units per renormalisation (16), samples per thread and block;
# scale 1.5: products that leave 2^+-8 and are renormalised
@pytest.mark.parametrize("lx,ly,model,cplx,nh,n,scale", [
    (3, 1, "tfim", False, 1, 1, 0.1), (17, 1, "tfim", False, 33, 70, 0.1), (65, 1, "tfim", False, 16, 4300, 0.1),
    (5, 3, "xxz", True, 17, 130, 0.1), (9, 9, "xxz", True, 31, 1300, 0.1), (7, 3, "j1j2", True, 48, 2500, 0.1),
    (33, 1, "tfim", False, 40, 257, 1.5), (4, 3, "j1j2", True, 40, 65, 1.0), (40, 1, "tfim", True, 20, 12000, 0.1)])
def test_local_energy_tiles(lx, ly, model, cplx, nh, n, scale):
    dim, ns = (2 if ly > 1 else 1), lx * ly
    L, OL = qb.SquareLattice(dim, lx, ly), olat.SquareLattice(dim, lx, ly)
    if model == "tfim":
        m, terms = qb.TransverseFieldIsing(L, j=1.0, hx=0.7, hz=0.3), oH.tfim_terms(OL, 1.0, 0.7, 0.3)
    elif model == "xxz":
        m, terms = qb.XXZ(L, jxy=-1.0, jz=-1.0), oH.xxz_terms(OL, -1.0, -1.0)
    else:
        m, terms = qb.J1J2Model(L, J1=-1.0, J2=-0.5), oH.j1j2_terms(OL, -1.0, -0.5)
    net, st, bits, p = _problem(cplx, ns, nh, n, scale / np.sqrt(ns))
    _, tn, _ = dv.rbm_forward(net.flat, ns, nh, bits, logpsi=False)
    h = dv.DeviceHamiltonian(m.lower())
    tables = dv.move_tables(net.flat, ns, nh, h.move_i, h.move_j, h.move_kind, move_major=False)
    e = dv.local_energy(net.flat, ns, nh, bits, tn, h, tables).cpu().numpy()
    rows = np.unique(np.linspace(0, n - 1, 40).astype(int))       # the full re-evaluation is the slow side
    ref = oest.local_energy_full(p, terms, st[rows])
    assert np.max(np.abs(e[rows] - ref)) <= 1e-5 * max(1.0, np.max(np.abs(ref)))
    assert np.all(np.isfinite(e))


# last chunks of 1 to 15 complex units
@pytest.mark.parametrize("lx,ly,model,nh,n", [(35, 1, "tfim", 1, 300), (6, 2, "xxz", 14, 9000), (5, 3, "j1j2", 18, 2500), (9, 1, "tfim", 47, 70)])
def test_local_energy_of_a_short_last_chunk(lx, ly, model, nh, n):
    test_local_energy_tiles(lx, ly, model, True, nh, n, 0.1)


# rows whose W blocks start on and off 16-byte boundaries (odd P, odd nh), fewer elements than one vector
@pytest.mark.parametrize("cplx,ns,nh,n", [(False, 1, 1, 3), (False, 5, 3, 7), (True, 4, 3, 5), (True, 7, 8, 2),
                                           (False, 33, 130, 4), (True, 20, 41, 9)])
def test_log_derivative_rows(cplx, ns, nh, n):
    net, st, bits, p = _problem(cplx, ns, nh, n, 0.2)
    _, tn, _ = dv.rbm_forward(net.flat, ns, nh, bits, logpsi=False)
    O = dv.log_derivatives(net.flat, ns, nh, bits, tn)
    sg = torch.as_tensor(np.where(st > 0, 1.0, -1.0)).cuda().to(tn.dtype)
    ref = torch.cat([sg, tn, (sg[:, :, None] * tn[:, None, :]).reshape(n, -1)], dim=1)
    assert torch.equal(O, ref)
    wide = torch.full((n, dv.n_params(ns, nh) + 3), 7.0, dtype=tn.dtype, device="cuda")       # rows of a wider array
    dv.log_derivatives(net.flat, ns, nh, bits, tn, out=wide)
    assert torch.equal(wide[:, :-3], ref) and bool((wide[:, -3:] == 7.0).all())


# narrow W rows as one run per sample (a warp or a block each), either form's last width, several blocks per sample
@pytest.mark.parametrize("cplx,ns,nh,n", [
    (False, 15, 15, 700), (False, 16, 15, 61), (True, 10, 9, 1201), (False, 300, 96, 1), (True, 300, 96, 2), (False, 2000, 97, 3),
    (True, 129, 97, 700), (False, 60, 4, 1300), (True, 2, 1, 5000)])
def test_log_derivative_rows_of_narrow_layers_and_few_samples(cplx, ns, nh, n):
    test_log_derivative_rows(cplx, ns, nh, n)


@pytest.mark.parametrize("dtype,ns,nh,n", [("float32", 5, 3, 1), ("float32", 63, 126, 700), ("complex64", 33, 40, 129)])
def test_forward_without_wait_is_the_forward(dtype, ns, nh, n):
    net = RBM((ns,), n_hidden=nh, dtype=dtype, seed=ns, init_scale=0.1)
    bits = dv.pack_states(np.where(np.random.default_rng(nh).random((n, ns)) < 0.5, 0.5, -0.5))
    tn, status = dv.rbm_tanh_nowait(net.flat, ns, nh, bits)
    _, ref, _ = dv.rbm_forward_step(net.flat, ns, nh, bits, theta=False, tanh=True, logpsi=False)
    assert torch.equal(tn, ref)
    assert status is None or int(status.item()) == 0


def test_a_failed_forward_updates_nothing(monkeypatch):
    model = qb.TransverseFieldIsing(qb.SquareLattice(1, 8), j=1.0, hx=1.0, hz=0.0)
    nqs = qb.NQS("rbm", model, alpha=1.0, dtype="float32", seed=1, s_numchains=64, s_numsamples=4)
    tdvp = TDVP(rhs_prefactor=-1.0, sr_diag_shift=1e-2)
    nqs.train_step(lr=0.01, tdvp=tdvp)
    weights, solution = nqs.net.flat.clone(), tdvp._solution
    real = dv.rbm_tanh_nowait
    monkeypatch.setattr(dv, "rbm_tanh_nowait", lambda *a: (real(*a)[0], torch.ones(1, dtype=torch.int32, device="cuda")))
    with pytest.raises(_lib.QESError) as err:
        nqs.train_step(lr=0.01, tdvp=tdvp)
    assert err.value.code == _lib.QES_ERR_TIMEOUT
    assert torch.equal(nqs.net.flat, weights) and tdvp._solution is solution


# unit groups of 16 (complex 8), 64 sites per pass, 16 samples per step and 512 per split; past 512 sites the CUDA-core form
@pytest.mark.parametrize("cplx,ns,nh,n", [(False, 1, 1, 1), (True, 1, 1, 17), (False, 64, 16, 512), (True, 65, 9, 513),
                                          (False, 33, 17, 1030), (True, 512, 8, 40), (False, 513, 3, 40),
                                          (False, 130, 140, 31)])
def test_logpsi_vjp_at_tile_edges(cplx, ns, nh, n):
    net, st, bits, _ = _problem(cplx, ns, nh, n, 0.2)
    _, tn, _ = dv.rbm_forward(net.flat, ns, nh, bits, tanh=True, logpsi=False)
    rng = np.random.default_rng(n)
    g = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    out = dv.logpsi_vjp(net.flat, ns, nh, bits, tn, torch.tensor(g, device="cuda")).cpu().numpy()
    t, s, u = tn.cpu().numpy().reshape(n, nh), 2.0 * st, g if cplx else g.real
    t, u = t.astype(np.complex128 if cplx else np.float64), u.astype(np.complex128 if cplx else np.float64)
    q = t.conj() * u[:, None]
    ref = np.concatenate([s.T @ u, q.sum(0), (s.T @ q).reshape(-1)])
    # products rounded once (complex: three times) and float32 sums of 512 terms: a few 2^-24 of the terms' norm, which the
    # random signs leave as the result's
    assert np.linalg.norm(out - ref) <= 1e-6 * np.linalg.norm(ref)


# the last split's samples end within, at and past a warp's share of 64 for g_a
@pytest.mark.parametrize("cplx,ns,nh,n", [(True, 40, 9, 64), (False, 70, 9, 65), (True, 33, 9, 577), (False, 400, 20, 3)])
def test_logpsi_vjp_of_few_samples(cplx, ns, nh, n):
    test_logpsi_vjp_at_tile_edges(cplx, ns, nh, n)


# one sample's infinity or NaN, or the largest float, leaves the same entries finite, infinite and NaN as the CUDA-core form
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
def test_logpsi_vjp_of_infinities(value):
    net, st, bits, _ = _problem(False, 20, 24, 70, 0.2)
    _, tn, _ = dv.rbm_forward(net.flat, 20, 24, bits, tanh=True, logpsi=False)
    g = torch.ones(70, dtype=torch.complex64, device="cuda")
    g[33] = value
    out = dv.logpsi_vjp(net.flat, 20, 24, bits, tn, g)
    _lib.set_sr_impl(_lib.SR_IMPL_CUDA_CORES)
    try:
        ref = dv.logpsi_vjp(net.flat, 20, 24, bits, tn, g)
    finally:
        _lib.set_sr_impl(0)
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.isinf(), ref.isinf())
    ok = ref.isfinite()
    assert (out[ok] - ref[ok]).abs().max() <= 1e-6 * ref[ok].abs().max() if ok.any() else True
    assert torch.equal(out[ref.isinf()], ref[ref.isinf()])


# flip of site 0: the first 16 factors multiply to 2^8.5, the next 16 to 2^grow; the visible bias brings the ratio back into range.  One to
# four samples per thread.
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [40, 3000, 30000])
@pytest.mark.parametrize("grow", [100.0, 115.0, 121.6, 126.6])
def test_local_energy_of_products_near_the_float_range(cplx, n, grow):
    ns, nh = 33, 32
    model = qb.TransverseFieldIsing(qb.SquareLattice(1, ns), j=1.0, hx=0.7, hz=0.0)
    rng = np.random.default_rng(int(grow))
    W = 0.01 * rng.normal(size=(ns, nh))
    W[0, :16], W[0, 16:] = 0.5 * 8.5 / 16 * np.log(2), 0.5 * grow / 16 * np.log(2)
    a = np.zeros(ns)
    a[0] = -30.0 * np.log(2)
    flat = torch.as_tensor(np.concatenate([a, np.full(nh, 80.0), W.reshape(-1)])).cuda()
    flat = flat.to(torch.complex64 if cplx else torch.float32)
    st = np.where(rng.random((n, ns)) < 0.5, 0.5, -0.5)
    st[:, 0] = -0.5
    bits = dv.pack_states(st)
    tn = torch.ones((n, nh), dtype=flat.dtype, device="cuda")                 # tanh(80 + ...) in float32
    h = dv.DeviceHamiltonian(model.lower())
    tables = dv.move_tables(flat, ns, nh, h.move_i, h.move_j, h.move_kind, move_major=False)
    e = dv.local_energy(flat, ns, nh, bits, tn, h, tables).cpu().numpy()
    # with tanh = 1 the ratio of a flip is exp(-2 sigma (a + sum_m W_m)), from the float32 parameters; site 0's is 2^48 and
    # more, beside which the other terms vanish
    f = flat.real.double().cpu().numpy()
    ref = float(h.move_coef[0]) * np.exp(2.0 * (f[0] + f[ns + nh:ns + 2 * nh].sum()))
    # 32 factors, each rounded once from tables with a relative error of up to (1 + 2 W) 2^-23, W <= 2.8
    assert np.all(np.abs(e - ref) <= 32 * 7 * 2.0 ** -23 * abs(ref)), (e[:4], ref)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_local_energy_and_forward_of_infinities(cplx, value):
    """An infinity or a NaN in one sample's T (one bias) reaches that sample (that unit) alone."""
    ns, nh, n = 33, 40, 300
    net, st, bits, _ = _problem(cplx, ns, nh, n, 0.1)
    model = qb.TransverseFieldIsing(qb.SquareLattice(1, ns), j=1.0, hx=0.7, hz=0.0)
    _, tn, _ = dv.rbm_forward(net.flat, ns, nh, bits, logpsi=False)
    h = dv.DeviceHamiltonian(model.lower())
    tables = dv.move_tables(net.flat, ns, nh, h.move_i, h.move_j, h.move_kind, move_major=False)
    ref = dv.local_energy(net.flat, ns, nh, bits, tn, h, tables)
    bad = tn.clone()
    bad[77, 20] = value
    e = dv.local_energy(net.flat, ns, nh, bits, bad, h, tables)
    others = torch.arange(n, device="cuda") != 77
    assert torch.equal(e[others], ref[others]) and not bool(e[77].isfinite())
    flat = net.flat.clone()
    flat[ns + 20] = value
    _, t2, lp = dv.rbm_forward(flat, ns, nh, bits)
    units = torch.arange(nh, device="cuda") != 20
    assert torch.equal(t2[:, units], tn[:, units])
    if np.isnan(value):
        assert bool(t2[:, 20].isnan().all()) and bool(lp.isnan().all())
    elif not cplx:
        assert bool((t2[:, 20] == np.sign(value)).all()) and bool((lp == np.inf).all())


def test_log_derivative_rows_past_a_grid():
    """More rows than one grid holds (2^31 - 1): 43 GB for the smallest network."""
    n = 2 ** 31 + 5
    bits = torch.zeros((n, 1), dtype=torch.int32, device="cuda")
    tn = torch.full((n, 1), 0.25, dtype=torch.float32, device="cuda")
    probe = [0, 2 ** 30 - 1, 2 ** 30, 2 ** 31 - 2, 2 ** 31 - 1, 2 ** 31, n - 1]
    for k, r in enumerate(probe):
        bits[r] = k % 2
        tn[r] = 0.5 + k
    flat = torch.zeros(3, dtype=torch.float32, device="cuda")
    O = torch.full((n, 3), 7.0, dtype=torch.float32, device="cuda")
    dv.log_derivatives(flat, 1, 1, bits, tn, out=O)
    for k, r in enumerate(probe):
        sg = 1.0 if k % 2 else -1.0
        assert O[r].tolist() == [sg, 0.5 + k, sg * (0.5 + k)]
    for r0 in range(0, n, 2 ** 29):                                            # every row is written
        assert not bool((O[r0:r0 + 2 ** 29, 0] == 7.0).any())
    del O, tn, bits
    torch.cuda.empty_cache()


@pytest.mark.parametrize("forward_failed", [True, False])
def test_a_failed_forward_is_reported_before_what_the_solve_makes_of_it(monkeypatch, forward_failed):
    model = qb.TransverseFieldIsing(qb.SquareLattice(1, 8), j=1.0, hx=1.0, hz=0.0)
    nqs = qb.NQS("rbm", model, alpha=1.0, dtype="float32", seed=1, s_numchains=64, s_numsamples=4)
    tdvp = TDVP(rhs_prefactor=-1.0, sr_diag_shift=1e-2)
    nqs.train_step(lr=0.01, tdvp=tdvp)
    weights, info = nqs.net.flat.clone(), tdvp.last_info
    real = dv.rbm_tanh_nowait
    status = torch.full((1,), int(forward_failed), dtype=torch.int32, device="cuda")
    monkeypatch.setattr(dv, "rbm_tanh_nowait", lambda *a: (real(*a)[0], status))

    def solve(*a, **k):
        tdvp.last_info = {"iterations": -1}
        raise _lib.QESError(_lib.QES_ERR_SIZE, "not positive definite")

    monkeypatch.setattr(tdvp, "solve", solve)
    with pytest.raises(_lib.QESError) as err:
        nqs.train_step(lr=0.01, tdvp=tdvp)
    assert err.value.code == (_lib.QES_ERR_TIMEOUT if forward_failed else _lib.QES_ERR_SIZE)
    assert torch.equal(nqs.net.flat, weights)
    if forward_failed:
        assert tdvp.last_info is info
