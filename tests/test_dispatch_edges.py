"""The kernels' dispatch rules at the sizes where they switch: each side of a
size rule, remainders of its tiles and the ends of its range, against the
oracle or a plain FP64 restatement."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth
from oracle import pyoracle as O
from tests import parity as P

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


@pytest.mark.parametrize("n", [2, 31, 33, 64, 65])
def test_quad_traces_one_warp_or_one_block_a_group(cuda, n):
    """trace_quads gives a group one warp up to Nev = 64 and a block above."""
    nt = 2
    prop = synth.make_prop(nt, n, seed=500 + n)
    rng = np.random.default_rng(501 + n)
    mom2 = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1)
    got = api.run_contract_sigma(_dev(prop, cuda), _dev(mom2, cuda), engine="split").cpu().numpy()
    rc = [O.sigma_row(prop, np.ascontiguousarray(mom2), tf) for tf in range(nt)]
    P.entrywise(got, np.stack([c for _, c in rc]), 1e-9, np.stack([P.sigma_rows_abs(r) for r, _ in rc]),
                "sigma Nev=%d" % n)


@pytest.mark.parametrize("n,nrows", [(7, 9), (20, 300), (65, 900)])
def test_quad_traces_cover_large_components(cuda, n, nrows):
    """Random tables whose traces link many blocks, sparse to dense: every trace is
    in one quad, whatever blocks it shares.  One row an output, so a trace may cancel:
    2^-40 of its products' Frobenius norms (the float-float products carry 2^-44 of
    their rows' and columns' largest entries), beside the engine's 1e-9."""
    nt, nphi = 2, 3
    rng = np.random.default_rng(800 + nrows)
    prop = synth.make_prop(nt, n, seed=801 + n)
    phi = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(nphi)], axis=1)
    rows = np.concatenate([rng.integers(0, 4, (nrows, 4)), rng.integers(0, nphi, (nrows, 2))], axis=1).astype(np.int16)
    coef = rng.integers(1, 3, (nrows, 2)).astype(np.float32)
    oi = np.arange(nrows, dtype=np.int32)
    got = api.twosided(_dev(prop, cuda), _dev(phi, cuda), rows, coef, oi, nrows, engine="split").cpu().numpy()
    want = np.stack([O.twosided_rows(prop[tf], phi, rows, coef, tf, 0, nt) for tf in range(nt)])
    a, b, c, d, L, R = rows.T
    norm = lambda x: np.linalg.norm(x, axis=(-2, -1))
    ab = np.abs(coef[:, 0] + 1j * coef[:, 1]) * np.array(
        [[norm(prop[tf, ti, c, d] @ phi[ti, L]) * norm(phi[tf, R] @ prop[tf, ti, a, b]) for ti in range(nt)]
         for tf in range(nt)])
    P.entrywise(got, want, 1e-9, ab, "random table of %d rows, Nev=%d" % (nrows, n), floor=2.0 ** -40)


@pytest.mark.parametrize("nt,n", [(1, 1), (5, 11), (3, 12), (22, 37), (64, 100), (200, 9)])
def test_loop_unity_cluster_sizes(cuda, nt, n):
    """One CTA a time slice up to a cluster of 8, ragged element ranges; per
    entry to the FP64 rounding floor of its 4 rows of Nev^2 terms."""
    rng = np.random.default_rng(600 + n)
    diag = rng.normal(size=(nt, 4, 4, n, n)) + 1j * rng.normal(size=(nt, 4, 4, n, n))
    mom = rng.normal(size=(nt, n, n)) + 1j * rng.normal(size=(nt, n, n))
    got = api.run_contract_loop_unity(_dev(diag, cuda), _dev(mom, cuda)).cpu().numpy()
    wide = np.clongdouble
    ref = np.einsum("tssij,tji->t", diag.astype(wide), mom.astype(wide)).astype(complex)
    # each sum adds at most Nev^2 / 128 + 11 rounded terms in sequence
    terms = np.einsum("tssij,tji->t", np.abs(diag), np.abs(mom))
    assert np.all(np.abs(got - ref) <= 2.0 ** -53 * (n * n / 128 + 16) * terms)


@pytest.mark.parametrize("nev", [1, 33, 51])
def test_elementals_pieces_and_reversed_momenta(cuda, nev):
    """K long enough for two pieces, tiles with remainders at both tile edges;
    momenta that are their own reverse (0, and half the lattice), reversed
    pairs, a pair reversed only modulo the lattice, repeats and one alone."""
    from oracle import elementals as E
    nt, nx, ny, nz = 1, 8, 6, 8
    moms = [(1, 0, 0), (0, 0, 0), (-1, 0, 0), (4, 3, 0), (7, 6, 8), (1, 2, -1), (1, 0, 0), (0, 0, 0)]
    V, U = synth.make_eigvecs(nt, nev, nx, ny, nz, 700 + nev), synth.make_links(nt, nx, ny, nz, 701)
    ref = E.elementals(V, moms, U)
    got = api.elementals(_dev(V, cuda), moms, links=_dev(U, cuda)).cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    plain = api.elementals(_dev(V, cuda), moms).cpu().numpy()
    assert np.abs(plain[:, 0] - ref[:, 0]).max() <= 1e-12 * np.abs(ref[:, 0]).max()


@pytest.mark.parametrize("n,rhopi,tri,nset", [(9, True, True, 11), (37, True, False, 12), (20, False, True, 2),
                                              (8, True, True, 20)])
def test_momentum_sets_sink_form(cuda, n, rhopi, tri, nset):
    """rho -> pi pi and triangle over enough sets that the sink operators' products
    replace the sets' (one Gram product per t_src), at ragged Nev, for the outputs
    alone and together, repeated sets among them, over a t_sink range."""
    from tests.test_parity_chains import SPLIT_TOL, ref_rhopi, ref_triangle
    nt, tr = 4, (1, 4)
    prop = synth.make_prop(nt, n, seed=800 + n, decay=0.25)
    moms = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0)]
    phis = synth.make_phi_momenta(nt, n, moms, seed=801 + n)
    rng = np.random.default_rng(802 + n)
    mom5 = np.ascontiguousarray(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1))
    mom2 = np.ascontiguousarray(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1))
    sets = [(k % 5, (k // 5 + k) % 5) for k in range(nset)] + [(0, 0)]
    tp = _dev(prop, cuda)
    got = api.run_contract_rhopi_sigmapi_sets(tp[tr[0]:tr[1]].contiguous(), api.prop_diag(tp),
                                              _dev(np.stack([phis[p] for p in moms], axis=1), cuda), sets,
                                              _dev(mom5, cuda), _dev(mom2, cuda), engine="split", tf_range=tr,
                                              rhopi=rhopi, triangle=tri)
    for k, (a, b) in enumerate(sets):
        pa, pb = phis[moms[a]], phis[moms[b]]
        for idir in range(3 if rhopi else 0):
            ref, ab = ref_rhopi(prop, pa, pb, mom5, idir, range(*tr))
            P.entrywise(got["rhopi"][k, idir].cpu().numpy(), ref, SPLIT_TOL, ab, "set %d idir %d" % (k, idir))
        if tri:
            ref, ab = ref_triangle(prop, pa, pb, mom2, range(*tr))
            P.entrywise(got["triangle"][k].cpu().numpy(), ref, SPLIT_TOL, ab, "set %d triangle" % k)


@pytest.mark.parametrize("engine,tol", [("fp64", 1e-11), ("split", 1e-8)])
@pytest.mark.parametrize("n,iso", [(1, 0), (33, 1), (7, 0), (129, 0)])
def test_profile_gradients_block_form(cuda, n, iso, engine, tol):
    """rho and pi pi profile gradients for arbitrary complex weights -- several t_sink
    a t_src and the reverse, pairs on the time diagonal, single slots, outputs of
    every operator pair -- with four different elementals, against autograd; Nev
    129 takes the tiled diagonal kernel (FP64 engine only)."""
    from contractions_code_scattering_gb300 import adjoint
    from oracle import torch_ref as R
    if n > 128 and engine == "split":
        pytest.skip("the split engine takes Nev <= 128")
    nt = 2 if n > 128 else 4
    prop = synth.make_prop(nt, n, seed=900 + n)
    rng = np.random.default_rng(901 + n)
    mom5 = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1)
    ps = [synth.make_phi_random(nt, n, rng) for _ in range(4)]
    f = adjoint.default_profile(n, seed=902)
    z = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
    wr, wp = np.zeros((nt, nt, 48), complex), np.zeros((nt, nt, 5), complex)
    if n <= 33:
        wr[0, 1], wr[2, 1, 5], wr[1, 1, 47], wr[1, 0, 3:9] = z(48), z(), z(), z(6)
        wp[0, 1], wp[3, 1], wp[2, 2], wp[0, 2, 4], wp[1, 3, 2] = z(5), z(5), z(5), z(), z()
    else:
        wr[0, 1, :2], wp[0, 1] = z(2), z(5)
    dp, df = _dev(prop, cuda), _dev(f, cuda)
    rho, gr = api.rho_profile_vjp(dp, _dev(mom5, cuda), df, _dev(wr, cuda), engine=engine)
    pipi, gp = api.pipi_profile_vjp(dp, *[_dev(p, cuda) for p in ps], df, _dev(wp, cuda), iso, engine=engine)
    ft = torch.tensor(f, requires_grad=True)
    tp = torch.from_numpy(prop)
    m5 = R.profiled(ft, torch.from_numpy(np.ascontiguousarray(mom5)))
    pr = tuple(R.profiled(ft, torch.from_numpy(p)) for p in ps)
    ref_r, ref_p, lr, lp = np.zeros_like(wr), np.zeros_like(wp), 0.0, 0.0
    for tf in range(nt):
        for ti in range(nt):
            on = np.flatnonzero(wr[tf, ti])
            if len(on):
                v = R.rho_pair(tp, m5, tf, ti, [int(o) for o in on])
                ref_r[tf, ti, on] = v.detach().numpy()
                lr = lr + (torch.from_numpy(wr[tf, ti, on]) * v).real.sum()
            if wp[tf, ti].any():
                v = R.pipi_pair(tp, pr, tf, ti, iso)
                ref_p[tf, ti] = v.detach().numpy()
                lp = lp + (torch.from_numpy(wp[tf, ti]) * v).real.sum()
    for got, ref, loss, g in ((rho, ref_r, lr, gr), (pipi, ref_p, lp, gp)):
        got, g = got.cpu().numpy(), g.cpu().numpy()
        assert np.all(got[ref == 0] == 0)
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
        want = torch.autograd.grad(loss, ft, retain_graph=True)[0].numpy()
        assert np.abs(g - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("n", [1, 31, 64, 65])
def test_profile_sums_tile_edges(cuda, n):
    """The gradients' sums over pairs of blocks take tiles of Nev / ceil(Nev / 32): one
    and several tiles, whole and ragged, against autograd; 1e-11 as for the block form."""
    from contractions_code_scattering_gb300 import adjoint
    from oracle import torch_ref as R
    nt, on = 2, [0, 9, 47]
    prop = synth.make_prop(nt, n, seed=950 + n)
    rng = np.random.default_rng(951 + n)
    mom5 = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1)
    f = adjoint.default_profile(n, seed=952)
    w = np.zeros((nt, nt, 48), complex)
    w[1, 0, on] = rng.normal(size=3) + 1j * rng.normal(size=3)
    got, g = api.rho_profile_vjp(_dev(prop, cuda), _dev(mom5, cuda), _dev(f, cuda), _dev(w, cuda), engine="fp64")
    ft = torch.tensor(f, requires_grad=True)
    v = R.rho_pair(torch.from_numpy(prop), R.profiled(ft, torch.from_numpy(np.ascontiguousarray(mom5))), 1, 0, on)
    loss = (torch.from_numpy(w[1, 0, on]) * v).real.sum()
    want = torch.autograd.grad(loss, ft)[0].numpy()
    ref = v.detach().numpy()
    assert np.abs(got.cpu().numpy()[1, 0, on] - ref).max() <= 1e-11 * np.abs(ref).max()
    assert np.abs(g.cpu().numpy() - want).max() <= 1e-11 * np.abs(want).max()


@pytest.mark.parametrize("n", [48, 49, 52, 53, 56, 57, 72])
def test_packed_tail_chunks(cuda, n):
    """Nev whose last chunk of 16 k holds 1 to 4, 5 to 8 or more valid ones (4, 2 and
    1 slice pairs an MMA): standard products to 1e-11 of their largest entry (45-bit
    operands), complex128 ones (one and four terms) through the triangle."""
    from tests.test_parity_chains import SPLIT_TOL, ref_triangle
    rng = np.random.default_rng(970 + n)
    x, y = (rng.normal(size=(2, n, n)) + 1j * rng.normal(size=(2, n, n)) for _ in range(2))
    got = api.zgemm_batched(_dev(x, cuda), _dev(y, cuda), engine="split").cpu().numpy()
    ref = x @ y
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    nt = 2
    prop = synth.make_prop(nt, n, seed=971 + n)
    pa, pb = synth.make_phi_random(nt, n, rng), synth.make_phi_random(nt, n, rng)
    mom2 = np.ascontiguousarray(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1))
    tp = _dev(prop, cuda)
    got = api.run_contract_rhopi_sigmapi_sets(tp, api.prop_diag(tp), _dev(np.stack([pa, pb], axis=1), cuda), [(0, 1)],
                                              _dev(np.zeros((nt, 5, n, n), complex), cuda), _dev(mom2, cuda),
                                              engine="split", tf_range=(0, nt), rhopi=False, triangle=True)
    tri = got["triangle"][0].cpu().numpy()
    want, ab = ref_triangle(prop, pa, pb, mom2)
    P.entrywise(tri, want, SPLIT_TOL, ab, "triangle Nev=%d" % n)


@pytest.mark.parametrize("tol", [1e-12, 1e-14])
def test_set_recomputation_in_two_steps(cuda, tol):
    """Set calls recompute flagged units with FP64 traces on the split engine, and what
    is still flagged on the FP64 engine: tolerances that flag some and most entries,
    against the FP64 engine's set call, per entry as the engine's default asks."""
    from contractions_code_scattering_gb300._lib import check, lib
    nt, n, tr = 4, 21, (1, 4)
    prop = synth.make_prop(nt, n, seed=990, decay=0.25)
    rng = np.random.default_rng(991)
    phi = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1)
    mom5 = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1)
    mom2 = np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1)
    sets = [(a, b) for a in range(5) for b in range(5)]
    tp = _dev(prop, cuda)
    run = lambda engine: api.run_contract_rhopi_sigmapi_sets(
        tp[tr[0]:tr[1]].contiguous(), api.prop_diag(tp), _dev(phi, cuda), sets, _dev(mom5, cuda), _dev(mom2, cuda),
        engine=engine, tf_range=tr, rhopi=True, triangle=True)
    ref = run("fp64")
    check(lib().ctr_split_set_refine(tol))
    try:
        got = run("split")
        assert lib().ctr_split_refined() > 0
    finally:
        check(lib().ctr_split_set_refine(1e-9))
    for k in ("rhopi", "triangle"):
        want = ref[k].cpu().numpy()
        P.entrywise(got[k].cpu().numpy(), want, 1e-9, np.abs(want), k)
