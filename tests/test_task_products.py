"""Accuracy of the complex128 split products.  Six slices without the pairs i + j > 5 of
Gaussian operands at full scale leave 7.5e-16 of a product's root mean square, whatever
its length (NumPy emulation with exact sums); the tests allow twice that."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth
from contractions_code_scattering_gb300._lib import check, lib

pytestmark = pytest.mark.gpu
WIDE = np.clongdouble
RMS = 1.5e-15


def _dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _dag(x):
    return x.conj().swapaxes(-2, -1)


def _rms(got, ref):
    return float(np.sqrt((np.abs(got.astype(WIDE) - ref) ** 2).mean() / (np.abs(ref) ** 2).mean()))


def _tasks(x, y, nterm, cuda, ad, bd):
    """sum_q op(x_q) op(y_q) on the split engine for operands given as op(x), op(y), and the wide reference."""
    got = api.zgemm_tasks(_dev(_dag(x) if ad else x, cuda), _dev(_dag(y) if bd else y, cuda),
                          [(list(range(nterm)), list(range(nterm)), 0)], a_dagger=ad, b_dagger=bd, engine="split")
    return got.cpu().numpy()[0], sum(np.matmul(x[q].astype(WIDE), y[q].astype(WIDE)) for q in range(nterm))


@pytest.mark.parametrize("n,nterm", [(128, 1), (33, 4), (43, 3), (65, 2), (100, 4), (128, 4)])
@pytest.mark.parametrize("ad,bd", [(False, False), (True, True)])
def test_products_over_128_terms_of_k(cuda, n, nterm, ad, bd):
    """Products of 128 k and of 129 to 512 (drained in pieces): Gaussian operands to the
    same error, and operands near full scale whose products all add up, where the first
    level is largest: to 4 roundings."""
    rng = np.random.default_rng(400 + n)
    x, y = (rng.normal(size=(nterm, n, n)) + 1j * rng.normal(size=(nterm, n, n)) for _ in range(2))
    got, ref = _tasks(x, y, nterm, cuda, ad, bd)
    assert _rms(got, ref) <= RMS
    x, y = (rng.uniform(0.9, 1.0, (nterm, n, n)) * (1 + s) for s in (1j, -1j))
    got, ref = _tasks(x, y, nterm, cuda, ad, bd)
    assert np.abs(got.astype(WIDE) - ref).max() <= 2.0 ** -51 * np.abs(ref).max()


@pytest.mark.parametrize("n", [49, 50, 51, 52, 53, 54, 56, 57])
@pytest.mark.parametrize("nterm", [1, 4])
@pytest.mark.parametrize("ad,bd", [(False, False), (True, True)])
def test_packed_tail_products(cuda, n, nterm, ad, bd):
    """Operands that live in the last chunk of 16 k alone, with 1 to 16 of them valid: no
    slice pair of a packed tail is lost among the other chunks' products."""
    rng = np.random.default_rng(450 + n)
    x, y = (rng.normal(size=(nterm, n, n)) + 1j * rng.normal(size=(nterm, n, n)) for _ in range(2))
    first = 16 * ((nterm * n - 1) // 16)
    x *= (np.arange(nterm * n) >= first).reshape(nterm, 1, n)
    got, ref = _tasks(x, y, nterm, cuda, ad, bd)
    assert _rms(got, ref) <= RMS


@pytest.mark.parametrize("n,tail", [(32, False), (49, True), (50, True), (53, True), (57, True)])
def test_stacked_products(cuda, n, tail):
    """The block grids' form of the same through the triangle: with P1 = P2 = 1 its X =
    tau G tau(t, t) is one four-term product, of which a sink operator with one entry
    takes a row; tail: tau(t, t) has rows in the last chunk alone.  The single products
    before and behind it copy tau to 2e-16.  Above 128 k the chain calls' operands halve
    their leading digit: four times the error, 3e-15."""
    nt = 4
    rng = np.random.default_rng(480 + n)
    prop = synth.make_prop(nt, n, seed=481 + n)
    diag = rng.normal(size=(nt, 4, 4, n, n)) + 1j * rng.normal(size=(nt, 4, 4, n, n))
    if tail:
        diag *= (np.arange(4 * n) >= 16 * ((4 * n - 1) // 16)).reshape(4, 1, n, 1)
    one = np.broadcast_to(np.eye(n, dtype=complex), (nt, n, n))
    mom2 = np.zeros((nt, 2, n, n), complex)
    mom2[:, 0, 1, n - 1] = mom2[:, 1, n // 2, 0] = 1.0
    check(lib().ctr_split_set_refine(0.0))
    try:
        tri = api.run_contract_sigmapi(_dev(prop, cuda), _dev(diag, cuda), _dev(one, cuda), _dev(one, cuda),
                                       _dev(mom2, cuda), engine="split", tf_range=(0, nt))[1].cpu().numpy()
    finally:
        check(lib().ctr_split_set_refine(1e-9))
    g5 = np.array([1.0, 1.0, -1.0, -1.0])
    ref = np.zeros((nt, nt, 2), WIDE)
    for tf in range(nt):
        for k, (i, j) in enumerate(((1, n - 1), (n // 2, 0))):
            # Op^dag tau has the one row j: tau's row i
            row = prop[tf, :, :, :, j].astype(WIDE) * g5[:, None]
            x = np.einsum("taki,tkbij->tabj", row, diag.astype(WIDE))
            ref[tf, :, k] = np.einsum("tabj,tabj,a->t", x, prop[tf, :, :, :, i].conj().astype(WIDE), g5)
    assert _rms(tri, ref) <= (2e-15 if 4 * n <= 128 else 6e-15)


@pytest.mark.parametrize("n", [40, 100])
def test_pipi_gradient_products_at_full_scale(cuda, n):
    """The pi pi gradient's block form (six products one after another, two of them of four
    terms): values within twice 6^(1/2) product errors of the FP64 engine's, as root mean
    squares over 36 pairs and the five diagrams."""
    nt = 6
    rng = np.random.default_rng(490 + n)
    prop = _dev(synth.make_prop(nt, n, seed=491 + n, decay=0.0), cuda)
    ps = [_dev(synth.make_phi_random(nt, n, rng), cuda) for _ in range(4)]
    f = torch.ones(n, dtype=torch.float64, device=cuda)
    w = _dev(rng.normal(size=(nt, nt, 5)) + 1j * rng.normal(size=(nt, nt, 5)), cuda)
    v, g = {}, {}
    for e in ("fp64", "split"):
        v[e], g[e] = api.pipi_profile_vjp(prop, *ps, f, w, 0, engine=e)
    rms = lambda x: (x.abs() ** 2).mean(dim=(0, 1)).sqrt()
    err = (rms(v["split"] - v["fp64"]) / rms(v["fp64"])).square().mean().sqrt()
    assert err <= 4e-15
    assert ((g["split"] - g["fp64"]).square().mean() / g["fp64"].square().mean()).sqrt() <= 4e-15
