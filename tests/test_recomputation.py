"""The split engine's recomputation: what its error scales have to flag, and that
flagged units get the FP64 engine's values."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth
from contractions_code_scattering_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


@pytest.mark.parametrize("tol", [1e-12, 1e-14])
def test_flagged_set_units_take_fp64_values(cuda, tol):
    """rho -> pi pi / sigma -> pi pi set calls: every recomputed entry is bitwise the FP64
    engine's (at these tolerances some, and most, of the units are recomputed)."""
    nt, n, tr = 4, 21, (1, 4)
    prop = synth.make_prop(nt, n, seed=990, decay=0.25)
    rng = np.random.default_rng(991)
    phi, mom5, mom2 = (np.stack([synth.make_phi_random(nt, n, rng) for _ in range(k)], axis=1) for k in (5, 5, 2))
    sets = [(a, b) for a in range(5) for b in range(5)]
    tp = _dev(prop, cuda)
    run = lambda engine: api.run_contract_rhopi_sigmapi_sets(
        tp[tr[0]:tr[1]].contiguous(), api.prop_diag(tp), _dev(phi, cuda), sets, _dev(mom5, cuda), _dev(mom2, cuda),
        engine=engine, tf_range=tr, rhopi=True, triangle=True)
    ref = run("fp64")
    check(lib().ctr_split_set_refine(tol))
    try:
        got = run("split")
        refined = lib().ctr_split_refined()
    finally:
        check(lib().ctr_split_set_refine(1e-9))
    same = sum(int((got[k] == ref[k]).sum()) for k in ("rhopi", "triangle", "hor_fish"))
    assert refined > 0 and same >= refined


@pytest.mark.parametrize("sets_call", [False, True])
def test_cancelling_twins_are_flagged(cuda, sets_call):
    """I = 0 star and fish where tau Phi tau^dagger cancels over its spin sum: with
    tau_{a1} = tau_{a0} S, tau_{a3} = tau_{a2} S and S Phi S = -Phi up to 1e-8 of Phi,
    the twin traces are 1e-8 of their terms, so both have to be recomputed."""
    nt, n = 2, 20
    prop = synth.make_prop(nt, n, seed=995)
    rng = np.random.default_rng(996)
    s = np.where(np.arange(n) < n // 2, 1.0, -1.0)
    prop[..., 1, :, :], prop[..., 3, :, :] = prop[..., 0, :, :] * s, prop[..., 2, :, :] * s
    odd = s[:, None] * s[None, :] < 0
    src = [synth.make_phi_random(nt, n, rng) * np.where(odd, 1.0, 1e-8) for _ in range(2)]
    snk = [synth.make_phi_random(nt, n, rng) for _ in range(2)]
    ps = [_dev(p, cuda) for p in src + snk]
    tp = _dev(prop, cuda)
    diag = api.prop_diag(_dev(synth.make_prop(nt, n, seed=997), cuda))

    def run(engine):
        if sets_call:
            return api.run_contract_pipi_sets(tp, diag, torch.stack(ps, dim=1).contiguous(), [(0, 1, 2, 3)], 0,
                                              engine=engine, tf_range=(0, nt))[0]
        return api.run_contract_pipi(tp, diag, *ps, 0, engine=engine, tf_range=(0, nt))

    ref, got = run("fp64"), run("split")
    assert lib().ctr_split_refined() == got.numel()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("power", [-76, 70])
def test_scaled_coefficients_flag_the_same_entries(cuda, power):
    """Coefficients whose squares leave FP32's range: the two-sided form recomputes the
    same entries as for coefficients near 1, with values scaled by the power of two."""
    nt, n, nout = 2, 16, 40
    rng = np.random.default_rng(998)
    prop = _dev(synth.make_prop(nt, n, seed=999), cuda)
    phi = _dev(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1), cuda)
    rows = np.concatenate([rng.integers(0, 4, (160, 4)), rng.integers(0, 2, (160, 2))], axis=1).astype(np.int16)
    coef = rng.integers(1, 4, (160, 2)).astype(np.float32)
    oi = np.repeat(np.arange(nout, dtype=np.int32), 4)
    check(lib().ctr_split_set_refine(4e-13))  # flags some of the entries
    try:
        ref = api.twosided(prop, phi, rows, coef, oi, nout, engine="split")
        flagged = lib().ctr_split_refined()
        got = api.twosided(prop, phi, rows, np.ldexp(coef, power).astype(np.float32), oi, nout, engine="split")
        assert 0 < flagged < ref.numel()
        assert lib().ctr_split_refined() == flagged
    finally:
        check(lib().ctr_split_set_refine(1e-9))
    assert torch.equal(got, ref * 2.0 ** power)


@pytest.mark.parametrize("iso", [0, 1])
@pytest.mark.parametrize("side", ["sink", "source"])
def test_cancelling_block_sums_are_flagged(cuda, iso, side):
    """Square and double triangle where W = T^dag L or S = T G R cancels in its spin sum:
    rows (columns, with gamma_5) of tau alike up to 1e-8 and those of tau(t, t) opposite.
    All pairs have to take the FP64 engine's values."""
    nt, n = 2, 20
    prop = synth.make_prop(nt, n, seed=1005)
    rng = np.random.default_rng(1006)
    diag = rng.normal(size=(nt, 4, 4, n, n)) + 1j * rng.normal(size=(nt, 4, 4, n, n))
    near = lambda x: x * (1.0 + 1e-8 * rng.normal(size=x.shape))
    for a, b in ((2, 0), (3, 1)):
        if side == "sink":
            prop[:, :, a], diag[:, a] = near(prop[:, :, b]), -diag[:, b]
        else:
            prop[:, :, :, a], diag[:, a] = near(prop[:, :, :, b]), diag[:, b]
    ps = [_dev(synth.make_phi_random(nt, n, rng), cuda) for _ in range(4)]
    run = lambda engine: api.run_contract_pipi(_dev(prop, cuda), _dev(diag, cuda), *ps, iso, engine=engine,
                                               tf_range=(0, nt))
    ref, got = run("fp64"), run("split")
    assert lib().ctr_split_refined() == got.numel()
    assert torch.equal(got, ref)
