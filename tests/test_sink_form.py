"""rho -> pi pi and triangle set calls in the sink form: products of the sink operators
that no set is part of, and one Gram product a t_src for every set."""
import ctypes
import json

import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth
from contractions_code_scattering_gb300._lib import check, lib
from tests import parity as P

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _inputs(cuda, nt, n, seed, decay=0.1):
    rng = np.random.default_rng(seed)
    prop = synth.make_prop(nt, n, seed=seed + 1, decay=decay)
    phi, mom5, mom2 = (np.stack([synth.make_phi_random(nt, n, rng) for _ in range(k)], axis=1) for k in (5, 5, 2))
    return prop, _dev(phi, cuda), _dev(mom5, cuda), _dev(mom2, cuda)


def _sink_launches(call):
    """The call's value, and how many Gram products of the sink form it launched."""
    torch.cuda.synchronize()
    lib().ctr_timing_enable(1)
    try:
        out = call()
        torch.cuda.synchronize()
        buf = ctypes.create_string_buffer(1 << 16)
        check(lib().ctr_timing_report(buf, len(buf)))
        return out, json.loads(buf.value).get("gram_rows_sum", [0])[0]
    finally:
        lib().ctr_timing_enable(0)


SETS = [(a, b) for a in range(5) for b in range(5)]


@pytest.mark.parametrize("rows,rhopi,tri,nset,sink", [(8, True, True, 11, True), (8, True, True, 10, False),
                                                      (8, True, False, 9, True), (8, False, True, 2, True),
                                                      (8, False, True, 1, False), (1, False, True, 2, False),
                                                      (1, True, True, 25, False), (1, False, True, 25, True),
                                                      (4, False, True, 3, True), (4, False, True, 2, False),
                                                      (21, True, True, 12, True)])
def test_sink_form_rule(cuda, rows, rhopi, tri, nset, sink):
    """Both sides of the rule -- sets, outputs, and sink times that fill a tile of a Gram
    product or leave most of it empty -- against the FP64 engine, per entry."""
    nt, n = max(rows, 2), 9
    prop, phi, mom5, mom2 = _inputs(cuda, nt, n, 1200 + nset)
    tp = _dev(prop, cuda)
    run = lambda engine: api.run_contract_rhopi_sigmapi_sets(
        tp[:rows].contiguous(), api.prop_diag(tp), phi, SETS[:nset], mom5, mom2, engine=engine, tf_range=(0, rows),
        rhopi=rhopi, triangle=tri, hor_fish=False)
    ref = run("fp64")
    got, launches = _sink_launches(lambda: run("split"))
    assert (launches > 0) == sink
    for k in ref:
        want = ref[k].cpu().numpy()
        P.entrywise(got[k].cpu().numpy(), want, 1e-9, np.abs(want), k)


@pytest.mark.parametrize("tol", [1e-9, 1e-13])
def test_sink_form_replayed(cuda, tol):
    """A recorded sink-form call, and its recomputation between the graph's segments, give
    the eager call's values bitwise."""
    nt, n = 8, 11
    prop, phi, mom5, mom2 = _inputs(cuda, nt, n, 1300)
    tp = _dev(prop, cuda)
    diag, s = api.prop_diag(tp), torch.cuda.Stream()
    new = lambda *sh: torch.zeros(sh, dtype=torch.complex128, device=cuda)
    outs = [dict(rhopi=new(11, 3, nt, nt, 4), triangle=new(11, nt, nt, 2), hor_fish=new(11, nt)) for _ in range(2)]
    run = lambda o: api.run_contract_rhopi_sigmapi_sets(tp, diag, phi, SETS[:11], mom5, mom2, engine="split", out=o,
                                                        stream=s)
    check(lib().ctr_split_set_refine(tol))
    try:
        torch.cuda.synchronize()
        _, launches = _sink_launches(lambda: run(outs[0]))
        refined = lib().ctr_split_refined()
        assert launches > 0
        with api.Graph(s) as g:
            run(outs[1])
        g.launch(s)
        s.synchronize()
        assert lib().ctr_split_refined() == refined and (refined > 0 or tol > 1e-12)
        for k in outs[0]:
            assert torch.equal(outs[1][k], outs[0][k]), k
        g.close()
    finally:
        check(lib().ctr_split_set_refine(1e-9))


@pytest.mark.parametrize("rhopi", [False, True])
def test_cancelling_sink_terms_are_flagged(cuda, rhopi):
    """tau_{2 s} = tau_{0 s} and tau_{3 s} = tau_{1 s} up to 1e-8: the triangle's sum over the
    closing spin, which the sink form takes inside its products, cancels to 1e-8 of its
    terms, so every entry has to be recomputed."""
    nt, n = 8, 10
    prop, phi, mom5, mom2 = _inputs(cuda, nt, n, 1400)
    rng = np.random.default_rng(1401)
    for a, b in ((2, 0), (3, 1)):
        prop[:, :, a] = prop[:, :, b] * (1.0 + 1e-8 * rng.normal(size=prop[:, :, b].shape))
    tp = _dev(prop, cuda)
    diag = api.prop_diag(_dev(synth.make_prop(nt, n, seed=1402), cuda))
    run = lambda engine: api.run_contract_rhopi_sigmapi_sets(tp, diag, phi, SETS[:11], mom5, mom2, engine=engine,
                                                             rhopi=rhopi, triangle=True, hor_fish=False)
    ref = run("fp64")
    got, launches = _sink_launches(lambda: run("split"))
    assert launches > 0 and lib().ctr_split_refined() >= ref["triangle"].numel()
    assert torch.equal(got["triangle"], ref["triangle"])


@pytest.mark.parametrize("power", [-200, 70, 200])
def test_sink_scales_follow_the_data(cuda, power):
    """tau times a power of two: the same entries are recomputed, and the values are those
    of the unscaled call times its square."""
    nt, n = 8, 9
    prop, phi, mom5, mom2 = _inputs(cuda, nt, n, 1500)
    diag = api.prop_diag(_dev(prop, cuda))
    run = lambda tau: api.run_contract_rhopi_sigmapi_sets(_dev(tau, cuda), diag, phi, SETS[:11], mom5, mom2,
                                                          engine="split", hor_fish=False)
    check(lib().ctr_split_set_refine(1e-13))
    try:
        (ref, launches), flagged = _sink_launches(lambda: run(prop)), lib().ctr_split_refined()
        got = run(prop * 2.0 ** power)
        assert launches > 0 and 0 < flagged < ref["rhopi"].numel() and lib().ctr_split_refined() == flagged
    finally:
        check(lib().ctr_split_set_refine(1e-9))
    for k in ref:
        assert torch.equal(got[k], ref[k] * 2.0 ** (2 * power)), k
