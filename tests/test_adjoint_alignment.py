"""Profile gradients: caller arrays that are aligned to doubles only, and the range of the weights."""
import ctypes

import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth
from contractions_code_scattering_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def _odd(a, cuda):
    """A copy of a complex128 array whose address is 8 modulo 16, and that address."""
    flat = torch.view_as_real(torch.from_numpy(np.ascontiguousarray(a))).reshape(-1)
    buf = torch.zeros(flat.numel() + 1, dtype=torch.float64, device=cuda)
    assert buf.data_ptr() % 16 == 0
    buf[1:] = flat.to(cuda)
    return buf, ctypes.c_void_p(buf.data_ptr() + 8)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("engine", ["fp64", "split"])
def test_arrays_aligned_to_doubles(cuda, engine):
    """p1..p4, the weights and the correlators of a gradient are copied where they are not
    16-byte aligned: bitwise the results for aligned arrays."""
    nt, n = 3, 7
    rng = np.random.default_rng(61)
    prop = torch.from_numpy(synth.make_prop(nt, n, seed=60)).to(cuda)
    mom5 = torch.from_numpy(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(5)], axis=1)).to(cuda)
    ps = [synth.make_phi_random(nt, n, rng) for _ in range(4)]
    f = torch.from_numpy(rng.uniform(0.5, 1.5, n)).to(cuda)
    wr, wp = (rng.normal(size=(nt, nt, k)) + 1j * rng.normal(size=(nt, nt, k)) for k in (48, 5))
    dev = lambda a: torch.from_numpy(a).to(cuda)
    rho, grad_r = api.rho_profile_vjp(prop, mom5, f, dev(wr), engine=engine)
    pipi, grad_p = api.pipi_profile_vjp(prop, *[dev(p) for p in ps], f, dev(wp), 0, engine=engine)
    e, s = api._engine(engine), api._stream(None)
    for ref, grad, w in ((rho, grad_r, wr), (pipi, grad_p, wp)):
        out, po = _odd(np.zeros(ref.shape, complex), cuda)
        wbuf, pw = _odd(w, cuda)
        g = torch.zeros(n, dtype=torch.float64, device=cuda)
        if ref is rho:
            check(lib().ctr_rho_profile_vjp(e, n, nt, _ptr(prop), _ptr(mom5), _ptr(f), pw, po, _ptr(g), s))
        else:
            bufs = [_odd(p, cuda) for p in ps]
            check(lib().ctr_pipi_profile_vjp(e, n, nt, 0, _ptr(prop), *[b[1] for b in bufs], _ptr(f), pw, po, _ptr(g), s))
        torch.cuda.synchronize()
        assert out[0] == 0 and torch.equal(out[1:], torch.view_as_real(ref).reshape(-1))
        assert torch.equal(g, grad)


@pytest.mark.parametrize("engine", ["fp64", "split"])
@pytest.mark.parametrize("power", [-1005, 900])
def test_pipi_gradient_weight_range(cuda, engine, power):
    """Weights near the ends of the doubles' range scale the pi pi gradient, to rounding."""
    nt, n = 3, 8
    rng = np.random.default_rng(65)
    prop = torch.from_numpy(synth.make_prop(nt, n, seed=66)).to(cuda)
    ps = [torch.from_numpy(synth.make_phi_random(nt, n, rng)).to(cuda) for _ in range(4)]
    f = torch.from_numpy(rng.uniform(0.5, 1.5, n)).to(cuda)
    w = torch.zeros((nt, nt, 5), dtype=torch.complex128, device=cuda)
    w[..., :2] = torch.from_numpy(rng.normal(size=(nt, nt, 2)) + 1j * rng.normal(size=(nt, nt, 2))).to(cuda)
    _, ref = api.pipi_profile_vjp(prop, *ps, f, w, 0, engine=engine)
    _, got = api.pipi_profile_vjp(prop, *ps, f, w * 2.0 ** power, 0, engine=engine)
    assert (got * 2.0 ** -power - ref).abs().max() <= 1e-13 * ref.abs().max()
