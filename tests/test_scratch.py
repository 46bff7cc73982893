"""Device memory that calls take beside a caller's own tensors."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api
from contractions_code_scattering_gb300._lib import check, lib

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _gauss(*shape):
    return torch.randn(shape, dtype=torch.complex128, device="cuda") / shape[-1] ** 0.5


def _growth(call):
    """Bytes of the library's scratch after a call that started with none."""
    call(1)  # modules and contexts load at the first call
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib().ctr_release_workspace()
    free = torch.cuda.mem_get_info()[0]
    call(None)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    used = free - torch.cuda.mem_get_info()[0]
    lib().ctr_release_workspace()
    return used


@pytest.mark.parametrize("kind", ["pipi", "triangles", "rho_vjp", "pipi_vjp"])
def test_single_calls_keep_to_three_gigabytes(cuda, kind):
    """A single set's calls and the profile gradients plan batches of 3 GB (4 GB in the
    scratch buffer, which grows by powers of two), however many pairs they have, and a
    few hundred MB of per-time-slice products and tables."""
    n, nt = (48, 40) if kind.endswith("vjp") else (64, 40)
    tau, diag = _gauss(nt, nt, 4, 4, n, n), _gauss(nt, 4, 4, n, n)
    p = [_gauss(nt, n, n) for _ in range(4)]
    mom5, mom2, f = _gauss(nt, 5, n, n), _gauss(nt, 2, n, n), torch.rand(n, dtype=torch.float64, device="cuda") + 0.5

    def call(rows):
        kw = {"engine": "fp64", "tf_range": (0, rows or nt)}
        if kind == "pipi":
            api.run_contract_pipi(tau, diag, *p, 0, **kw)
        elif kind == "triangles":
            api.run_contract_rhopi(tau, diag, p[0], p[1], mom5, 0, **kw)
            api.run_contract_sigmapi(tau, diag, p[0], p[1], mom2, **kw)
        else:
            w = torch.zeros((nt, nt, 48 if kind == "rho_vjp" else 5), dtype=torch.complex128, device="cuda")
            w[:rows or nt, :, :3] = 1.0
            if kind == "rho_vjp":
                api.rho_profile_vjp(tau, mom5, f, w, engine="fp64")
            else:
                api.pipi_profile_vjp(tau, *p, f, w, 0, engine="fp64")

    assert _growth(call) <= 5 * 1024 * MB


def test_gradient_tables_are_bounded(cuda):
    """Every output of a rho gradient weighted at a small Nev: the pair tables pass through
    a pinned buffer, in batches of 64 MB."""
    n, nt = 2, 96
    tau, mom5 = _gauss(nt, nt, 4, 4, n, n), _gauss(nt, 5, n, n)
    f = torch.rand(n, dtype=torch.float64, device="cuda") + 0.5

    def call(rows):
        w = torch.zeros((nt, nt, 48), dtype=torch.complex128, device="cuda")
        w[:rows or nt] = 1.0
        api.rho_profile_vjp(tau, mom5, f, w, engine="fp64")

    assert _growth(call) <= 400 * MB


def test_elementals_partial_tiles(cuda):
    """The partial tiles of the elementals: 128 MB beside the derivative fields and phases."""
    n, nt, l = 100, 4, 8
    v = _gauss(nt, n, l, l, l, 3)
    links = _gauss(nt, l, l, l, 3, 3, 3)
    moms = [(a, b, c) for a in range(4) for b in range(4) for c in range(8)]
    assert _growth(lambda rows: api.elementals(v, moms[:rows or len(moms)], links=links)) <= 240 * MB
