"""The autotuner measures each kernel once."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kernels", [(16, 11), (65, 12)])
def test_trace_candidates(cuda, n, kernels):
    """Up to Nev = 64 the two quad-group candidates are one kernel: measured once; both
    numbers may be forced at any Nev, with the same result."""
    nt = 2
    rng = np.random.default_rng(77)
    tau = torch.from_numpy(synth.make_prop(nt, n, seed=78)).to(cuda)
    mom2 = torch.from_numpy(np.stack([synth.make_phi_random(nt, n, rng) for _ in range(2)], axis=1)).to(cuda)
    run = lambda: api.run_contract_sigma(tau, mom2, engine="split")
    ref = run()
    try:
        api.tune_clear()
        api.tune_set_mode(1)
        run()
        ms = [v["ms"] for k, v in api.tune_report().items() if k.startswith("trace_rows|")]
        assert [len(m) for m in ms] == [kernels]
        api.tune_set_mode(0)
        for v in (10, 11):
            api.tune_force("trace_rows", v)
            got = run()
            assert (got - ref).abs().max() <= 1e-12 * ref.abs().max()
    finally:
        api.tune_force("trace_rows", -1)
        api.tune_set_mode(0)
        api.tune_clear()
