"""The split GEMMs' MMA schedules: every slice pair of a packed tail in its level, and the
left operand's collector buffer."""
import numpy as np
import pytest
import torch

from contractions_code_scattering_gb300 import api
from tests.test_split_gemm import _emulate_slices, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [49, 52, 53, 56, 57])
@pytest.mark.parametrize("tail_only", [False, True])
def test_accumulation_levels_of_packed_tails(cuda, n, tail_only):
    """Last chunks of 1 to 4 valid k (four slice pairs an MMA), 5 to 8 (two) and 9 (one):
    levels 0, 1 and 2 are exact sums of their pairs' digits, with operands in all chunks
    and in the last one alone; level 3 to 2^-16 of its size, the tensor core's truncation."""
    rng = np.random.default_rng(30 + n)
    x, y = _rand(rng, (n, n)), _rand(rng, (n, n))
    if tail_only:
        x[:, :48] = 0.0
    lv = api.split_levels(*(torch.from_numpy(a).to(cuda) for a in (x, y))).cpu().numpy().astype(np.float64)
    (xr, xi), (yr, yi) = _emulate_slices(x, 1), _emulate_slices(y, 0)
    exact = np.zeros((8, n, n))
    for i in range(5):
        for j in range(5 - i):
            l = min(i + j, 3)
            exact[l] += xr[i] @ yr[j] - xi[i] @ yi[j]
            exact[4 + l] += xr[i] @ yi[j] + xi[i] @ yr[j]
    for a in (0, 1, 2, 4, 5, 6):
        assert np.array_equal(lv[a], exact[a]), a
    for a in (3, 7):
        assert np.abs(lv[a] - exact[a]).max() <= 2.0 ** -16 * np.abs(exact[a]).max()


def test_collector_buffer_feeds_the_mmas(cuda):
    """An MMA of the complex128 form takes 48 clocks of the tensor pipe; reading its left
    operand from shared memory each time, it is bound by that at 56."""
    cpm, _ = api.mma_schedule_probe(True, 200)
    assert cpm <= 52.0, cpm
