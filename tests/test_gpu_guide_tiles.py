"""Network inference in tiles of 32 rows: partial tiles, CTAs with idle warps and
warps with several tiles give a row the same bits wherever it stands, and
those of the numpy restatement within the BF16 rounding of its activations."""
import numpy as np
import pytest

from kazen_proto_gb300 import api
from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu

N = 200_003  # more rows than all resident warps take in one go


@pytest.fixture(scope="module")
def net(gpu):
    rng = np.random.default_rng(21)
    g = api.Guide(seed=3)
    p = G.init_params(9)
    g.set_params(p)
    p01 = rng.random((N, 3)).astype(np.float32)
    nrm = rng.standard_normal((N, 3)).astype(np.float32)
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    return g, p, p01, nrm, g.forward(p01, nrm)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 127, 128, 129, 4097])
def test_rows_do_not_depend_on_their_tile(net, n):
    g, p, p01, nrm, all_rows = net
    assert np.array_equal(g.forward(p01[:n], nrm[:n]), all_rows[:n])
    last = g.forward(p01[N - n:], nrm[N - n:])
    assert np.array_equal(last, all_rows[N - n:])
    ref = G.forward(p, p01[N - n:], nrm[N - n:], use_bf16=True)["O"]
    # an activation that rounds to the other BF16 neighbour moves an output by 2^-8 of a term
    assert np.abs(last - ref).max() <= 2e-2 * np.abs(ref).max() + 1e-3
