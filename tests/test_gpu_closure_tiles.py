"""Closure batches at the edges of the grouped kernels' tiles (256 queries, 512
from 2^16 and 1,024 from 2^18 queries on): every query's result is the one it
has in a batch of its own kind in small pieces, bit for bit, whatever surrounds
it."""
import numpy as np
import pytest

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api
from test_gpu_closures import N_KINDS, dirs, lobe_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 513, 2 ** 16 - 1, 2 ** 16, 2 ** 16 + 513, 2 ** 18 - 1, 2 ** 18,
                               2 ** 18 + 1, 2 ** 18 + 1025])
def test_batches_match_their_pieces(gpu, n):
    rng = np.random.default_rng(n)
    base = lobe_grid(rng, 40 * N_KINDS)
    pick = rng.integers(0, len(base), n)
    lobes, wi, wo = base[pick], dirs(rng, n), dirs(rng, n)
    u = rng.random((n, 3)).astype(np.float32)
    whole = [*api.closure_eval(lobes, wi, wo, N.KZ_CONVENTION_INTEGRATOR),
             *api.closure_eval(lobes, wi, wo, N.KZ_CONVENTION_REFERENCE), *api.closure_sample(lobes, wi, u)]
    at = np.argsort(pick, kind="stable")[:: max(1, n // 4000)]  # a few thousand queries, kind by kind
    for k in range(0, len(at), 200):
        p = at[k:k + 200]
        piece = [*api.closure_eval(lobes[p], wi[p], wo[p], N.KZ_CONVENTION_INTEGRATOR),
                 *api.closure_eval(lobes[p], wi[p], wo[p], N.KZ_CONVENTION_REFERENCE),
                 *api.closure_sample(lobes[p], wi[p], u[p])]
        for a, b in zip(whole, piece):
            assert a[p].tobytes() == b.tobytes()
