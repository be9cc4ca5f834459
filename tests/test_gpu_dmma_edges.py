"""LibShalom_dgemm_batched with DMMA at the edges of its warp tiles: the three
shapes of C block (split at 16 rows and 16 columns), 8-row and 8-column
fragments, and K around the 4 values of a DMMA and the 12 loaded at a time.

Tolerance: normwise 1e-14 against the extended-precision oracle, the bound the
DMMA path has elsewhere (K <= 70 terms a product: K eps = 1.6e-14 is the worst
case of every rounding going one way; random signs give under 1e-15).  Rows
between N and ldc must come back bit for bit."""
import numpy as np
import pytest

import libshalom_b200 as ls
from tests._util import normwise_err, to_host
from tests.test_gpu_dgemm_tc import _general

pytestmark = pytest.mark.gpu

EDGES = [1, 8, 9, 16, 17, 32]
KS = [0, 1, 4, 5, 11, 12, 13, 24, 32]


@pytest.mark.parametrize("transb", [0, 1], ids=["nn", "nt"])
@pytest.mark.parametrize("M", EDGES)
def test_tile_edges(M, transb):
    runs = []
    for i, N in enumerate(EDGES):
        for j, K in enumerate(KS):
            beta = [1.0, 0.0, -0.5][(i + j) % 3]
            # C is NaN where beta = 0 says it must not be read; a second product
            # with the other layout and another K follows in the same run
            runs.append((M, N, N + (j % 2), beta == 0.0,
                         [(K, transb, 1.0 if j % 2 else 0.75, beta, j % 3, i % 2, j & 1),
                          (KS[-1 - j], 1 - transb, -1.0, 1.0, i % 2, j % 2, i & 1)]))
    dE, count, dC, refs = _general(runs, 100 * M + transb)
    before = to_host(dC).copy()
    ls.set_dgemm_method(ls.DGEMM_DMMA, 0)
    try:
        ls.dgemm_batched(dE, count)
    finally:
        ls.set_dgemm_method(ls.DGEMM_FMA, 0)
    got = to_host(dC)
    for (o, M_, N, ldc, _, C) in refs:
        blk = got[o:o + M_ * ldc].reshape(M_, ldc)
        old = before[o:o + M_ * ldc].reshape(M_, ldc)
        assert np.isfinite(blk[:, :N]).all()
        assert normwise_err(blk[:, :N], C) <= 1e-14 or not np.abs(C).max()
        assert np.array_equal(blk[:, N:], old[:, N:])
