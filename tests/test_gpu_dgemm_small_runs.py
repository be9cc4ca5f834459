"""LibShalom_dgemm_batched on the CUDA cores at the edges of its warp tiles:
C blocks whose two halves are two warps' work (above 16 x 16), 16-column and
32-column tiles, K around the 16 values staged at a time, runs next to blocks
above 32 x 32 that take the tile kernel.

Tolerance: normwise 1e-14 against the extended-precision oracle, as for the
other FP64 paths (K <= 33 terms a product: K eps = 7.4e-15 if every rounding
went one way).  Columns between N and ldc must come back bit for bit."""
import numpy as np
import pytest

import libshalom_b200 as ls
from tests._util import normwise_err, to_host
from tests.test_gpu_dgemm_tc import _general

pytestmark = pytest.mark.gpu

EDGES = [1, 4, 5, 16, 17, 32, 33]
KS = [0, 1, 8, 15, 16, 17, 32, 33]


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
    ls.dgemm_batched(dE, count)
    got = to_host(dC)
    for (o, M_, N, ldc, _, C) in refs:
        blk = got[o:o + M_ * ldc].reshape(M_, ldc)
        old = before[o:o + M_ * ldc].reshape(M_, ldc)
        assert np.isfinite(blk[:, :N]).all()
        assert normwise_err(blk[:, :N], C) <= 1e-14 or not np.abs(C).max()
        assert np.array_equal(blk[:, N:], old[:, N:])
