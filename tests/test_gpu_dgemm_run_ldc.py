"""FP64 runs: the leading dimension of C is the first product's, whatever the
later products of the run name (they find C in registers)."""
import numpy as np
import pytest

import libshalom_b200 as ls
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [ls.DGEMM_FMA, ls.DGEMM_DMMA])
@pytest.mark.parametrize("M,N", [(5, 7), (13, 30), (30, 13), (20, 20), (32, 32), (40, 33)])
def test_run_takes_the_first_products_ldc(method, M, N):
    rng = np.random.default_rng(M)
    K, ldc, runs = 9, N + 5, 3
    A = rng.standard_normal((runs, 3, M, K))
    B = rng.standard_normal((runs, 3, K, N))
    C0 = rng.standard_normal((runs, M, ldc))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    _, ddt = ls.entry_dtypes()
    e = np.zeros((runs, 3), ddt)
    e["M"], e["N"], e["K"], e["alpha"], e["beta"] = M, N, K, 1.0, 1.0
    e["A"] = dA.data_ptr() + 8 * M * K * np.arange(3 * runs).reshape(runs, 3)
    e["B"] = dB.data_ptr() + 8 * K * N * np.arange(3 * runs).reshape(runs, 3)
    e["C"] = dC.data_ptr() + 8 * M * ldc * np.arange(runs)[:, None]
    e["ldc"] = [ldc, 0, N + 2]
    ls.set_dgemm_method(method)
    ls.dgemm_batched(to_dev(e.reshape(-1).view(np.uint8)), 3 * runs)
    C = to_host(dC)
    ref = C0.copy()
    ref[:, :, :N] += np.einsum("rpmk,rpkn->rmn", A, B)
    assert np.array_equal(C[:, :, N:], C0[:, :, N:])
    # K + 1 roundings a product, against the sum of magnitudes
    bound = abs(C0[:, :, :N]) + np.einsum("rpmk,rpkn->rmn", abs(A), abs(B))
    assert np.max(abs(C - ref)[:, :, :N] / bound) <= 3 * (K + 2) * 2.0 ** -53
