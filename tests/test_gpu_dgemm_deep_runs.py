"""LibShalom_dgemm_batched on the CUDA cores: deep runs (many blocks of 16 k) on
small C blocks take the tile kernel when there are few runs and the warp kernel
among many, in the one-block plan (up to 2,048 entries) and in the plan over the
chip.  Both apply each product as an FMA chain over k and add it to C with one
more FMA: the same bits, on both routes and as the restatement gives them."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fill", [0, 100, 2_200], ids=["few", "many", "many-large-plan"])
@pytest.mark.parametrize("M,N,K,products", [(32, 32, 32, 16), (5, 7, 512, 1), (13, 30, 64, 9),
                                            (30, 13, 24, 20), (17, 17, 16, 40), (32, 32, 33, 90)])
def test_deep_runs(M, N, K, products, fill):
    runs = 4 if products < 90 else 30  # 2,700 entries: the plan over the chip
    n = runs * products
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((n, M, K)), rng.standard_normal((n, K, N))
    C0 = rng.standard_normal((runs, M, N))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    dF = to_dev(np.zeros(max(1, fill)))
    e = np.zeros(n + fill, ls.entry_dtypes()[1])
    e["M"], e["N"], e["K"], e["alpha"], e["beta"] = 1, 1, 1, 1.0, 1.0
    e["M"][:n], e["N"][:n], e["K"][:n] = M, N, K
    e["A"], e["B"] = dA.data_ptr(), dB.data_ptr()
    e["A"][:n] += (8 * M * K * np.arange(n)).astype(np.uint64)
    e["B"][:n] += (8 * K * N * np.arange(n)).astype(np.uint64)
    e["C"][:n] = dC.data_ptr() + 8 * M * N * (np.arange(n) // products)
    e["C"][n:] = dF.data_ptr() + 8 * np.arange(fill)
    ls.dgemm_batched(to_dev(e.view(np.uint8)), n + fill)
    got = to_host(dC)
    for r in (0, runs - 1):
        want = C0[r].astype(np.longdouble)
        for p in range(r * products, (r + 1) * products):
            # beta = 1: C + product, the product a k-sequential FMA chain
            want = (want + orc.dgemm_kseq(A[p], B[p], 0)).astype(np.float64)
        assert np.array_equal(got[r], want)
