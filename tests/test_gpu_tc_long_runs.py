"""Split-BF16 grouped batches: long runs on few C go to the pipelined kernel, the
same runs among many others to the small-product kernel.  Both give the same
bits, within 2^-24 of each product's result (one rounding of C) and 8 * 2^-24 of
|A||B| (the bound of one chunk)."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [ls.PREC_BF16X6, ls.PREC_BF16X3])
@pytest.mark.parametrize("M,N,K,products", [(33, 40, 33, 20), (64, 64, 64, 8), (32, 32, 17, 16),
                                            (31, 33, 32, 40), (130, 70, 300, 3),
                                            (256, 129, 520, 1), (8, 8, 8, 30)])
def test_same_bits_on_both_routes(mode, M, N, K, products):
    runs, fill = 5, 160
    n = runs * products
    A, B = orc.uniform_f32(1, n * M * K), orc.uniform_f32(2, n * K * N)
    C0 = orc.uniform_f32(3, runs * M * N)
    dA, dB, dF = to_dev(A), to_dev(B), to_dev(np.zeros(fill, np.float32))
    out = []
    for extra in (0, fill):  # 1 x 1 products, each with a C of its own
        dC = to_dev(C0)
        e = np.zeros(n + extra, ls.entry_dtypes()[0])
        e["M"], e["N"], e["K"], e["alpha"], e["beta"] = M, N, K, 1.0, 1.0
        e["A"][:n] = dA.data_ptr() + 4 * M * K * np.arange(n)
        e["B"][:n] = dB.data_ptr() + 4 * K * N * np.arange(n)
        e["C"][:n] = dC.data_ptr() + 4 * M * N * (np.arange(n) // products)
        for k in ("M", "N", "K"):
            e[k][n:] = 1
        e["A"][n:], e["B"][n:] = dA.data_ptr(), dB.data_ptr()
        e["C"][n:] = dF.data_ptr() + 4 * np.arange(extra)
        ls.set_precision(mode)
        ls.sgemm_batched(to_dev(e.view(np.uint8)), n + extra)
        out.append(to_host(dC))
    assert np.array_equal(out[0], out[1])
    eps = 2.0 ** -24 if mode == ls.PREC_BF16X6 else 2.0 ** -17
    c = C0.reshape(runs, M, N).astype(np.float64)
    bound = np.zeros_like(c)
    a = A.reshape(runs, products, M, K).astype(np.float64)
    b = B.reshape(runs, products, K, N).astype(np.float64)
    for p in range(products):
        c = c + a[:, p] @ b[:, p]
        bound += 2.0 ** -24 * abs(c) + (8 + K // 128) * eps * (abs(a[:, p]) @ abs(b[:, p]))
    assert np.max(abs(out[0].reshape(c.shape) - c) / bound) <= 1.0
