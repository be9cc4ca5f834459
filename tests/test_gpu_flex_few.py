"""Plain FP32 batches by their number of products: grouped batches without lists
(up to 32 entries), with the one-block plan and the quarters of 64 x 64 tiles (few
tiles), with the one-block plan alone (up to 2,048) and with the plan over the
chip; uniform batches on 32 x 32 tiles (few) and on the larger ones.  Bit-exact
with the k-sequential FMA restatement, run by run."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host
from tests.test_gpu_flex import _apply

pytestmark = pytest.mark.gpu

SIZES = (1, 5, 31, 32, 33, 64, 65, 100, 129)
KS = (0, 1, 31, 32, 33, 64, 96, 97, 130)


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 60, 300, 2048, 2049])
def test_grouped_counts(count):
    rng = np.random.default_rng(count)
    small = count > 100  # (keeps the oracle's work small)
    prods, na, nb, nc = [], 0, 0, 0
    while len(prods) < count:
        M, N = (int(x) for x in rng.choice(SIZES[:3] if small and rng.random() < 0.9 else SIZES, 2))
        ldc = N + int(rng.integers(3))
        for p in range(min(int(rng.integers(1, 5)), count - len(prods))):
            K, tb, pad = int(rng.choice(KS)), int(rng.integers(2)), int(rng.integers(2))
            q = dict(M=M, N=N, K=K, tb=tb, lda=max(1, K + pad),
                     ldb=max(1, (K if tb else N) + pad), ldc=ldc,
                     alpha=(1.0, -0.5)[p % 2], beta=(0.0, 1.0, 0.5)[int(rng.integers(3))])
            q["a"], q["b"], q["c"] = na + int(rng.integers(4)), nb + int(rng.integers(4)), nc
            na, nb = q["a"] + M * q["lda"], q["b"] + (N if tb else max(1, K)) * q["ldb"]
            prods.append(q)
        nc += M * ldc + 1
    A, B, C0 = (orc.uniform_f32(s, n + 8) for s, n in ((1, na), (2, nb), (3, nc)))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    e = np.zeros(count, ls.entry_dtypes()[0])
    for k in ("M", "N", "K", "lda", "ldb", "ldc", "alpha", "beta"):
        e[k] = [q[k] for q in prods]
    e["transb"] = [q["tb"] for q in prods]
    for name, t, k in (("A", dA, "a"), ("B", dB, "b"), ("C", dC, "c")):
        e[name] = t.data_ptr() + 4 * np.array([q[k] for q in prods])
    ls.sgemm_batched(to_dev(e.view(np.uint8)), count)
    want = C0.copy()
    for q in prods:
        M, N, K = q["M"], q["N"], q["K"]
        a = A[q["a"]:q["a"] + M * q["lda"]].reshape(M, -1)[:, :K]
        b = B[q["b"]:q["b"] + (N if q["tb"] else max(1, K)) * q["ldb"]].reshape(-1, q["ldb"])
        b = b[:, :K] if q["tb"] else b[:K, :N]
        acc = (orc.sgemm_kseq(np.ascontiguousarray(a), np.ascontiguousarray(b), q["tb"]) if K
               else np.zeros((M, N), np.float32))
        at = q["c"] + q["ldc"] * np.arange(M)[:, None] + np.arange(N)[None, :]
        want[at] = _apply(want[at], acc, q["alpha"], q["beta"])
    assert np.array_equal(to_host(dC), want)


@pytest.mark.parametrize("transb", [0, 1])
def test_uniform_counts(transb):
    for M, N, K in ((5, 7, 33), (31, 33, 40), (64, 64, 65), (33, 65, 32), (65, 31, 100),
                    (129, 130, 33), (128, 64, 3)):
        tiles = -(-M // 32) * -(-N // 32)
        for count in (3, 888 // tiles, 888 // tiles + 150):
            A, B = orc.uniform_f32(1, count * M * K), orc.uniform_f32(2, count * N * K)
            C0 = orc.uniform_f32(3, count * M * N)
            C = to_dev(C0)
            ls.sgemm_batched_strided(transb, M, N, K, -0.5, to_dev(A), M * K, to_dev(B), N * K,
                                     0.5, C, M * N, count)
            C = to_host(C).reshape(count, M, N)
            for g in (0, count // 2, count - 1):
                acc = orc.sgemm_kseq(
                    A[g * M * K:(g + 1) * M * K].reshape(M, K),
                    B[g * K * N:(g + 1) * K * N].reshape((N, K) if transb else (K, N)), transb)
                want = _apply(C0.reshape(count, M, N)[g], acc, -0.5, 0.5)
                assert np.array_equal(C[g], want), (M, N, K, count, g)
