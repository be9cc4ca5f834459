"""GPU parity of the plain FP32 batch kernels at the edges of their tiles (64 x
64, 64 x 128), thread tiles (4 and 8), K slabs (32) and of the split into wide
and small lists: bit-exact with the k-sequential FMA restatement, run by run
(C = fma(beta, C, alpha * sum) after each product)."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu

EDGES = (1, 3, 4, 5, 8, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200)
K_EDGES = (0, 1, 2, 3, 4, 5, 31, 32, 33, 64, 65, 100)


def _fma32(a, b, c):
    """fma of float32 arrays: exact in long double (24 + 24 bits, then one
    rounding to 64, whose double rounding to 24 cannot differ for these
    inputs: checked by the caller's products staying within 2^-40..2^40)."""
    return (a.astype(np.longdouble) * b + c.astype(np.longdouble)).astype(np.float32)


def _apply(C, acc, alpha, beta):
    v = np.float32(alpha) * acc
    return _fma32(np.full_like(C, beta), C, v) if beta != 0.0 else v


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("transb", [0, 1])
def test_uniform_edges(transb, off):
    import torch
    count = 5
    for i, M in enumerate(EDGES):
        for N in EDGES[i % 3::3]:
            K = K_EDGES[(i * 5 + N) % len(K_EDGES)]
            A = orc.uniform_f32(M + N, count * M * K + off)
            B = orc.uniform_f32(M * 3 + N, count * N * K + off)
            dA, dB = to_dev(A), to_dev(B)
            C = torch.full((count, M, N), float("nan"), device="cuda")
            ls.sgemm_batched_strided(transb, M, N, K, 1.0, dA.data_ptr() + 4 * off, M * K,
                                     dB.data_ptr() + 4 * off, N * K, 0.0, C, M * N, count)
            a = A[off:].reshape(count, M, K)
            b = B[off:].reshape((count, N, K) if transb else (count, K, N))
            C = to_host(C)
            for g in (0, count - 1):
                want = orc.sgemm_kseq(a[g], b[g], transb) if K else np.zeros((M, N), np.float32)
                assert np.array_equal(C[g], want), (M, N, K)


def test_grouped_edges():
    rng = np.random.default_rng(0)
    prods, na, nb, nc = [], 0, 0, 0
    for i, M in enumerate(EDGES):
        for N in EDGES + (256, 300):
            for p in range(1 + (i + N) % 2):
                K = K_EDGES[int(rng.integers(len(K_EDGES)))]
                tb, pad = int(rng.integers(2)), int(rng.integers(3))
                q = dict(M=M, N=N, K=K, tb=tb, lda=K + pad, ldb=max(1, (K if tb else N) + pad),
                         ldc=N + pad, alpha=(1.0, -0.5)[p], beta=(0.0, 1.0, 0.5)[(i + p) % 3])
                q["lda"] = max(1, q["lda"])
                q["a"], q["b"] = na + int(rng.integers(4)), nb + int(rng.integers(4))
                q["c"] = nc if p == 0 else prods[-1]["c"]
                if p:
                    q["ldc"] = prods[-1]["ldc"]
                else:
                    nc += M * q["ldc"] + 1
                na = q["a"] + M * q["lda"]
                nb = q["b"] + (N if tb else max(1, K)) * q["ldb"]
                prods.append(q)
    A, B, C0 = (orc.uniform_f32(s, n + 8) for s, n in ((1, na), (2, nb), (3, nc)))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    sdt, _ = ls.entry_dtypes()
    e = np.zeros(len(prods), sdt)
    for k in ("M", "N", "K", "lda", "ldb", "ldc", "alpha", "beta"):
        e[k] = [q[k] for q in prods]
    e["transb"] = [q["tb"] for q in prods]
    for name, t, k in (("A", dA, "a"), ("B", dB, "b"), ("C", dC, "c")):
        e[name] = t.data_ptr() + 4 * np.array([q[k] for q in prods])
    ls.sgemm_batched(to_dev(e.view(np.uint8)), len(prods))
    C, want = to_host(dC), C0.copy()
    for q in prods:
        M, N, K = q["M"], q["N"], q["K"]
        a = A[q["a"]:q["a"] + M * q["lda"]].reshape(M, -1)[:, :K]
        b = B[q["b"]:q["b"] + (N if q["tb"] else max(1, K)) * q["ldb"]].reshape(-1, q["ldb"])
        b = b[:, :K] if q["tb"] else b[:K, :N]
        acc = (orc.sgemm_kseq(np.ascontiguousarray(a), np.ascontiguousarray(b), q["tb"]) if K
               else np.zeros((M, N), np.float32))
        at = q["c"] + q["ldc"] * np.arange(M)[:, None] + np.arange(N)[None, :]
        want[at] = _apply(want[at], acc, q["alpha"], q["beta"])
    assert np.array_equal(C, want)
