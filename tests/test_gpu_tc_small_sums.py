"""Split-BF16 products of the small-product kernel with K above one accumulation
chunk (128): the chunks are summed apart from C, so a C that is large beside the
product is rounded once a product.  Bound: 2^-24 of the result a product (that
rounding) and 2^-24 (8 + chunks) of |alpha| |A||B| (the bound of one chunk, and
one rounding a chunk sum).  Uniform batches and single calls give the cp.async
kernel's bits, subnormal C included."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


@pytest.mark.parametrize("aligned", [False, True])
def test_grouped_adds_to_a_large_c(aligned):
    runs, i = [], 0
    for M in (1, 31, 32, 33, 64, 65, 100, 256):
        for N in (7, 64, 65, 200):
            ks = ((2052,), (130, 64, 2052), (128, 300), (129, 129))[i % 4]
            runs.append([dict(M=M, N=N, K=K + (-K % 4 if aligned else i % 2), tb=(i + p) % 2,
                              alpha=(1.0, -0.75)[i // 2 % 2], beta=(1.0, 0.5)[(i + p) // 3 % 2])
                         for p, K in enumerate(ks)])
            i += 1
    prods = [q for r in runs for q in r]
    A = orc.uniform_f32(5, sum(q["M"] * q["K"] for q in prods))
    B = orc.uniform_f32(6, sum(-(-q["N"] // 4) * 4 * q["K"] for q in prods))
    C0 = orc.uniform_f32(7, sum(r[0]["M"] * r[0]["N"] for r in runs)) * np.float32(1e7)
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    sdt, _ = ls.entry_dtypes()
    e = np.zeros(len(prods), sdt)
    ref, bound = C0.astype(np.float64), np.zeros(C0.size)
    at_a = at_b = at_c = j = 0
    for r in runs:
        M, N = r[0]["M"], r[0]["N"]
        c = ref[at_c:at_c + M * N].reshape(M, N)
        bd = bound[at_c:at_c + M * N].reshape(M, N)
        for q in r:
            K, tb = q["K"], q["tb"]
            ldb = K if tb else (-(-N // 4) * 4 if aligned else N)
            e[j]["M"], e[j]["N"], e[j]["K"], e[j]["transb"], e[j]["ldb"] = M, N, K, tb, ldb
            e[j]["alpha"], e[j]["beta"] = q["alpha"], q["beta"]
            e[j]["A"], e[j]["B"], e[j]["C"] = (dA.data_ptr() + 4 * at_a, dB.data_ptr() + 4 * at_b,
                                               dC.data_ptr() + 4 * at_c)
            a = A[at_a:at_a + M * K].reshape(M, K).astype(np.float64)
            b = B[at_b:at_b + (N if tb else K) * ldb].reshape(-1, ldb).astype(np.float64)
            b = b.T if tb else b[:, :N]
            c[:] = q["alpha"] * (a @ b) + q["beta"] * c
            bd[:] = (abs(q["beta"]) * bd + EPS * abs(c)
                     + EPS * (8 + -(-K // 128)) * abs(q["alpha"]) * (abs(a) @ abs(b)))
            at_a += M * K
            at_b += -(-N // 4) * 4 * K
            j += 1
        at_c += M * N
    ls.set_precision(ls.PREC_BF16X6)
    ls.sgemm_batched(to_dev(e.view(np.uint8)), len(prods))
    assert np.max(np.abs(to_host(dC) - ref) / bound) <= 1.0


@pytest.mark.parametrize("mode", [ls.PREC_BF16X6, ls.PREC_BF16X3])
@pytest.mark.parametrize("transb", [0, 1])
def test_uniform_gives_the_cp_async_kernels_bits(mode, transb):
    shapes = ((45, 37, 129), (65, 129, 257), (31, 5, 2049), (33, 64, 2052), (130, 3, 300),
              (64, 200, 128), (20, 33, 51))
    for i, (M, N, K) in enumerate(shapes):
        for alpha, beta in ((1.0, 1.0), (0.3, 0.0), (0.3, 0.5), (-0.7, -2.0), (0.3, 1.0)):
            count, sc = 7, M * N + 3  # three floats between the C matrices stay as they are
            A = to_dev(orc.uniform_f32(i + 1, count * M * K + 1))
            B = to_dev(orc.uniform_f32(i + 2, count * K * N))
            C0 = orc.uniform_f32(i + 3, count * sc) * np.float32(1e4)
            out = []
            for tma in (True, False):
                C = to_dev(C0)
                ls.set_tma(tma)
                ls.set_precision(mode)
                ls.sgemm_batched_strided(transb, M, N, K, alpha, A.data_ptr() + 4, M * K, B,
                                         K * N, beta, C, sc, count)
                out.append(to_host(C).reshape(count, sc))
            assert np.array_equal(out[0], out[1]), (M, N, K, alpha, beta)
            assert np.array_equal(out[0][:, M * N:], C0.reshape(count, sc)[:, M * N:])


@pytest.mark.parametrize("alpha,beta", [(1.0, 1.0), (0.3, 0.5), (-0.7, 0.0)])
def test_single_gives_the_cp_async_kernels_bits(alpha, beta):
    for M, N, K in ((70, 131, 301), (257, 33, 1025), (5, 9, 77)):
        lda, ldb, ldc = K + 2, N + 1, N + 3
        A, B = to_dev(orc.uniform_f32(1, M * lda)), to_dev(orc.uniform_f32(2, K * ldb))
        C0 = orc.uniform_f32(3, M * ldc) * np.float32(1e4)
        out = []
        for tma in (True, False):
            C = to_dev(C0)
            ls.set_tma(tma)
            ls.set_precision(ls.PREC_BF16X6)
            ls.sgemm_ex(0, 0, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc)
            out.append(to_host(C).reshape(M, ldc))
        assert np.array_equal(out[0], out[1])
        assert np.array_equal(out[0][:, N:], C0.reshape(M, ldc)[:, N:])


def test_subnormal_c_is_kept():
    ls.set_precision(ls.PREC_BF16X6)
    for M, N, K in ((5, 7, 3), (40, 33, 300), (5, 7, 0)):
        C0 = np.linspace(1e-44, 1e-39, 2 * M * N, dtype=np.float32)
        A = to_dev(np.zeros(2 * M * max(K, 1), np.float32))
        B = to_dev(orc.uniform_f32(1, 2 * max(K, 1) * N))
        C = to_dev(C0)
        ls.sgemm_batched_strided(0, M, N, K, 1.0, A, M * K, B, K * N, 1.0, C, M * N, 2)
        assert np.array_equal(to_host(C), C0)
        C = to_dev(C0)
        ls.sgemm_ex(0, 0, M, N, K, 1.0, A, max(K, 1), B, N, 1.0, C, N)
        assert np.array_equal(to_host(C), C0)


@pytest.mark.parametrize("alpha", [1.0, 0.3])
def test_products_on_one_c(alpha):
    """Equal products that all name one C (strides 0): every element is the
    product's, also while the others write it."""
    ls.set_precision(ls.PREC_BF16X6)
    for M, N, K in ((45, 37, 300), (130, 129, 1025)):
        A, B = to_dev(orc.uniform_f32(1, M * K)), to_dev(orc.uniform_f32(2, K * N))
        C = [to_dev(np.full(M * N, np.nan, np.float32)) for _ in range(2)]
        ls.sgemm_batched_strided(0, M, N, K, alpha, A, 0, B, 0, 0.0, C[0], 0, 2000)
        ls.sgemm_batched_strided(0, M, N, K, alpha, A, 0, B, 0, 0.0, C[1], 0, 1)
        assert np.array_equal(to_host(C[0]), to_host(C[1]))
