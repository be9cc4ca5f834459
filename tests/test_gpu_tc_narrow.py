"""GPU parity of the long-K split-BF16 kernel for tiles of at most 64 columns (A
in TMEM, op(B)'s parts side by side, two converter groups) at the edges of its
tiles, slabs (32) and accumulation chunks (128).  Tolerances as in test_gpu_tc:
normwise 1e-6 (bf16x6) / 2e-5 (bf16x3), componentwise 8 * 2^-24 / 2^-14 of
|A||B|."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import componentwise_err, normwise_err, to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = {ls.PREC_BF16X6: (1e-6, 8 * 2.0 ** -24), ls.PREC_BF16X3: (2e-5, 2.0 ** -14)}


@pytest.mark.parametrize("mode", [ls.PREC_BF16X6, ls.PREC_BF16X3])
@pytest.mark.parametrize("transb", [0, 1])
@pytest.mark.parametrize("M,N,K", [(129, 4, 132), (100, 16, 256), (128, 20, 260), (300, 32, 1024),
                                   (65, 36, 144), (1, 48, 388), (256, 60, 512), (200, 64, 160),
                                   (97, 33, 2052)])
def test_narrow_long_k(M, N, K, transb, mode):
    import torch
    if N % 4 and not transb:
        N -= N % 4  # rows of op(B) that TMA can address
    A = orc.uniform_f32(M + K, M * K).reshape(M, K)
    B = orc.uniform_f32(N + K, N * K).reshape((N, K) if transb else (K, N))
    ref, absp = orc.sgemm_f64(A, B, transb), orc.sgemm_absprod(A, B, transb)
    ls.set_precision(mode)
    dA, dB = to_dev(A), to_dev(B)
    for splits in (1, 0, 4):
        C = torch.full((M, N), float("nan"), device="cuda")
        ls.set_splitk(splits)
        ls.sgemm_mp(0, transb, C, dA, dB, M, N, K)
        C = to_host(C)
        assert normwise_err(C, ref) <= TOL[mode][0], splits
        assert componentwise_err(C, ref, absp) <= TOL[mode][1], splits


def test_narrow_uniform_batch_beta():
    import torch
    count, M, N, K = 7, 140, 40, 192
    A = orc.uniform_f32(1, count * M * K).reshape(count, M, K)
    B = orc.uniform_f32(2, count * N * K).reshape(count, N, K)
    C0 = orc.uniform_f32(3, count * M * N).reshape(count, M, N)
    ls.set_precision(ls.PREC_BF16X6)
    dC = to_dev(C0)
    ls.sgemm_batched_strided(1, M, N, K, -0.5, to_dev(A), M * K, to_dev(B), N * K, 0.75, dC, M * N,
                             count)
    C = to_host(dC)
    for g in range(count):
        ref = orc.sgemm_f64(A[g], B[g], 1, alpha=-0.5, beta=0.75, C=C0[g])
        assert normwise_err(C[g], ref) <= 1e-6
