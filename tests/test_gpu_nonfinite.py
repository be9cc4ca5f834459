"""Infinities and NaN stay where they are: a row of A or a column of op(B) that
holds one changes its own row or column of C and no other element, bit for bit.
(The batch kernels repeat edge rows, and the MMAs read shared memory past a
product's rows.)"""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu

SHAPES = ((33, 45, 51), (64, 128, 40), (7, 3, 130), (20, 30, 33))


def _grouped(kind, A, B, shape, count):
    import torch
    M, N, K = shape
    double = A.dtype == np.float64
    dA, dB = to_dev(A), to_dev(B)
    C = torch.full((count, M, N), 0.25, device="cuda",
                   dtype=torch.float64 if double else torch.float32)
    e = np.zeros(count, ls.entry_dtypes()[double])
    e["M"], e["N"], e["K"], e["alpha"], e["beta"] = M, N, K, 1.0, 1.0
    for name, t, n in (("A", dA, M * K), ("B", dB, K * N), ("C", C, M * N)):
        e[name] = t.data_ptr() + A.itemsize * n * np.arange(count)
    if double:
        ls.set_dgemm_method(kind)
        ls.dgemm_batched(to_dev(e.view(np.uint8)), count)
    else:
        ls.set_precision(kind)
        ls.sgemm_batched(to_dev(e.view(np.uint8)), count)
    return to_host(C)


def _uniform(kind, A, B, shape, count):
    import torch
    M, N, K = shape
    C = torch.full((count, M, N), 0.25, device="cuda")
    ls.set_precision(kind)
    ls.sgemm_batched_strided(0, M, N, K, 1.0, to_dev(A), M * K, to_dev(B), K * N, 1.0, C, M * N,
                             count)
    return to_host(C)


@pytest.mark.parametrize("run,kind,dtype", [
    (_uniform, ls.PREC_FP32, np.float32), (_uniform, ls.PREC_BF16X6, np.float32),
    (_grouped, ls.PREC_FP32, np.float32), (_grouped, ls.PREC_BF16X6, np.float32),
    (_grouped, ls.DGEMM_FMA, np.float64), (_grouped, ls.DGEMM_DMMA, np.float64)],
    ids=["uniform-fp32", "uniform-bf16x6", "fp32", "bf16x6", "fma", "dmma"])
@pytest.mark.parametrize("count", [4, 300])
def test_rows_and_columns_apart(run, kind, dtype, count):
    for shape in SHAPES:
        M, N, K = shape
        A = orc.uniform_f32(1, count * M * K).astype(dtype).reshape(count, M, K)
        B = orc.uniform_f32(2, count * K * N).astype(dtype).reshape(count, K, N)
        clean = run(kind, A, B, shape, count)
        r, c = M - 1, N // 2  # the edge row that kernels repeat; a column inside
        A[::2, r, K // 2] = np.nan
        A[1::2, r, K - 1] = np.inf
        B[::2, 0, c] = -np.inf
        B[1::2, K - 1, c] = np.nan
        got = run(kind, A, B, shape, count)
        keep = np.ones((M, N), bool)
        keep[r, :] = False
        keep[:, c] = False
        assert np.isfinite(clean).all()
        assert np.array_equal(got[:, keep], clean[:, keep])
        assert not np.isfinite(got[:, r, :]).any() and not np.isfinite(got[:, :, c]).any()
