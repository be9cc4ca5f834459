"""GPU parity of the small-product split-BF16 kernel (grouped batches, and
uniform batches TMA cannot address) at the edges of its tiles (64 x 128), row
groups (8), MMA shapes (64 / 128 columns), k-steps (16), slabs (32) and K chunks
(128), for every alignment of the rows and every way of updating C, against
the exact-math oracle.  Tolerances as in test_gpu_tc: normwise 1e-6 (bf16x6) /
2e-5 (bf16x3), componentwise 8 * 2^-24 / 2^-14 of |A||B| (+ |C| for the
updates of C: one rounding of the result and of alpha D a product)."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = {ls.PREC_BF16X6: (1e-6, 8 * 2.0 ** -24), ls.PREC_BF16X3: (2e-5, 2.0 ** -14)}
M_EDGES = (1, 7, 8, 9, 17, 63, 64, 65, 128, 129, 255, 256, 257)
N_EDGES = (1, 8, 15, 16, 17, 33, 63, 64, 65, 127, 128, 129, 256, 257)
K_EDGES = (1, 2, 15, 16, 17, 31, 32, 33, 48, 64, 127, 128, 129, 160, 256, 257, 300)


def _products(seed):
    """Every (M, N) of the edges once, K cycling through its edges; runs of up
    to three products on one C; betas 0, 1 and 0.5; padded leading dimensions
    and odd offsets on some."""
    rng = np.random.default_rng(seed)
    out, i = [], 0
    for M in M_EDGES:
        for N in N_EDGES:
            for p in range(1 + (i % 3)):
                K = K_EDGES[(5 * i + 3 * p + seed) % len(K_EDGES)]
                tb = int(rng.integers(2))
                pad = int(rng.integers(3))
                first = p == 0
                out.append(dict(M=M, N=N, K=K, tb=tb, lda=K + pad, ldb=(K if tb else N) + pad,
                                ldc=N + (i % 2), first=first,
                                alpha=1.0 if i % 4 else -0.75,
                                beta=(0.0, 1.0, 0.5)[(i + p) % 3] if first else
                                (1.0, 0.5)[(i + p) % 2],
                                off=int(rng.integers(4))))
            i += 1
    return out


@pytest.mark.parametrize("mode", [ls.PREC_BF16X6, ls.PREC_BF16X3])
@pytest.mark.parametrize("aligned", [False, True])
def test_grouped_edges(mode, aligned):
    prods = _products(3 + aligned)
    a_at, b_at, c_at, na, nb, nc = [], [], [], 0, 0, 0
    for q in prods:
        if aligned:  # 16-byte rows: the 16-byte load path
            q["lda"] = -(-q["lda"] // 4) * 4
            q["ldb"] = -(-q["ldb"] // 4) * 4
            q["off"] = 0
            na, nb = -(-na // 4) * 4, -(-nb // 4) * 4
        na += q["off"]
        nb += q["off"]
        a_at.append(na)
        b_at.append(nb)
        na += q["M"] * q["lda"]
        nb += (q["N"] if q["tb"] else q["K"]) * q["ldb"]
        if q["first"]:
            nc += 1
            c_at.append(nc)
            nc += q["M"] * q["ldc"]
        else:
            c_at.append(c_at[-1])
    A, B, C0 = (orc.uniform_f32(s, n) for s, n in ((11, na), (12, nb), (13, nc + 4)))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C0)
    sdt, _ = ls.entry_dtypes()
    e = np.zeros(len(prods), sdt)
    for k in ("M", "N", "K", "lda", "ldb", "ldc", "alpha", "beta"):
        e[k] = [q[k] for q in prods]
    e["transb"] = [q["tb"] for q in prods]
    e["A"] = dA.data_ptr() + 4 * np.array(a_at)
    e["B"] = dB.data_ptr() + 4 * np.array(b_at)
    e["C"] = dC.data_ptr() + 4 * np.array(c_at)
    ls.set_precision(mode)
    ls.sgemm_batched(to_dev(e.view(np.uint8)), len(prods))
    C = to_host(dC)
    touched = np.zeros(C.size, bool)
    ref = C0.astype(np.float64)
    bound = np.abs(ref)
    nw, cw = TOL[mode]
    for q, ao, bo, co in zip(prods, a_at, b_at, c_at):
        M, N, K = q["M"], q["N"], q["K"]
        a = A[ao:ao + M * q["lda"]].reshape(M, -1)[:, :K].astype(np.float64)
        b = B[bo:bo + (N if q["tb"] else K) * q["ldb"]].reshape(-1, q["ldb"])
        b = (b[:, :K].T if q["tb"] else b[:, :N]).astype(np.float64)
        at = (co + q["ldc"] * np.arange(M)[:, None] + np.arange(N)[None, :])
        ref[at] = q["alpha"] * (a @ b) + q["beta"] * ref[at]
        bound[at] = abs(q["alpha"]) * (abs(a) @ abs(b)) + abs(q["beta"]) * bound[at]
        touched[at] = True
    assert np.array_equal(C[~touched], C0[~touched])  # nothing outside the products
    err = np.abs(C - ref)[touched]
    assert np.all(np.isfinite(C[touched]))
    assert np.max(err / bound[touched]) <= cw
    i = 0
    while i < len(prods):  # normwise, block by block
        q, co = prods[i], c_at[i]
        at = (co + q["ldc"] * np.arange(q["M"])[:, None] + np.arange(q["N"])[None, :])
        if q["M"] * q["N"] >= 64:  # a single element can cancel
            assert np.max(np.abs(C[at] - ref[at])) <= nw * np.max(np.abs(ref[at]))
        i += 1


def test_grouped_either_kernel():
    """Full aligned NT tiles: few of them run as small products, many as large
    ones; both meet the bound and the ragged products beside them do too."""
    import torch
    for n_full in (8, 400):
        shapes = [(128, 128, 128)] * n_full + [(37, 45, 51)] * 40
        a = [orc.uniform_f32(20 + i % 7, m * k).reshape(m, k) for i, (m, n, k) in enumerate(shapes)]
        b = [orc.uniform_f32(40 + i % 5, n * k).reshape(n, k) for i, (m, n, k) in enumerate(shapes)]
        dA, dB = [to_dev(x) for x in a], [to_dev(x) for x in b]
        dC = [torch.full((m, n), float("nan"), device="cuda") for m, n, _ in shapes]
        sdt, _ = ls.entry_dtypes()
        e = np.zeros(len(shapes), sdt)
        e["M"], e["N"], e["K"] = np.array(shapes).T
        e["transb"], e["alpha"] = 1, 1.0
        for name, t in (("A", dA), ("B", dB), ("C", dC)):
            e[name] = [x.data_ptr() for x in t]
        ls.set_precision(ls.PREC_BF16X6)
        ls.sgemm_batched(to_dev(e.view(np.uint8)), len(shapes))
        for x, y, c in zip(a, b, dC):
            ref = x.astype(np.float64) @ y.astype(np.float64).T
            assert np.max(np.abs(to_host(c) - ref)) <= 1e-6 * np.max(np.abs(ref))


@pytest.mark.parametrize("transb", [0, 1])
def test_uniform_unaligned_equals_cp_async_kernel(transb):
    """Uniform batches of rows TMA cannot address, K within one accumulation
    chunk: the small-product kernel gives the cp.async kernel's bits."""
    import torch
    for M, N, K in ((45, 37, 51), (64, 128, 127), (65, 129, 33), (1, 200, 5), (130, 3, 128)):
        count = 50
        A = orc.uniform_f32(1, count * M * K + 1)
        B = orc.uniform_f32(2, count * N * K)
        dA, dB = to_dev(A), to_dev(B)
        out = []
        for tma in (True, False):
            C = torch.full((count, M, N), float("nan"), device="cuda")
            ls.set_tma(tma)
            ls.set_precision(ls.PREC_BF16X6)
            ls.sgemm_batched_strided(transb, M, N, K, 1.0, dA.data_ptr() + 4, M * K, dB, K * N,
                                     0.0, C, M * N, count)
            out.append(to_host(C))
        assert np.array_equal(out[0], out[1])
