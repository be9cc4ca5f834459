"""The work that a program linked against this library has it do, as cases to time.

Five kinds of work, each through a public entry point of ``libshalom_b200``:

  single   one small product per call, the drop-in LibShalom_sgemm / _dgemm in
           the default synchronous mode (what an unchanged caller does)
  uniform  LibShalom_sgemm_batched_strided: thousands of products of one shape
  mp       LibShalom_sgemm_mp: one irregular product (im2col layers, tall-skinny)
  mixed    LibShalom_sgemm_batched: one batch of products of many shapes
  runs     LibShalom_dgemm_batched: FP64 block products, runs of them adding to
           one C block

FP32 work runs in any of the library's arithmetics (plain FP32, the default;
split-BF16 with three or six products), FP64 runs on the CUDA cores (default)
or the FP64 tensor cores.  Calls other than ``single`` are stream-ordered.
"""
import math

import numpy as np
import torch

import libshalom_b200 as ls

_PREC = {"fp32": ls.PREC_FP32, "bf16x3": ls.PREC_BF16X3, "bf16x6": ls.PREC_BF16X6}
_METHOD = {"fma": ls.DGEMM_FMA, "dmma": ls.DGEMM_DMMA}
# block sizes of the atom-block products
_BLOCKS = (5, 9, 13, 16, 22, 23, 26, 32)
# bounds of one pass: the largest uniform batch, the largest irregular product
_MAX_UNIFORM_BYTES = 4.0 * 3 * 128 * 128 * 10_000
_MAX_MP_FLOPS = 2.0 * 20480 * 32 * 20480
_MAX_MP_FLOATS = 20480 * 20480


def listed():
    return [
        # one 80^3 product with B transposed: the smallest call of all, and the
        # reference's own benchmark of call latency
        {"name": "single_80_nt", "kind": "single", "m": 80, "n": 80, "k": 80, "tb": 1,
         "double": False},
        # uniform batches in the default arithmetic, from the lower and the
        # upper end of the cube sweep 8..128
        {"name": "uniform_fp32_24_nn", "kind": "uniform", "m": 24, "n": 24, "k": 24, "tb": 0,
         "count": 10_000, "arith": "fp32"},
        {"name": "uniform_fp32_104_nt", "kind": "uniform", "m": 104, "n": 104, "k": 104, "tb": 1,
         "count": 10_000, "arith": "fp32"},
        # the same sweep on the tensor cores at FP32 error: a small cube, the
        # largest, and a ragged shape whose rows are not 16-byte aligned
        {"name": "uniform_bf16x6_40_nt", "kind": "uniform", "m": 40, "n": 40, "k": 40, "tb": 1,
         "count": 10_000, "arith": "bf16x6"},
        {"name": "uniform_bf16x6_128_nn", "kind": "uniform", "m": 128, "n": 128, "k": 128,
         "tb": 0, "count": 10_000, "arith": "bf16x6"},
        {"name": "uniform_bf16x6_ragged_nn", "kind": "uniform", "m": 45, "n": 37, "k": 51,
         "tb": 0, "count": 10_000, "arith": "bf16x6"},
        # a convolution layer as its im2col product, default arithmetic
        {"name": "mp_fp32_layer", "kind": "mp", "m": 256, "n": 196, "k": 2304, "tb": 0,
         "arith": "fp32"},
        # few rows against a wide matrix, default arithmetic
        {"name": "mp_fp32_wide", "kind": "mp", "m": 32, "n": 20480, "k": 4096, "tb": 0,
         "arith": "fp32"},
        # the largest product: tall-skinny with a long K, on the tensor cores
        {"name": "mp_bf16x6_tall", "kind": "mp", "m": 20480, "n": 32, "k": 20480, "tb": 0,
         "arith": "bf16x6"},
        # 50,000 products of any size from 4 to 256, on the tensor cores and in
        # the default arithmetic
        {"name": "mixed_bf16x6", "kind": "mixed", "count": 50_000, "shapes": 5,
         "arith": "bf16x6"},
        {"name": "mixed_fp32", "kind": "mixed", "count": 50_000, "shapes": 6, "arith": "fp32"},
        # 200,000 FP64 block products in runs of eight that add to one C block
        {"name": "runs_dmma", "kind": "runs", "count": 200_000, "run": 8, "shapes": 7,
         "method": "dmma"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("single", "uniform", "uniform", "uniform", "mp", "mp", "mixed", "runs"))
    arith = rng.choice(("fp32", "fp32", "bf16x6", "bf16x6", "bf16x3"))
    tb = rng.randrange(2)
    if kind == "single":
        return {"kind": kind, "m": _log_int(rng, 8, 128), "n": _log_int(rng, 8, 128),
                "k": _log_int(rng, 8, 128), "tb": tb, "double": rng.random() < 0.3}
    if kind == "uniform":
        if rng.random() < 0.5:  # cubes, any size
            m = n = k = _log_int(rng, 8, 128)
        else:
            m, n, k = (_log_int(rng, 8, 128) for _ in range(3))
        most = min(20_000, int(_MAX_UNIFORM_BYTES / (4.0 * (m * k + k * n + m * n))))
        return {"kind": kind, "m": m, "n": n, "k": k, "tb": tb,
                "count": _log_int(rng, 1_000, most), "arith": arith}
    if kind == "mp":
        while True:
            m, n, k = _log_int(rng, 32, 20480), _log_int(rng, 32, 20480), _log_int(rng, 256, 20480)
            if rng.random() < 0.5:  # im2col sizes: channels and K of a layer are round
                m, k = -(-m // 32) * 32, -(-k // 32) * 32
            if (1e7 <= 2.0 * m * n * k <= _MAX_MP_FLOPS
                    and m * k + k * n + m * n <= _MAX_MP_FLOATS):
                return {"kind": kind, "m": m, "n": n, "k": k, "tb": tb, "arith": arith}
    if kind == "mixed":
        return {"kind": kind, "count": _log_int(rng, 1_000, 50_000),
                "shapes": rng.randrange(1 << 30), "arith": arith}
    return {"kind": kind, "count": _log_int(rng, 4_000, 200_000), "run": rng.randint(1, 12),
            "shapes": rng.randrange(1 << 30), "method": rng.choice(("fma", "dmma"))}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, dtype=torch.float32):
    return torch.rand(int(n), generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _starts(lengths):
    return np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.int64)


def _mixed_shapes(case):
    """M, N, K log-uniform in [4, 256], half of the products NT; one product
    in five adds (beta = 1) to the C of the product before it."""
    rng = np.random.default_rng(case["shapes"])
    count = case["count"]
    dims = np.exp(rng.uniform(np.log(4), np.log(257), size=(count, 3))).astype(np.int64)
    m, n, k = (np.minimum(d, 256) for d in dims.T)
    tb = rng.integers(2, size=count)
    adds = rng.random(count) < 0.2
    adds[0] = False
    first = np.maximum.accumulate(np.where(adds, 0, np.arange(count)))
    return m[first], n[first], k, tb, first


def _run_shapes(case):
    """M, N, K each one of the block sizes; `run` consecutive products name one
    C block (same M and N), the first with beta = 0, the others adding to it."""
    rng = np.random.default_rng(case["shapes"])
    count = case["count"]
    m, n, k = rng.choice(np.array(_BLOCKS), size=(3, count))
    first = np.arange(count) // case["run"] * case["run"]
    return m[first], n[first], k, np.zeros(count, np.int64), first


def _shapes(case):
    return _mixed_shapes(case) if case["kind"] == "mixed" else _run_shapes(case)


def _layout(case):
    m, n, k, tb, first = _shapes(case)
    own = first == np.arange(len(m))  # products that start a C block
    c_at = _starts(np.where(own, m * n, 0))[first]
    return m, n, k, tb, own, _starts(m * k), _starts(k * n), c_at, int((m * n)[own].sum())


def _grouped_inputs(case, seed):
    m, n, k, tb, own, a_at, b_at, c_at, c_len = _layout(case)
    g = _gen(seed)
    dtype = torch.float32 if case["kind"] == "mixed" else torch.float64
    a_len, b_len = int((m * k).sum()), int((k * n).sum())
    if case["kind"] == "mixed":
        a, b = _uniform(g, a_len), _uniform(g, b_len)
    else:
        # normal entries under a scale of 10^-3 .. 10^3 per matrix
        def pool(lengths):
            x = torch.randn(int(lengths.sum()), generator=g, device="cuda", dtype=dtype)
            scale = torch.rand(len(lengths), generator=g, device="cuda", dtype=dtype)
            scale = torch.pow(10.0, scale * 6 - 3)
            return x.mul_(torch.repeat_interleave(scale, torch.from_numpy(lengths).cuda()))

        a, b = pool(m * k), pool(k * n)
    return a, b, torch.zeros(c_len, device="cuda", dtype=dtype)


def _plain_inputs(case, seed):
    m, n, k, count = case["m"], case["n"], case["k"], case.get("count", 1)
    g = _gen(seed)
    dtype = torch.float64 if case.get("double") else torch.float32
    return (_uniform(g, count * m * k, dtype), _uniform(g, count * k * n, dtype),
            torch.zeros(count * m * n, device="cuda", dtype=dtype))


def prepare(case, seed):
    state = dict(case)
    if case["kind"] in ("mixed", "runs"):
        m, n, k, tb, own, a_at, b_at, c_at, _ = _layout(case)
        a, b, c = _grouped_inputs(case, seed)
        sdt, ddt = ls.entry_dtypes()
        e = np.zeros(case["count"], sdt if case["kind"] == "mixed" else ddt)
        size = a.element_size()
        e["A"] = a.data_ptr() + size * a_at
        e["B"] = b.data_ptr() + size * b_at
        e["C"] = c.data_ptr() + size * c_at
        e["M"], e["N"], e["K"], e["transb"] = m, n, k, tb
        e["alpha"] = 1.0
        e["beta"] = np.where(own, 0.0, 1.0)
        state["entries"] = torch.from_numpy(e.view(np.uint8)).cuda()
    else:
        a, b, c = _plain_inputs(case, seed)
    state.update(a=a, b=b, c=c)
    return state


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

_settings = None


def _use(sync, prec, method):
    """The library's settings, given when they change."""
    global _settings
    if _settings != (sync, prec, method):
        ls.set_sync(sync)
        ls.set_precision(_PREC[prec])
        ls.set_dgemm_method(_METHOD[method])
        _settings = (sync, prec, method)


def run(state):
    kind = state["kind"]
    _use(kind == "single", state.get("arith", "fp32"), state.get("method", "fma"))
    a, b, c = state["a"], state["b"], state["c"]
    if kind == "single":
        call = ls.dgemm if state["double"] else ls.sgemm
        call(ls.NoTrans, state["tb"], c, a, b, state["m"], state["n"], state["k"])
    elif kind == "mp":
        ls.sgemm_mp(ls.NoTrans, state["tb"], c, a, b, state["m"], state["n"], state["k"])
    elif kind == "uniform":
        m, n, k = state["m"], state["n"], state["k"]
        ls.sgemm_batched_strided(state["tb"], m, n, k, 1.0, a, m * k, b, k * n, 0.0, c, m * n,
                                 state["count"])
    elif kind == "mixed":
        ls.sgemm_batched(state["entries"], state["count"])
    else:
        ls.dgemm_batched(state["entries"], state["count"])
    return c


# --------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# --------------------------------------------------------------------------

def work(case):
    if case["kind"] in ("mixed", "runs"):
        m, n, k, tb, own, _, _, _, c_len = _layout(case)
        size = 4 if case["kind"] == "mixed" else 8
        return {"bytes": float(size * ((m * k + k * n).sum() + c_len)),
                "flops": float(2 * (m * n * k).sum())}
    m, n, k, count = case["m"], case["n"], case["k"], case.get("count", 1)
    size = 8 if case.get("double") else 4
    return {"bytes": float(size * count * (m * k + k * n + m * n)),
            "flops": 2.0 * count * m * n * k}


def exact(case, seed):
    if case["kind"] not in ("mixed", "runs"):
        m, n, k, count = case["m"], case["n"], case["k"], case.get("count", 1)
        a, b, _ = _plain_inputs(case, seed)
        out = torch.empty(count * m * n, device="cuda", dtype=torch.float64)
        step = max(1, 1_000_000_000 // max(1, m * k + k * n))
        for i in range(0, count, step):
            j = min(count, i + step)
            x = a[i * m * k:j * m * k].double().view(-1, m, k)
            y = b[i * k * n:j * k * n].double()
            y = y.view(-1, n, k).transpose(1, 2) if case["tb"] else y.view(-1, k, n)
            out[i * m * n:j * m * n] = torch.bmm(x, y).reshape(-1)
        return out
    m, n, k, tb, own, a_at, b_at, c_at, c_len = _layout(case)
    a, b, _ = _grouped_inputs(case, seed)
    a, b = a.double(), b.double()
    out = torch.zeros(c_len, device="cuda", dtype=torch.float64)
    if case["kind"] == "runs":  # few shapes: all products of a shape at once
        key = (m * 64 + n) * 64 + k
        for v in np.unique(key):
            g = np.flatnonzero(key == v)
            mm, nn, kk = int(m[g[0]]), int(n[g[0]]), int(k[g[0]])

            def at(starts, length):
                return (torch.from_numpy(starts[g]).cuda()[:, None]
                        + torch.arange(length, device="cuda")[None, :])

            p = torch.bmm(a[at(a_at, mm * kk)].view(-1, mm, kk),
                          b[at(b_at, kk * nn)].view(-1, kk, nn))
            out.index_add_(0, at(c_at, mm * nn).reshape(-1), p.reshape(-1))
        return out
    for i in range(case["count"]):
        mm, nn, kk = int(m[i]), int(n[i]), int(k[i])
        x = a[a_at[i]:a_at[i] + mm * kk].view(mm, kk)
        y = b[b_at[i]:b_at[i] + kk * nn]
        y = y.view(nn, kk).t() if tb[i] else y.view(kk, nn)
        out[c_at[i]:c_at[i] + mm * nn].view(mm, nn).addmm_(x, y)
    return out
