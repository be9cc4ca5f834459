"""A cached call is replayed only under the settings that it was captured with:
after LibShalom_set_tma the other kernel runs (on this shape it adds the
correction products in another order)."""
import numpy as np
import pytest

import libshalom_b200 as ls
from oracle import oracle as orc
from tests._util import to_dev, to_host

pytestmark = pytest.mark.gpu


def test_operand_staging_is_part_of_the_key():
    import torch
    M, N, K = 256, 32, 4096
    A, B = to_dev(orc.uniform_f32(1, M * K)), to_dev(orc.uniform_f32(2, K * N))
    C = to_dev(np.zeros(M * N, np.float32))
    s = torch.cuda.Stream()
    ls.set_precision(ls.PREC_BF16X6)
    ls.set_splitk(1)
    want = {}
    for tma in (True, False):
        ls.set_tma(tma)
        ls.sgemm_mp(0, 0, C, A, B, M, N, K)
        want[tma] = to_host(C).copy()
    assert not np.array_equal(want[True], want[False])
    ls.set_stream(s)
    try:
        ls.set_graph_cache(True)
        for tma in (True, True, True, False, False, True):
            ls.set_tma(tma)
            C.zero_()
            torch.cuda.synchronize()
            ls.sgemm_mp(0, 0, C, A, B, M, N, K)
            s.synchronize()
            assert np.array_equal(to_host(C), want[tma])
    finally:
        ls.set_graph_cache(False)
        ls.set_stream(None)
