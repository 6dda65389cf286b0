"""Attention over f32 caches a row at a time: parts of a row whose sums are no numbers."""
import numpy as np
import pytest
import torch

from oracle.check import assert_close, dev, load, oracle_step
from yaxus_b200 import workloads as W
from yaxus_b200._lib import F16, F32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("ctx,rows,kernel", [(40, 1, 1), (1500, 1, 1), (1500, 40, 3)])   # one part, many parts; the tiled kernel and its merge
def test_a_key_without_a_score_shows(backend, oracle, bad, ctx, rows, kernel):
    """Every row that sees a key of score NaN or +inf comes out as no number, however its keys are cut; others are untouched."""
    s = W.build("f32-no-score", 21, 16, 4, F32, [ctx, 900], [rows, rows])
    s.q[:, ::128] = np.abs(s.q[:, ::128]) + 0.1          # (dim 0 of every head: a score of +inf, never -inf)
    want = oracle_step(oracle, s)
    at = ctx // 2
    s.k_bits[int(s.tables[0][at // 128]) * 128 + at % 128, ::128] = bad
    kv = load(backend, s)
    backend.begin_pass(s.meta)
    backend.kv_append(kv, 0, dev(backend, s.k_new), dev(backend, s.v_new))
    q = dev(backend, s.q)
    backend.set_tuning(force_path=kernel)
    got = backend.to_host(backend.attend(kv, 0, q, s.hq)).reshape(2 * rows, s.hq, 128)
    assert backend.last_plan().launches == (1 if kernel == 1 else 2)
    assert not np.isfinite(got[:rows]).any()
    assert_close(got[rows:].reshape(rows, -1), want[rows:], abs_tol=2e-5, rel_tol=0.0, what="the rows beside it")
    _, l, o = (backend.to_host(t) for t in backend.attend_partial(kv, 0, q, s.hq, None, 0, 1 << 40))
    backend.set_tuning()
    assert not np.isfinite(l[:rows]).any()
    assert_close(o[rows:] / l[rows:, :, None], got[rows:], abs_tol=2e-5, rel_tol=0.0, what="triples of the rows beside it")
    kv.close()


@pytest.mark.parametrize("dtype", [F32, F16])
def test_a_result_over_its_queries(backend, dtype):
    # A row of 16-bit results lies over the queries of a row half as far up.
    s = W.build("f32-over", 23, 16, 4, F32, [2500] * 32 + [10] * 32, [1] * 64)
    kv = load(backend, s)
    backend.begin_pass(s.meta)
    backend.kv_append(kv, 0, dev(backend, s.k_new), dev(backend, s.v_new))
    q = dev(backend, s.q)
    want = backend.attend(kv, 0, q, s.hq, out_dtype=torch.float32 if dtype == F32 else torch.float16)
    assert backend.last_plan().launches == 1
    assert backend._L.yx_attend(backend._ctx, kv._h, 0, q.data_ptr(), F32, s.hq, -1, q.data_ptr(), dtype) == 0
    backend.sync()
    assert torch.equal(q.view(-1).view(want.dtype)[:want.numel()], want.view(-1))
    kv.close()
