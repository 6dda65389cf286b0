"""Attention over f32 caches at the edges of its tiles of 32 keys and 16, 32 or 64 queries: ragged
contexts and windows, every grouping of heads, shared prefixes, values that masked keys may hold.  The same
through the kernel that takes a row at a time, and which of the two a pass goes to."""
import numpy as np
import pytest

from oracle.check import assert_close, dev, load, oracle_step, run_step
from yaxus_b200 import workloads as W
from yaxus_b200._lib import F32

pytestmark = pytest.mark.gpu


def close(got, want, what):
    # Outputs are means of values of size one: f32 scores of size ten err by 1e-6 or so, and so do their exponentials.
    assert_close(got, want, abs_tol=2e-5, rel_tol=0.0, what=what)


ROWS, TILES = 1, 3   # force_path; the row kernel is one launch, the tiled one and the merge behind it are two


@pytest.mark.parametrize("kernel", [ROWS, TILES])
@pytest.mark.parametrize("hq,hkv,ctx,rows,window", [
    (2, 2, [0, 31, 32, 33], [1, 1, 1, 1], None),
    (4, 1, [127, 128, 500, 0], [1, 4, 5, 8], None),          # 4, 16, 20 and 32 queries an item
    (6, 2, [95, 700], [21, 16], 33),                         # 48 of 64 queries
    (16, 1, [64, 250, 3], [1, 2, 5], 32),                    # four rows an item at most
    (5, 5, [10, 300], [64, 65], 31),
    (8, 2, [0, 129], [130, 70], None),
    (8, 2, [600], [100], 1),
    (16, 4, [2000], [1], 200)])
def test_edges(backend, oracle, hq, hkv, ctx, rows, window, kernel):
    s = W.build("f32-edges", 100 + hq, hq, hkv, F32, ctx, rows, window=window)
    kv = load(backend, s)
    backend.set_tuning(force_path=kernel)
    got = run_step(backend, kv, s)
    backend.set_tuning()
    assert backend.last_plan().path == 1 and backend.last_plan().launches == (1 if kernel == ROWS else 2)
    close(got, oracle_step(oracle, s), "f32 tiles" if kernel == TILES else "f32 rows")
    kv.close()


def test_shared_prefix_and_row_kernel(backend, oracle):
    s = W.build("f32-shared", 5, 8, 2, F32, [300, 256, 700, 400, 290, 300], [1, 1, 1, 1, 1, 5], shared_prefix=256)
    kv = load(backend, s)
    want = oracle_step(oracle, s)
    backend.set_tuning(force_path=TILES)
    got = run_step(backend, kv, s)
    assert backend.last_plan().shared_groups > 0
    close(got, want, "shared prefix")
    backend.set_tuning(force_path=ROWS)
    rows = run_step(backend, kv, s)
    backend.set_tuning()
    close(rows, want, "a row at a time")
    kv.close()


RAGGED = [2500 - 160 * i for i in range(12)]


@pytest.mark.parametrize("hq,hkv,ctx,rows,window,launches", [
    (16, 4, RAGGED, [1] * 12, None, 1), (16, 4, RAGGED, [1] * 11 + [5], None, 1),     # one sequence of many rows does not
    (16, 4, RAGGED, [1] * 11 + [40], None, 1), (16, 4, RAGGED, [5] * 12, None, 2),    # decide for eleven of one
    (16, 4, [1000], [16], None, 1), (16, 4, [1000], [100], None, 2), (16, 4, [1000], [100], 20, 1),
    (8, 8, [1000], [3], None, 1), (8, 8, [1000], [16], None, 2)])
def test_the_quicker_kernel_takes_a_pass(backend, oracle, hq, hkv, ctx, rows, window, launches):
    s = W.build("f32-choice", 6, hq, hkv, F32, ctx, rows, window=window)
    kv = load(backend, s)
    got = run_step(backend, kv, s)
    assert backend.last_plan().launches == launches
    close(got, oracle_step(oracle, s), "f32")
    kv.close()


@pytest.mark.parametrize("kernel", [ROWS, TILES])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_masked_value_reaches_nobody(backend, oracle, bad, kernel):
    # The last row of a chunk holds a value that is no number; rows before it do not see that key.
    s = W.build("f32-masked", 9, 8, 2, F32, [40], [37])
    want = oracle_step(oracle, s)
    kv = load(backend, s)
    v, k = s.v_new.copy(), s.k_new.copy()
    v[-1], k[-1] = bad, bad
    backend.begin_pass(s.meta)
    backend.kv_append(kv, 0, dev(backend, k), dev(backend, v))
    backend.set_tuning(force_path=kernel)
    got = backend.to_host(backend.attend(kv, 0, dev(backend, s.q), s.hq))
    backend.set_tuning()
    close(got[:-1], want[:-1], "rows before it")
    assert not np.isfinite(got[-1]).all()
    kv.close()
