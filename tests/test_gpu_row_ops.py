"""The row operators at the edges of their kernels' ranges: vectors a thread holds, columns that need
the scalar form, parts of an argmax row, index lists past what kernel parameters carry."""
import numpy as np
import pytest
import torch

from yaxus_b200.kvcache import PassMeta

pytestmark = pytest.mark.gpu


def dev(backend, x):
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).to(backend.device)


@pytest.mark.parametrize("rows,cols", [(1, 4), (3, 1024), (2, 1028), (2, 4096), (2, 4100), (1, 8192), (1, 8196), (3, 1023)])
def test_norms(backend, oracle, rows, cols):
    rng = np.random.default_rng(cols)
    x, d = (rng.standard_normal((rows, cols)).astype(np.float32) for _ in range(2))
    w1, w2 = (0.1 * rng.standard_normal(cols).astype(np.float32) for _ in range(2))
    # Sums of `cols` squares in another order: cols * 2^-24 of the sum at most, half of it after the root.
    tol = 4e-7 + cols * 2.0 ** -25
    ref = oracle.rmsnorm(d, w1, 1.0, 1e-6)
    got = backend.to_host(backend.rmsnorm(dev(backend, d), dev(backend, w1), 1.0, 1e-6))
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    xd = dev(backend, x)
    out = backend.add_norm(xd, dev(backend, d), dev(backend, w1), 0.2, dev(backend, w2), 1.0, 1e-6)
    x_ref, out_ref = oracle.add_norm(x, d, w1, 0.2, w2, 1.0, 1e-6)
    assert np.abs(backend.to_host(xd) - x_ref).max() <= tol * np.abs(x_ref).max()
    assert np.abs(backend.to_host(out) - out_ref).max() <= 2 * tol * np.abs(out_ref).max()


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 2048), (2, 2049), (1, 600001), (130, 4097)])
def test_argmax(backend, oracle, rows, cols):
    x = np.random.default_rng(cols).standard_normal((rows, cols)).astype(np.float32)
    x[0, cols - 1] = x[0, cols // 2] = 9.0            # a tie across parts: the first one
    for _ in range(2):                                # the arrival counters are left clean
        assert np.array_equal(backend.argmax_rows(dev(backend, x)), oracle.argmax_rows(x))


@pytest.mark.parametrize("rows,h", [(1, 8), (513, 64), (512, 2056), (3, 30)])
def test_gathers(backend, oracle, rows, h):
    rng = np.random.default_rng(h)
    bits = oracle.to_bf16(rng.standard_normal((700, h)).astype(np.float32))
    meta = PassMeta.from_rows([(0, p) for p in range(rows)], [np.arange(1 + rows // 128)])
    meta.ids = rng.integers(0, 700, rows).astype(np.uint32)
    backend.begin_pass(meta)
    e = backend.embed(backend.load_weight(bits))
    want = oracle.embed(bits, meta.ids)
    assert np.array_equal(backend.to_host(e), want)
    sel = rng.integers(0, rows, rows)
    assert np.array_equal(backend.to_host(backend.select_rows(e, sel)), want[sel])


@pytest.mark.parametrize("h", [65535 * 2048 + 8, 65535 * 2048 + 1])
def test_gathers_of_rows_wider_than_a_grid(backend, h):
    table = torch.arange(h, device=backend.device, dtype=torch.int32).remainder_(251).to(torch.bfloat16).view(1, h)
    backend.begin_pass(PassMeta.from_rows([(0, 0)], [[0]]))
    e = backend.embed(table)
    backend.sync()
    assert torch.equal(e, table.float())
    del table
    assert torch.equal(backend.select_rows(e, [0]), e)
    backend.sync()
