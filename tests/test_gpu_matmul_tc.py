"""The matmul kernels at the edges of their tiles: ragged weight rows and pass rows, one and two tiles of
pass rows, tiles shared along k by several CTAs or CTA pairs, whole tiles before and after them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# x = hi + lo drops at most 2^-17 of each term (half a unit of lo's last place, against hi); the f32 sums
# of 2 K terms err by a few 2^-24 of the terms' magnitudes.
TOL = 2.0 ** -17 + 32 * 2.0 ** -24


def dev(backend, x):
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).to(backend.device)


def magnitudes(x, w_bits):
    """The sum of every product's terms' magnitudes."""
    return np.abs(x.astype(np.float64)) @ np.abs((w_bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)).T


def inputs(oracle, t, n, k):
    rng = np.random.default_rng(t * 7919 + n + k)
    x = rng.standard_normal((t, k)).astype(np.float32)
    return x, oracle.to_bf16((rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32))


@pytest.mark.parametrize("t,n,k", [
    # few rows: each size of operand; one k step a CTA, a tile of 148 shares and more, several whole tiles a CTA
    (1, 1, 128), (7, 127, 256), (8, 129, 1024), (9, 300, 128), (16, 1000, 640), (17, 4100, 256), (32, 257, 1152),
    (1, 128, 19200), (3, 40000, 128), (32, 39000, 128),
    # many rows: fewer tiles than pairs; rounds and a remainder
    (33, 1, 128), (64, 255, 128), (65, 257, 384), (280, 300, 512), (256, 256, 1024), (257, 300, 640),
    (300, 9700, 256), (513, 6400, 128), (200, 18944, 128),
    (40, 19300, 128), (49, 18000, 256), (128, 19201, 256), (97, 38400, 128)])
def test_matmul_tiles(backend, oracle, t, n, k):
    x, w_bits = inputs(oracle, t, n, k)
    w, ref = backend.load_weight(w_bits), oracle.matmul(x, w_bits)
    xd = dev(backend, x)
    first = backend.to_host(backend.matmul(xd, w))
    assert (np.abs(first - ref) <= TOL * magnitudes(x, w_bits)).all()
    # the arrival counters are left clean, and shares are added up in one order
    assert np.array_equal(backend.to_host(backend.matmul(xd, w)), first)


@pytest.mark.parametrize("t,inner,k", [
    (1, 16, 128), (8, 1040, 256), (13, 48, 1024), (32, 9696, 128), (5, 24, 256),
    (33, 16, 128), (48, 144, 1024), (257, 1040, 256), (100, 24, 256), (150, 9696, 128), (35, 9696, 128), (60, 19456, 128),
    (300, 9696, 256)])                                      # two tiles of pass rows, two whole rounds of tiles and a remainder
def test_glu_tiles(backend, oracle, t, inner, k):
    x, w_bits = inputs(oracle, t, 2 * inner, k)
    w = backend.load_weight(w_bits)
    xd = dev(backend, x)
    got = backend.to_host(backend.matmul_glu(xd, w))
    # silu(g) u moves by at most 1.1 |u| dg + |g| du: each product errs by TOL times its terms' magnitudes
    s = oracle.matmul(x, w_bits)
    mag = magnitudes(x, w_bits)
    g, u = np.abs(s[:, :inner]), np.abs(s[:, inner:])
    bound = TOL * (1.1 * u * mag[:, :inner] + g * mag[:, inner:]) + 1e-6 * np.maximum(1.0, g * u)
    assert (np.abs(got - oracle.swiglu(s)) <= bound).all()
    assert np.array_equal(backend.to_host(backend.matmul_glu(xd, w)), got)


@pytest.mark.parametrize("t,n,k", [(170, 18944, 3072), (512, 9700, 6016)])   # 18 and 32 steps, the most
def test_a_longer_first_chain(backend, t, n, k):
    # more than 160 rows a tile (two accumulators) and whole tiles of 48 and 94 k steps: a piece begins with a longer chain
    gen = torch.Generator(device=backend.device)
    gen.manual_seed(k)
    x = torch.randn(t, k, generator=gen, device=backend.device)
    w = (torch.randn(n, k, generator=gen, device=backend.device) * k ** -0.5).bfloat16()
    got = backend.matmul(x, w)
    backend.sync()
    xd, wd = x.double(), w.double().T
    # an accumulator is added to up to 256 times (32 steps, four of 16 k in each, two parts) and may drop its last place each time
    assert ((got - xd @ wd).abs() <= (2.0 ** -17 + 256 * 2.0 ** -23) * (xd.abs() @ wd.abs())).all()


@pytest.mark.parametrize("t,n,k", [(275, 34914, 1152), (262, 1460, 6784), (202, 4108, 3712), (90, 527, 13312), (20, 11264, 2048)])
def test_sums_lose_no_more_than_a_library_product(backend, t, n, k):
    gen = torch.Generator(device=backend.device)
    gen.manual_seed(n)
    x = torch.randn(t, k, generator=gen, device=backend.device)
    w = (torch.randn(n, k, generator=gen, device=backend.device) * k ** -0.5).bfloat16()
    got = backend.matmul(x, w)
    backend.sync()
    hi = x.bfloat16()
    parts = hi.double() + (x - hi.float()).bfloat16().double()   # what reaches the tensor cores, so that the sums' error stands alone
    want = parts @ w.double().T
    # two library products, one for each part: 0.9 to 1.2e-6 of these; chains of 16 steps 2.1e-6
    assert (got - want).norm() <= 1.4e-6 * want.norm()


@pytest.mark.parametrize("t", [5, 70])
def test_unaligned_rows(backend, oracle, t):
    # pass rows that start 8 bytes past a 16-byte boundary
    x, w_bits = inputs(oracle, t, 200, 256)
    store = torch.zeros(t * 256 + 2, dtype=torch.float32, device=backend.device)
    xd = store[2:].view(t, 256)
    xd.copy_(torch.from_numpy(x))
    got = backend.to_host(backend.matmul(xd, backend.load_weight(w_bits)))
    assert (np.abs(got - oracle.matmul(x, w_bits)) <= TOL * magnitudes(x, w_bits)).all()


@pytest.mark.parametrize("t,n,glu", [(1, 60000, 0), (1, 60000, 1), (32, 4096, 0), (70, 4096, 0), (70, 8192, 1)])
def test_a_result_over_its_own_rows(backend, t, n, glu):
    k = 4096
    gen = torch.Generator(device=backend.device)
    gen.manual_seed(t)
    x, w = torch.randn(t, k, generator=gen, device=backend.device), torch.randn(n, k, generator=gen, device=backend.device).mul_(k ** -0.5).bfloat16()
    want = (backend.matmul_glu if glu else backend.matmul)(x, w)
    both = torch.zeros_like(want)
    both.view(-1)[:t * k] = x.view(-1)
    call = backend._L.yx_matmul_glu if glu else backend._L.yx_matmul
    assert call(backend._ctx, both.data_ptr(), w.data_ptr(), t, n, k, both.data_ptr()) == 0
    backend.sync()
    assert torch.equal(both, want)


def test_more_outputs_than_a_32_bit_thread_index_reaches(backend):
    # a warp an output: 2^27 outputs are 2^32 threads
    t, n = 4097, 32768
    gen = torch.Generator(device=backend.device)
    gen.manual_seed(11)
    x, w = torch.randn(t, 1, generator=gen, device=backend.device), backend.load_weight(torch.randn(n, 1, generator=gen, device=backend.device))
    torch.full((t, n), float("nan"), device=backend.device)               # (given back at once: the result's memory, most likely)
    got = backend.matmul(x, w)
    backend.sync()
    assert torch.equal(got, x * w.float().T)                              # one product each: the same rounding


def test_no_scratch_grows_where_fewer_rows_follow_more():
    # Calls recorded into a graph after passes of as many rows: growing a buffer would
    # synchronise the stream, which ends the recording.
    from yaxus_b200 import CudaBackend
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        b = CudaBackend(0, stream=stream)
        x = torch.randn(512, 256, device=b.device)
        few, many, odd = (torch.randn(n, 256, device=b.device).bfloat16() for n in (256, 9000, 2 * 24))
        for rows in (1, 512):
            b.matmul(x[:rows], few)
        b.matmul(x[:1], many)
        b.matmul_glu(x[:1], odd)
        b.sync()
        calls = [(b.matmul, 16, many), (b.matmul, 300, many), (b.matmul, 100, many), (b.matmul_glu, 16, odd)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outs = [op(x[:rows], w) for op, rows, w in calls]
        graph.replay()
        b.sync()
        for out, (op, rows, w) in zip(outs, calls):
            assert torch.equal(out, op(x[:rows], w))
    del graph
    b.close()
