"""Norm, RoPE and append of a pass large enough that a warp takes several heads of a row: the same cache,
bit for bit, as passes small enough for a warp a head leave."""
import numpy as np
import pytest
import torch

from oracle.check import assert_close
from yaxus_b200._lib import BF16, F16, F32
from yaxus_b200.backend import LayerMeta, Rope
from yaxus_b200.kvcache import PassMeta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,kv_dtype", [(12, 3, F16), (8, 1, BF16), (5, 5, F32)])   # 18, 10 and 15 heads: the last warp of a row is not full
def test_many_rows_like_few(backend, hq, hkv, kv_dtype):
    rows, pages = 1250, 10
    table = np.random.default_rng(hq).permutation(pages)
    gen = torch.Generator(device=backend.device)
    gen.manual_seed(hq)
    qkv = torch.randn(rows, (hq + 2 * hkv) * 128, generator=gen, device=backend.device)
    norms = [0.1 * torch.randn(128, generator=gen, device=backend.device) for _ in range(2)]
    layer = LayerMeta(index=0, window=200, rope=Rope.default())
    caches, outs = [], []
    for step in (rows, 125):
        kv = backend.new_kv(hkv, [layer], pages, pages * 128, kv_dtype)
        out = []
        for r in range(0, rows, step):
            backend.begin_pass(PassMeta.from_rows([(0, p) for p in range(r, r + step)], [table]))
            out.append(backend.attention(qkv[r:r + step].contiguous(), *norms, kv, hq, 1e-6, layer))
        outs.append(backend.to_host(torch.cat(out)))
        caches.append(backend.read_pages(kv, 0, 0, pages))
        kv.close()
    assert np.array_equal(caches[0][0], caches[1][0]) and np.array_equal(caches[0][1], caches[1][1])
    assert_close(outs[0], outs[1], what="outputs")
