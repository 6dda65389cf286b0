"""What a user of this library has it do, as cases to time.

Two kinds of work, both through the public face (`CudaBackend`, `KvCache`, `PassMeta`):

* "step": one forward pass of a decoder in the order of the reference's `Model::forward` (pending page
  copies, the pass's metadata, embedding, then per layer norm, qkv projection, attention, output
  projection, residual step, gated MLP, residual step, then the logits of every sequence's last row),
  with random weights.  A greedy step picks its tokens on the device too.
* "attend": the attention of a pass alone, layer after layer, as an engine with projections of its own
  calls it: `attention` on qkv rows, or (`halves`) `kv_append` and `attend` on final q, k and v.

Sizes are the benchmark's and the tests' (16 query / 4 KV heads, 32 / 8 heads, hidden 4096 with a
28672-row gate and up weight, a shared prefix of 1536 tokens, verification of five rows, prompt chunks
of 512 rows, 131072 keys, a window of 2048 keys), a model a quarter as wide, and ragged lengths.
"""
from types import SimpleNamespace

import numpy as np
import torch

from yaxus_b200 import CudaBackend
from yaxus_b200._lib import BF16, F16, F32, HEAD_DIM, PAGE
from yaxus_b200.backend import LayerMeta, Rope
from yaxus_b200.kvcache import KvCache

CACHE = {"f32": F32, "f16": F16, "bf16": BF16}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
EPS = 1e-6
# Norm offsets of the reference's model (crates/yaxus-model/src/lib.rs:24-27).
PRE_NORM, POST_MIXER_NORM, POST_MLP_NORM = 1.0, 0.2, 0.08944272

SMALL = dict(hidden=1024, inner=2816, hq=16, hkv=4, vocab=32000)
MEDIUM = dict(hidden=2048, inner=5632, hq=16, hkv=4, vocab=32000)
LARGE = dict(hidden=4096, inner=14336, hq=32, hkv=8, vocab=50257)

# What a case holds unless it says otherwise: `seqs` sequences of up to `ctx` cached tokens (`ragged`: from a
# quarter of that up), the first `shared` of them common to all, `rows` new tokens each; one sequence more
# with a chunk of `chunk` prompt rows after `chunk_ctx` (0: none); `fork`: the last sequence has just been
# forked inside a page, which leaves a page copy to make; `window`: keys seen in every other layer (0: all).
BASE = dict(cache="f16", layers=1, seqs=1, rows=1, ctx=1024, ragged=False, shared=0, chunk=0, chunk_ctx=0, fork=False, window=0)


def _step(name=None, **kw):
    c = dict(BASE, kind="step", greedy=True)
    c.update(kw)
    return dict(c, name=name) if name else c


def _attend(name=None, **kw):
    c = dict(BASE, kind="attend", halves=False, q="f32")
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One user's next token on a small model with the reference's own f32 cache: all latency.
        _step("token_small_f32", **SMALL, cache="f32", layers=4, ctx=1000),
        # The same on a large model: the weights stream past one row.
        _step("token_large_f16", **LARGE, cache="f16", layers=2, ctx=3000),
        # The serving loop: sixteen sequences over a common system prompt, every other layer windowed.
        _step("batch_decode_f16", **LARGE, cache="f16", layers=2, seqs=16, ctx=4096, ragged=True, shared=1536, window=2048),
        # Speculative decoding: one accepted token and four drafts for each of sixteen sequences.
        _step("verify_bf16", **LARGE, cache="bf16", seqs=16, rows=5, ctx=2048),
        # Reading prompts: a 512-row chunk of each of four, on top of 1024 tokens read before.
        _step("prompt_large_bf16", **LARGE, cache="bf16", seqs=4, rows=512, ctx=1024, greedy=False),
        # The second half of one user's prompt on a small model with an f32 cache.
        _step("prompt_small_f32", **SMALL, cache="f32", layers=2, rows=1000, ctx=1000, greedy=False),
        # Continuous batching: eleven sequences decode, one of them just forked, while a prompt of 300 rows comes in.
        _step("mixed_f16", **MEDIUM, cache="f16", layers=2, seqs=11, ctx=1500, ragged=True, chunk=300, chunk_ctx=200, fork=True),
        # Attention of one sequence on the f32 cache, 1024 keys: the smallest call.
        _attend("attend_single_f32", hq=16, hkv=4, cache="f32", layers=2, ctx=1023),
        # Attention of the serving loop over four layers.
        _attend("attend_batch_f16", hq=32, hkv=8, cache="f16", layers=4, seqs=16, ctx=4096, ragged=True, shared=1536, halves=True),
        # One very long context, a full and a windowed layer.
        _attend("attend_long_f16", hq=32, hkv=8, cache="f16", layers=2, ctx=131071, window=2048, halves=True, q="f16"),
        # The last 512-row chunk of eight prompts of 4096 tokens, all bf16.
        _attend("attend_prompt_bf16", hq=32, hkv=8, cache="bf16", seqs=8, rows=512, ctx=3584, halves=True, q="bf16"),
        # Twelve sequences of ragged length on the f32 cache.
        _attend("attend_batch_f32", hq=16, hkv=4, cache="f32", layers=2, seqs=12, ctx=2500, ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    cache = rng.choice(["f32", "f16", "bf16"])
    heads = rng.choice([(16, 4), (32, 8), (8, 2), (16, 8), (24, 8)])
    window = rng.choice([0, 0, _log(rng, 48, 2048)])
    what = rng.choice(["token", "batch", "verify", "prompt", "mixed", "attend_few", "attend_many", "attend_prompt", "attend_long"])
    common = dict(cache=cache, hq=heads[0], hkv=heads[1], window=window, layers=rng.choice([1, 2]))
    model = dict(hidden=128 * _log(rng, 6, 32), inner=128 * _log(rng, 14, 112), vocab=_log(rng, 8000, 50257))
    if what == "token":
        return _step(**common, **model, ctx=_log(rng, 30, 4000))
    if what == "batch":
        shared = rng.choice([0, 128 * _log(rng, 1, 12)])
        return _step(**common, **model, seqs=_log(rng, 2, 32), ctx=shared + _log(rng, 200, 2600), ragged=True, shared=shared)
    if what == "verify":
        return _step(**common, **model, seqs=_log(rng, 1, 16), rows=rng.randint(2, 8), ctx=_log(rng, 100, 2048), ragged=rng.random() < 0.5)
    if what == "prompt":
        if cache == "f32":
            return _step(**dict(common, hq=16, hkv=4), **model, rows=_log(rng, 70, 1000), ctx=_log(rng, 1, 1000), greedy=False)
        return _step(**common, **model, seqs=rng.choice([1, 2, 4]), rows=_log(rng, 70, 512), ctx=_log(rng, 1, 1024), greedy=False)
    if what == "mixed":
        return _step(**common, **model, seqs=_log(rng, 2, 16), ctx=_log(rng, 200, 2000), ragged=True, chunk=_log(rng, 20, 400),
                     chunk_ctx=_log(rng, 1, 500), fork=rng.random() < 0.5)
    q = rng.choice(["f32", "f32" if cache == "f32" else cache])
    common.update(halves=rng.random() < 0.5, q=q)
    if what == "attend_few":
        return _attend(**common, ctx=_log(rng, 20, 8000), rows=rng.choice([1, 1, 3]))
    if what == "attend_many":
        shared = rng.choice([0, 128 * _log(rng, 1, 12)])
        return _attend(**common, seqs=_log(rng, 2, 32), ctx=shared + _log(rng, 200, 2600), ragged=True, shared=shared, rows=rng.choice([1, 1, 5]))
    if what == "attend_prompt":
        if cache == "f32":
            return _attend(**dict(common, hq=16, hkv=4), rows=_log(rng, 70, 1000), ctx=_log(rng, 1, 1000))
        return _attend(**common, seqs=rng.choice([1, 2, 4, 8]), rows=_log(rng, 70, 512), ctx=_log(rng, 1, 3584))
    return _attend(**common, ctx=_log(rng, 10000, 100000))


def _lengths(case):
    """Cached tokens of every sequence, by the case alone (no two seeds differ in work)."""
    n, ctx = case["seqs"], case["ctx"]
    least = max(case["shared"], ctx // 4) if case["ragged"] else ctx
    out = [least + int((ctx - least) * ((0.5 + 0.6180339887 * i) % 1.0)) for i in range(n)]
    if case["ragged"]:
        out[0] = ctx
    return out


def _windows(case):
    n = case["layers"]
    return [case["window"] if case["window"] and (n == 1 or l % 2 == 1) else None for l in range(n)]


_BACKEND = []


def _backend():
    """One backend to a process, as a server holds one."""
    if not _BACKEND:
        _BACKEND.append(CudaBackend(0))
    return _BACKEND[0]


def _context(b, case, rng, gen):
    """The KV cache with every sequence's context in it, and the pass to run: (kv, metas, pass, page copies)."""
    lengths, shared = _lengths(case), case["shared"]
    longest = max(lengths + [case["chunk_ctx"]]) + max(case["rows"], case["chunk"])
    pages = sum((n + case["rows"]) // PAGE + 2 for n in lengths) + (case["chunk_ctx"] + case["chunk"]) // PAGE + 4
    max_pos = (longest // PAGE + 2) * PAGE
    metas = [LayerMeta(index=l, window=w, rope=Rope.default()) for l, w in enumerate(_windows(case))]
    kv = b.new_kv(case["hkv"], metas, pages, max_pos, CACHE[case["cache"]])
    book = KvCache(pages, max_pos)
    kvd = case["hkv"] * HEAD_DIM
    fill = TORCH[case["cache"]]

    def ids(n):
        return rng.integers(0, case.get("vocab", 32000), n)

    def append(items):
        meta = book.append(items)
        for src, dst in book.take_copies():
            b.copy_page(kv, src, dst)
        b.begin_pass(meta)
        for l in range(case["layers"]):
            k, v = (torch.randn(meta.rows, kvd, generator=gen, device=b.device).to(fill) for _ in range(2))
            b.kv_append(kv, l, k, v)

    first = book.new_seq()
    if shared:
        append([(first, ids(shared))])
    # (page tables fork at whole pages: the prefix is held once)
    seqs = [first] + [book.fork(first, shared) if shared else book.new_seq() for _ in lengths[1:]]
    if case["chunk"]:
        seqs.append(book.new_seq())
        lengths = lengths + [case["chunk_ctx"]]
    # Contexts grow side by side, as they do in service, so that a sequence's pages lie scattered.
    left = [n - (shared if i < case["seqs"] else 0) for i, n in enumerate(lengths)]
    part = 256 if len(seqs) > 1 else 16384
    while any(left):
        items = []
        for i, s in enumerate(seqs):
            n = min(left[i], part)
            if n:
                items.append((s, ids(n)))
                left[i] -= n
        append(items)
    if case["fork"]:
        at = case["seqs"] - 1
        old, n = seqs[at], lengths[at]
        seqs[at] = book.fork(old, n - 1 if n % PAGE == 0 else n)
    new = [case["rows"]] * case["seqs"] + ([case["chunk"]] if case["chunk"] else [])
    meta = book.append([(s, ids(n)) for s, n in zip(seqs, new)])
    return kv, metas, meta, book.take_copies()


def prepare(case, seed):
    b = _backend()
    rng, gen = np.random.default_rng(seed), torch.Generator(device=b.device)
    gen.manual_seed(seed)
    kv, metas, meta, copies = _context(b, case, rng, gen)
    hq, hkv = case["hq"], case["hkv"]
    normal = lambda *shape: torch.randn(*shape, generator=gen, device=b.device)  # noqa: E731
    vector = lambda n: b.load_weight(0.1 * normal(n))                            # noqa: E731
    s = SimpleNamespace(b=b, case=case, kv=kv, metas=metas, meta=meta, copies=copies, hq=hq)
    if case["kind"] == "step":
        hidden, inner, vocab = case["hidden"], case["inner"], case["vocab"]
        matrix = lambda n, k: b.load_weight(normal(n, k).mul_(k ** -0.5))        # noqa: E731
        s.embed, s.norm, s.head = b.load_weight(normal(vocab, hidden)), vector(hidden), matrix(vocab, hidden)
        s.layers = [SimpleNamespace(
            pre_mixer=vector(hidden), qkv=matrix((hq + 2 * hkv) * HEAD_DIM, hidden), q_norm=vector(HEAD_DIM), k_norm=vector(HEAD_DIM),
            o=matrix(hidden, hq * HEAD_DIM), post_mixer=vector(hidden), pre_mlp=vector(hidden), gate_up=matrix(2 * inner, hidden),
            down=matrix(hidden, inner), post_mlp=vector(hidden)) for _ in metas]
    elif case["halves"]:
        fill = TORCH[case["cache"]]
        s.q = [normal(meta.rows, hq * HEAD_DIM).to(TORCH[case["q"]]) for _ in metas]
        s.k, s.v = ([normal(meta.rows, hkv * HEAD_DIM).to(fill) for _ in metas] for _ in range(2))
    else:
        s.q_norm, s.k_norm = vector(HEAD_DIM), vector(HEAD_DIM)
        s.qkv = [normal(meta.rows, (hq + 2 * hkv) * HEAD_DIM) for _ in metas]
    return s


def _forward(s):
    b, m = s.b, s.meta
    for src, dst in s.copies:
        b.copy_page(s.kv, src, dst)
    b.begin_pass(m)
    x = b.embed(s.embed)
    h = b.rmsnorm(x, s.layers[0].pre_mixer, PRE_NORM, EPS)
    for i, l in enumerate(s.layers):
        a = b.attention(b.matmul(h, l.qkv), l.q_norm, l.k_norm, s.kv, s.hq, EPS, s.metas[i])
        h = b.add_norm(x, b.matmul(a, l.o), l.post_mixer, POST_MIXER_NORM, l.pre_mlp, PRE_NORM, EPS)
        d = b.matmul(b.matmul_glu(h, l.gate_up), l.down)
        nxt = s.layers[i + 1].pre_mixer if i + 1 < len(s.layers) else s.norm
        h = b.add_norm(x, d, l.post_mlp, POST_MLP_NORM, nxt, PRE_NORM, EPS)
    # A verification needs the logits of every row, a decode or prompt pass those of each sequence's last.
    every = len(m.last) == m.rows or 1 < s.case["rows"] <= 8
    return b.matmul(h if every else b.select_rows(h, m.last), s.head)


def run(state):
    b, case = state.b, state.case
    if case["kind"] == "step":
        logits = _forward(state)
        if not case["greedy"]:
            return {"logits": logits}
        tokens = b.argmax_rows(logits)
        # (on a 16-bit cache two correct implementations may pick apart where two logits all but tie)
        return {"logits": logits, "tokens": tokens} if case["cache"] == "f32" else {"logits": logits}
    b.begin_pass(state.meta)
    out = []
    for l, meta in enumerate(state.metas):
        if case["halves"]:
            b.kv_append(state.kv, l, state.k[l], state.v[l])
            out.append(b.attend(state.kv, l, state.q[l], state.hq, out_dtype=state.q[l].dtype))
        else:
            out.append(b.attention(state.qkv[l], state.q_norm, state.k_norm, state.kv, state.hq, EPS, meta))
    return out


def work(case):
    rows = [case["rows"]] * case["seqs"] + ([case["chunk"]] if case["chunk"] else [])
    ctx = _lengths(case) + ([case["chunk_ctx"]] if case["chunk"] else [])
    t, hq, hkv = sum(rows), case["hq"], case["hkv"]
    size = 4 if case["cache"] == "f32" else 2
    qsize = 2 if case["kind"] == "attend" and case["halves"] and case["q"] != "f32" else 4
    nbytes = flops = 0
    for w in _windows(case):
        private = common = seen = 0
        for n, c in zip(rows, ctx):
            lo = max(0, c + 1 - w) if w else 0
            shared = case["shared"] if c >= case["shared"] else 0
            common = max(common, max(0, shared - lo))
            private += c + n - max(lo, shared)
            if w:
                seen += sum(min(p + 1, w) for p in range(c, c + n))
            else:
                seen += n * c + n * (n + 1) // 2
        nbytes += (private + common) * 2 * hkv * HEAD_DIM * size      # keys and values read (this pass's rows among them)
        nbytes += t * 2 * hkv * HEAD_DIM * size                       # and this pass's written
        if case["kind"] == "attend":
            new = size if case["halves"] else 4
            nbytes += t * HEAD_DIM * (2 * hq * qsize + 2 * hkv * new)  # queries in, rows out; new keys and values in
        flops += 4 * HEAD_DIM * hq * seen
    if case["kind"] == "step":
        hidden, inner, vocab = case["hidden"], case["inner"], case["vocab"]
        params = hidden * ((2 * hq + 2 * hkv) * HEAD_DIM + 3 * inner)
        logits = t if 1 < case["rows"] <= 8 else len(rows)
        nbytes += 2 * (case["layers"] * params + vocab * hidden) + t * hidden * 2 + logits * vocab * 4
        flops += 2 * t * params * case["layers"] + 2 * logits * vocab * hidden
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Four times (about) the 2-norm error against the same path in 64-bit arithmetic on the same stored keys and values.

    Measured over the listed and forty drawn cases: attention on an f32 cache 3e-7; a step on one 3e-6, up to 9e-6
    (activations go to the matmuls as a high and a low bf16 part, 16 bits of mantissa); f32 queries on a bf16 cache
    (both operands in two parts) and a step on one up to 3e-5 (a new key or value may round to the other neighbour);
    attention on an f16 cache 2.8e-4 (queries and probabilities are f16), of which a step's logits show 8e-5; rows
    written as bf16 1.7e-3."""
    if case["kind"] == "step":
        return {"rel": {"f32": 4e-5, "bf16": 1.2e-4, "f16": 3.5e-4}[case["cache"]]}
    if case["halves"] and case["q"] == "bf16":
        return {"rel": 7e-3}
    return {"rel": {"f32": 3e-6, "bf16": 1.2e-4, "f16": 1.2e-3}[case["cache"]]}
