"""Attention over latents as a part, with heads of 128 and prompt portions long enough for expanded keys and values: whole,
behind a cached context, beside single tokens and short portions, against the plain implementations; with row widths that
the expanded form's copies cannot start on, and beside a request whose numbers are not finite."""
import pytest
import torch

import plain_zufotar as PF
import plain_zukotar as PK
import zufotar_tiny as ZF
import zukotar_tiny as ZK
from test_gpu_zufotar import lat_weights
from test_gpu_zukotar import DEV, DT, Harness, as_stored, bind, latent_weights, rel, rnd

pytestmark = pytest.mark.gpu
W, EPS, ROWS = 64, 1e-6, 300


@pytest.fixture(autouse=True)
def expand_small_steps(monkeypatch):
    """The sizes below show what there is to see and are not worth their launches."""
    from rllm_b200.kernels import backend
    monkeypatch.setattr(backend, "LATENT_GAIN", -1e9)
    monkeypatch.setattr(backend, "LATENT_GAIN_MIXED", -1e9)


def built(heads, rot, rank, window=None, q_rank=None):
    """(part, weights, plain implementation) of a layer with a gate a head, or (q_rank) a query latent and a gate an output."""
    from rllm_b200.parts import InterleavedRotary, LatentAttention
    scale = (128 + rot) ** -0.5
    position = InterleavedRotary(rot, 10000.0, rot) if rot else None
    if q_rank is None:
        m = ZK.latent(heads, 128, rot, 128, rank, scale, 10000.0, rot, window)
        w = latent_weights(W, m, seed=3)
        plain = lambda x, st: PK.latent_attention(x, st, "x.", m, EPS)
    else:
        m = ZF.lat(heads, 128, rot, 128, q_rank, rank, scale, None, (10000.0, rot, None) if rot else None)["mixer"]
        w = lat_weights(W, m, seed=3)
        plain = lambda x, st: PF.latent_attention(x, st, "x.", m, EPS)
    part = LatentAttention(W, heads, 128, rot, 128, rank, scale, position, window=window, eps=EPS,
                           gate="head" if q_rank is None else "full", q_rank=q_rank)
    # keys, queries and values of some size: weights a tenth of the tiny models'
    w = {k: v if k.endswith("norm") else v * 0.4 for k, v in w.items()}
    return part, w, plain


def steps(part, w, plan, src, spoil=None):
    """Run `plan` (a list of steps {request: rows}) in bfloat16; -> each request's outputs, steps that ran expanded, backend."""
    bind(part, w, "bfloat16", "x.")
    hs = Harness("bfloat16", [part.cache_spec()], page_size=16, pages=160, slots=len(src))
    real, expanded = hs.backend.latent_attention_expanded, []
    hs.backend.latent_attention_expanded = lambda *a, **k: (expanded.append(True), real(*a, **k))[1]
    at, got = {k: 0 for k in src}, {k: [] for k in src}
    for st in plan:
        rows = torch.cat([src[k][at[k]: at[k] + n] for k, n in st.items()])
        y = hs.run(list(st.items()), lambda ctx, cache: part.forward(rows, ctx, cache))
        o = 0
        for k, n in st.items():
            got[k].append(y[o: o + n]); o += n; at[k] += n
        hs.engine.check()
    return {k: torch.cat(v) for k, v in got.items()}, len(expanded), hs


PLAN = [{"a": ROWS}, {"b": 40, "a": 1, "c": ROWS}, {"a": 2, "b": ROWS, "c": 1}, {"a": 1, "b": 1, "c": 1}]


@pytest.mark.parametrize("heads,rot,rank,window,q_rank,fits", [
    (8, 64, 64, None, None, True),       # 8 * 192 + 64 + 64 + 8 columns: rows start on 16 bytes
    (12, 64, 64, None, None, False),     # ... + 12 columns: they do not
    (8, 64, 128, 70, None, True),
    (3, 64, 128, None, None, False),
    (3, 64, 64, None, 104, True),
    (3, 64, 64, None, 100, False),       # the gate begins at column 100 + 64 + 64
    (2, 0, 64, None, 48, True),
])
def test_long_portions_beside_others(heads, rot, rank, window, q_rank, fits):
    part, w, plain = built(heads, rot, rank, window, q_rank)
    src = {k: rnd(sum(st.get(k, 0) for st in PLAN), W, seed=i).bfloat16() for i, k in enumerate("abc")}
    got, expanded, _ = steps(part, w, PLAN, {k: x.to(DEV) for k, x in src.items()})
    assert expanded == (3 if fits else 0)
    for k, x in src.items():
        # projections, latents, weights and outputs rounded to bfloat16, as the part's other bfloat16 tests have it
        assert rel(got[k], plain(x.double(), as_stored(w, "bfloat16"))) < 4e-2, k


@pytest.mark.parametrize("order", ["ab", "ba"])
@pytest.mark.parametrize("rot", [0, 64])
def test_a_request_beside_one_that_is_not_finite(order, rot):
    """Sequences lie one after the other in the expanded rows: a tile's rows beyond its own sequence are the next one's."""
    part, w, _ = built(8, rot, 64)
    src = {k: rnd(ROWS, W, seed=i).bfloat16().to(DEV) for i, k in enumerate("ab")}
    plan = [{k: ROWS for k in order}]
    want, expanded, _ = steps(part, w, plan, src)
    src["b"][:20] = float("inf")
    got, _, _ = steps(part, w, plan, src)
    assert expanded == 1 and not bool(got["b"].isfinite().any())
    assert bool(want["a"].isfinite().all()) and torch.equal(got["a"], want["a"])


def test_single_tokens_beside_a_long_portion():
    """The short portions' part is sized by their rows: against the same step with every row over the latents, and its memory."""
    part, w, _ = built(8, 64, 512)
    order = "abcdefghp"
    src = {k: rnd(3000 if k == "p" else 21 + 7 * i, W, seed=i).bfloat16().to(DEV) for i, k in enumerate(order)}
    first = {k: 1100 if k == "p" else len(src[k]) - 1 for k in order}
    bind(part, w, "bfloat16", "x.")
    got = []
    for expanded in (True, False):
        hs = Harness("bfloat16", [part.cache_spec()], page_size=16, pages=240, slots=9)
        if not expanded:
            hs.backend.latent_expanded = lambda *a: None
        run = lambda step, rows: hs.run(list(step.items()), lambda ctx, cache: part.forward(rows, ctx, cache))
        run(first, torch.cat([src[k][: first[k]] for k in order]))
        rows = torch.cat([src[k][first[k]:] for k in order])
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        got.append(run({k: len(src[k]) - first[k] for k in order}, rows))
        if expanded:
            assert torch.cuda.max_memory_allocated() - before < 200 << 20
        hs.engine.check()
    assert rel(got[0], got[1]) < 2e-2 and bool(got[0].isfinite().all())


def test_no_room_for_the_forms_that_take_scratch():
    """An engine whose memory does not hold the expansion or the chunks: the step runs in the forms without them."""
    from rllm_b200.kernels import hybrid
    part, w, plain = built(8, 64, 64)
    src = {k: rnd(ROWS + 1, W, seed=i).bfloat16() for i, k in enumerate("ab")}
    bind(part, w, "bfloat16", "x.")
    hs = Harness("bfloat16", [part.cache_spec()], page_size=16, pages=60, slots=2)
    hs.backend._no_room = 0
    rows = torch.cat([src["a"], src["b"]]).to(DEV)
    got = hs.run([("a", ROWS + 1), ("b", ROWS + 1)], lambda ctx, cache: part.forward(rows, ctx, cache)).split(ROWS + 1)
    for y, x in zip(got, src.values()):
        assert rel(y, plain(x.double(), as_stored(w, "bfloat16"))) < 4e-2

    def scan(ctx, cache):
        T, H, d = 300, 2, 64
        x = [rnd(T, H * d, seed=i).to(DEV) for i in range(4)]
        state = [torch.zeros(2, H, d, d, device=DEV) for _ in range(2)]
        a = hs.backend.state_scan(x[0], H, x[1], H, x[2], torch.sigmoid(x[3]), H, d, d, ctx, state[0])
        return torch.equal(a, hybrid.state_scan(x[0], H, x[1], H, x[2], torch.sigmoid(x[3]), H, d, d, ctx.cu_q, 1, ctx.state_slots,
                                                state[1])) and torch.equal(*state)
    hs.engine.end(["a", "b"])
    assert hs.run([("c", 300)], scan)


@pytest.mark.parametrize("dtype,heads,vdim,kept", [("bfloat16", 4, 128, True), ("bfloat16", 4, 64, False), ("float32", 4, 128, False)])
def test_weights_are_kept_once(dtype, heads, vdim, kept):
    """Keys' and values' weights under each other are the weights themselves, and are not made where nothing reads them."""
    from rllm_b200.parts import InterleavedRotary, LatentAttention
    m = ZK.latent(heads, 128, 64, vdim, 64, 0.1, 10000.0, 64, None)
    part = LatentAttention(W, heads, 128, 64, vdim, 64, 0.1, InterleavedRotary(64, 10000.0, 64))
    w = latent_weights(W, m, seed=3)
    bind(part, w, dtype, "x.")
    assert (part._ukv is not None) == kept
    for got, name in ((part.w_uk, "x.uk"), (part.w_uv, "x.uv")):
        assert torch.equal(got.cpu(), w[name].to(DT[dtype])) and got.is_contiguous()
        assert not kept or got.untyped_storage().data_ptr() == part._ukv.untyped_storage().data_ptr()
    assert part._uv.data_ptr() == part.w_uv.data_ptr()
