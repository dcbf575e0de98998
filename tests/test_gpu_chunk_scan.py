"""Recurrences in chunks of 64 rows as products of matrices (csrc/chunk_scan.cuh) against the recurrence itself in 64 bits,
token by token, beside the row-by-row kernels on the same inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ERR():
    from rllm_b200.kernels import sm100
    return sm100.init(torch.device(DEV)).err


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(DEV)


def decays(*shape, seed):
    """Mostly near one, some strong, some so strong that a few of them leave nothing."""
    g = torch.Generator().manual_seed(seed)
    x = torch.rand(*shape, generator=g)
    return torch.where(x < 0.85, 1 - 0.05 * x, torch.where(x < 0.97, x - 0.8, torch.where(x < 0.99, 1e-20, 0.0))).to(DEV)


def recurrence(q, k, v, a, S, beta=None, bonus=None):
    """One sequence in 64 bits: q, k, a [n, H, d] (a of 1 or d channels), v [n, H, dv], S [H, d, dv]."""
    S, out = S.clone(), []
    for t in range(q.shape[0]):
        before = S
        S = a[t][:, :, None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        kv = k[t][:, :, None] * u[:, None]
        S = S + kv
        out.append(torch.einsum("hkv,hk->hv", S if bonus is None else before + bonus[:, :, None] * kv, q[t]))
    return torch.stack(out), S


def layout(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu, torch.tensor(cu, dtype=torch.int32, device=DEV)


# lengths at the edges of blocks of 16 and chunks of 64, beside rows that stay with the other kernel
LENS = [(64,), (65, 1, 130), (127, 3, 64, 81), (512, 66)]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,vdim,H,G", [(128, 128, 4, 2), (64, 48, 6, 3), (128, 64, 8, 2), (128, 16, 40, 40)])
@pytest.mark.parametrize("channel", [True, False])
@pytest.mark.parametrize("delta", [True, False])
def test_state_scan_in_chunks(lens, dim, vdim, H, G, channel, delta):
    from rllm_b200.kernels import hybrid
    cu, cud = layout(lens)
    T, S = cu[-1], len(lens)
    q = torch.nn.functional.normalize(rnd(T, G, dim, seed=1), dim=-1)
    k = torch.nn.functional.normalize(rnd(T, G, dim, seed=2), dim=-1)
    v = rnd(T, H * vdim, seed=3)
    a = decays(T, H, dim if channel else 1, seed=4)
    beta = rnd(T, H + 3, seed=5)[:, :H] if delta else None
    vs, skip = (None, None) if delta else (rnd(T, H, seed=6), rnd(H, seed=7))
    slots = torch.tensor([-1 if s == 1 else S - s for s in range(S)], dtype=torch.int32, device=DEV)
    state = rnd(S + 1, H, dim, vdim, seed=8)
    got = {}
    for name, long in (("chunks", dict(long_from=64, any_short=min(lens) < 64, err=ERR())), ("rows", {})):
        st = state.clone()
        o = hybrid.state_scan(q.view(T, -1), G, k.view(T, -1), G, v, a.view(T, -1), H, dim, vdim, cud, S, slots, st, beta=beta,
                              vscale=vs, skip=skip, **long)
        got[name] = (o, st)
    d = lambda x: x.double()
    which = torch.arange(H, device=DEV) // (H // G)
    keep = state.double()
    want = []
    for s, n in enumerate(lens):
        r, sl = slice(cu[s], cu[s + 1]), int(slots[s])
        u = d(v[r]).view(n, H, vdim)
        o, end = recurrence(d(q[r])[:, which], d(k[r])[:, which], u if delta else u * d(vs[r])[:, :, None], d(a[r]),
                            keep[sl] if sl >= 0 else torch.zeros_like(keep[0]), torch.sigmoid(d(beta[r])) if delta else None)
        want.append(o if delta else o + d(skip)[:, None] * u)
        if sl >= 0:
            keep[sl] = end
    want = torch.cat(want)
    e = {name: (rel(o, want), rel(st, keep)) for name, (o, st) in got.items()}
    # sums of up to 128 + 64 products in float: some 5e-7 either way
    assert e["chunks"][0] < 2e-6 and e["chunks"][1] < 2e-6, e
    assert torch.equal(got["chunks"][1][0], state[0])                      # a slot of nobody's
    if min(lens) < 64:
        s = min(range(S), key=lambda i: lens[i])
        assert torch.equal(got["chunks"][0][cu[s]: cu[s + 1]], got["rows"][0][cu[s]: cu[s + 1]])


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,vdim,H", [(128, 128, 3), (64, 80, 5), (64, 16, 160)])
@pytest.mark.parametrize("bonus", [True, False])
def test_gated_linear_attention_in_chunks(lens, dim, vdim, H, bonus):
    from rllm_b200.kernels import mix
    cu, cud = layout(lens)
    T, S = cu[-1], len(lens)
    proj = rnd(T, 8 + H * (2 * dim + vdim), seed=1).bfloat16()
    a, u = decays(T, H * dim, seed=2), rnd(H, dim, seed=3) if bonus else None
    slots = torch.tensor([-1 if s == 1 else S - s for s in range(S)], dtype=torch.int32, device=DEV)
    state = rnd(S + 1, H, dim, vdim, seed=4)
    got = {}
    for name, long in (("chunks", dict(long_from=64, any_short=min(lens) < 64, err=ERR())), ("rows", {})):
        st = state.clone()
        o = mix.gla_scan(proj, 8, 8 + H * dim, 8 + 2 * H * dim, a, dim ** -0.5, H, dim, vdim, cud, S, slots, st, bonus=u, **long)
        got[name] = (o, st)
    p, keep, want = proj.double(), state.double(), []
    for s, n in enumerate(lens):
        r, sl = slice(cu[s], cu[s + 1]), int(slots[s])
        q, k = (p[r, 8 + i * H * dim: 8 + (i + 1) * H * dim].view(n, H, dim) for i in (0, 1))
        o, end = recurrence(q * dim ** -0.5, k, p[r, 8 + 2 * H * dim:].view(n, H, vdim), a[r].double().view(n, H, dim),
                            keep[sl] if sl >= 0 else torch.zeros_like(keep[0]), bonus=u.double() if bonus else None)
        want.append(o)
        if sl >= 0:
            keep[sl] = end
    want = torch.cat(want)
    e = {name: (rel(o, want), rel(st, keep)) for name, (o, st) in got.items()}
    assert e["chunks"][0] < 2e-6 and e["chunks"][1] < 2e-6, e
    assert torch.equal(got["chunks"][1][0], state[0])
    if min(lens) < 64:
        s = min(range(S), key=lambda i: lens[i])
        assert torch.equal(got["chunks"][0][cu[s]: cu[s + 1]], got["rows"][0][cu[s]: cu[s + 1]])


@pytest.mark.parametrize("what", ["q", "k", "v", "decay", "beta"])
@pytest.mark.parametrize("kind", ["channel", "head", "gla"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_token_that_is_not_finite(what, kind, bad):
    """What a token brings is felt from it on, or (a query) by it alone: the tokens before it in its chunk are as they were."""
    from rllm_b200.kernels import hybrid, mix
    if what == "beta" and kind == "gla":
        pytest.skip("gated linear attention has none")
    H, dim, vdim, at = 2, 64, 64, 64 + 37
    cu, cud = layout((150, 70))
    T, slots = cu[-1], torch.arange(2, dtype=torch.int32, device=DEV)
    x = {"q": rnd(T, H * dim, seed=1), "k": torch.nn.functional.normalize(rnd(T, H, dim, seed=2), dim=-1).view(T, -1),
         "v": rnd(T, H * vdim, seed=3), "decay": decays(T, H * (1 if kind == "head" else dim), seed=4), "beta": rnd(T, H, seed=5)}

    def scan():
        state = torch.zeros(2, H, dim, vdim, device=DEV)
        if kind == "gla":
            proj = torch.cat([x["q"], x["k"], x["v"]], 1).bfloat16()
            return mix.gla_scan(proj, 0, H * dim, 2 * H * dim, x["decay"], 1.0, H, dim, vdim, cud, 2, slots, state, long_from=64,
                                any_short=False, err=ERR())
        return hybrid.state_scan(x["q"], H, x["k"], H, x["v"], x["decay"], H, dim, vdim, cud, 2, slots, state, beta=x["beta"],
                                 long_from=64, any_short=False, err=ERR())
    want = scan()
    x[what][at] = bad
    got = scan()
    mine = slice(at, at + 1) if what == "q" else slice(at, 150)
    if what != "beta" or bad != bad:                     # the sigmoid of an infinity is one
        assert not bool(got[mine].isfinite().all())
    same = torch.ones(T, dtype=torch.bool, device=DEV)
    same[mine] = False
    assert bool(want.isfinite().all()) and torch.equal(got[same], want[same])


def test_the_step_says_how_many_chunks_there_are():
    """Grids and scratch of the long sequences alone, in any order among short ones: the same bits as with the bounds."""
    from types import SimpleNamespace
    from rllm_b200.engine.context import StepContext
    from rllm_b200.kernels import hybrid, mix
    lens, H, dim = (1, 300, 63, 64, 1, 65) + (1,) * 40, 2, 64
    cu, cud = layout(lens)
    T, S = cu[-1], len(lens)
    long = StepContext.long_rows(SimpleNamespace(graph_safe=False, max_q_len=300, q_lens_host=list(lens), num_seqs=S), H, dim)
    assert long == dict(long_from=64, any_short=True, longs=3, chunks=5 + 1 + 2)
    q, k, v = rnd(T, H * dim, seed=1), torch.nn.functional.normalize(rnd(T, H, dim, seed=2), dim=-1).view(T, -1), rnd(T, H * dim, seed=3)
    a, beta, slots = decays(T, H * dim, seed=4), rnd(T, H, seed=5), torch.arange(S, dtype=torch.int32, device=DEV)
    got = []
    for kw in (dict(long_from=64, any_short=True), long):
        state = [rnd(S, H, dim, dim, seed=6) for _ in range(2)]
        got.append((hybrid.state_scan(q, H, k, H, v, a, H, dim, dim, cud, S, slots, state[0], beta=beta, err=ERR(), **kw),
                    mix.gla_scan(torch.cat([q, k, v], 1).bfloat16(), 0, H * dim, 2 * H * dim, a, 1.0, H, dim, dim, cud, S, slots,
                                 state[1], err=ERR(), **kw), *state))
    assert all(torch.equal(x, y) for x, y in zip(*got)) and all(bool(x.isfinite().all()) for x in got[0])


@pytest.mark.parametrize("pad,off", [(2, 0), (0, 2), (4, 0)])
def test_rows_that_the_chunks_cannot_read(pad, off):
    """A projection whose rows, or their parts, do not start on four numbers keeps the passes over chunks that it had."""
    from rllm_b200.kernels import mix
    H, dim, T = 2, 64, 400
    cu, cud = layout((T,))
    proj = rnd(T, off + H * 3 * dim + pad, seed=1).bfloat16()
    a = torch.exp(-0.01 * rnd(T, H * dim, seed=2).abs())          # slow, so that how the sums are grouped shows
    args = (proj, off, off + H * dim, off + 2 * H * dim, a, 1.0, H, dim, dim, cud, 1, torch.zeros(1, dtype=torch.int32, device=DEV))
    state = [rnd(1, H, dim, dim, seed=3) for _ in range(3)]
    passes = mix.gla_scan(*args, state[0], 128)
    got = mix.gla_scan(*args, state[1], 128, long_from=64, any_short=False, err=ERR())
    rows = mix.gla_scan(*args, state[2])
    same = (torch.equal(got, passes), torch.equal(got, rows))
    assert same == ((False, False) if pad % 4 == off % 4 == 0 else (True, False)) and torch.equal(state[0], state[1]) == same[0]
    assert rel(got, rows.double()) < 2e-6


@pytest.mark.parametrize("kind", ["channel", "head", "plain", "gla"])
@pytest.mark.parametrize("slow", [True, False])
def test_no_further_from_64_bits_than_row_by_row(kind, slow):
    """Roundings at random add up like the root of the links of a chain; both forms' chains have some 16 to 20 links."""
    from rllm_b200.kernels import hybrid, mix
    H, dim, T = 4, 128, 1024
    cu, cud = layout((T,))
    slots = torch.zeros(1, dtype=torch.int32, device=DEV)
    unit = lambda seed: torch.nn.functional.normalize(rnd(T, H, dim, seed=seed), dim=-1)
    q, k, v = (x.view(T, H * dim) for x in (unit(1), unit(2), rnd(T, H, dim, seed=3)))
    u = torch.rand(T, H, dim if kind in ("channel", "gla") else 1, generator=torch.Generator().manual_seed(4)).to(DEV)
    a = torch.exp(-0.01 * u) if slow else u
    beta = rnd(T, H, seed=5) if kind in ("channel", "head") else None
    if kind == "gla":
        proj = torch.cat([q, k, v], 1).bfloat16()
        q, k, v = (x.contiguous() for x in proj.float().split(H * dim, 1))
        run = lambda kw: mix.gla_scan(proj, 0, H * dim, 2 * H * dim, a.view(T, -1), 1.0, H, dim, dim, cud, 1, slots,
                                      torch.zeros(1, H, dim, dim, device=DEV), **kw)
    else:
        run = lambda kw: hybrid.state_scan(q, H, k, H, v, a.view(T, -1), H, dim, dim, cud, 1, slots,
                                           torch.zeros(1, H, dim, dim, device=DEV), beta=beta, **kw)
    d = lambda x: x.double().view(T, H, -1)
    want, _ = recurrence(d(q), d(k), d(v), a.double(), torch.zeros(H, dim, dim, dtype=torch.float64, device=DEV),
                         torch.sigmoid(beta.double()) if beta is not None else None)
    rows, chunks = rel(run({}), want), rel(run(dict(long_from=64, any_short=False, err=ERR())), want)
    assert chunks < 1.2 * rows, (chunks, rows)
