"""Long portions of attention over latents (expanded keys and values) and of attention with mixed heads on the tcgen05 kernel of
prompt portions, beside short ones, against the formulas in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def batch(lens, page, width, seed):
    """cu_q, kv_lens, token_seq, positions and a block table over pages in mixed order for [(rows, keys)]."""
    S, pages = len(lens), [(n + page - 1) // page for _, n in lens]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    table, at, cu = torch.full((S, max(pages)), -1, dtype=torch.int32), 0, [0]
    for s, n in enumerate(pages):
        table[s, :n] = torch.tensor(order[at: at + n])
        at += n
        cu.append(cu[-1] + lens[s][0])
    pos = [p for q, n in lens for p in range(n - q, n)]
    seq = [s for s, (q, _) in enumerate(lens) for _ in range(q)]
    return cu, i32(cu), i32([n for _, n in lens]), i32(seq), i32(pos), table.to(DEV), len(order)


def visible(q, n, window, chunk=None):
    i, j = torch.arange(n - q, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    ok = j <= i
    if window:
        ok &= i - j < window
    if chunk:
        ok &= i // chunk == j // chunk
    return ok


# tiles of 128 rows and 64 keys: one row more and less, contexts longer than the portion, short portions left out in between
LENS = [((128, 128),), ((257, 300), (1, 90), (129, 129), (2, 200)), ((40, 45), (300, 771), (128, 640))]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("rot", [0, 64])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("gate", [None, "head", "full"])
def test_expanded_latents(lens, rot, window, gate):
    from rllm_b200.kernels import mix, sm100
    H, rank, page, long = 3, 64, 16, 128
    cu, cud, kvl, _, _, table, pages = batch(lens, page, rank + rot, 1)
    T = cu[-1]
    cache = rnd(pages, page, rank + rot, seed=2).bfloat16()
    q = rnd(T, H * (128 + rot) + 8, seed=3).bfloat16()
    qfull = rnd(T, H, rank + rot, seed=4).bfloat16()
    w = rnd(2 * H * 128, rank, seed=5, scale=rank ** -0.5).bfloat16()
    g = {None: None, "head": rnd(T, 8 + H, seed=6).bfloat16()[:, 8:], "full": rnd(T, 8 + H * 128, seed=6).bfloat16()[:, 8:]}[gate]
    rows, scale = sum(n for r, n in lens if r >= long), (128 + rot) ** -0.5
    c = mix.latent_gather(cache, table, cud, kvl, len(lens), long, rows, max(n for _, n in lens))
    want_c = torch.cat([cache[table[s, : (n + page - 1) // page].long()].reshape(-1, rank + rot)[:n] for s, (r, n) in enumerate(lens) if r >= long])
    assert torch.equal(c, want_c)
    kv = (c[:, :rank].float() @ w.float().T).bfloat16()
    out = torch.full((T, H * 128), 7.0, dtype=torch.bfloat16, device=DEV)
    sm100.attention_prefill_dense(q, 128 + rot, qfull[:, :, rank:] if rot else None, kv, 0, H * 128, c[:, rank:] if rot else None, cud, kvl,
                                  max(r for r, _ in lens), H, scale, window, out, long, g, gate == "full")
    sm100.check_error(torch.device(DEV))
    at = 0
    for s, (r, n) in enumerate(lens):
        mine = slice(cu[s], cu[s + 1])
        if r < long:
            assert bool((out[mine] == 7).all())
            continue
        k, v = kv[at: at + n].double().view(n, 2, H, 128).unbind(1)
        qq = q[mine, : H * (128 + rot)].double().view(r, H, 128 + rot)[..., :128]
        sc = torch.einsum("ihd,jhd->hij", qq, k)
        if rot:
            sc += torch.einsum("ihd,jd->hij", qfull[mine, :, rank:].double(), c[at: at + n, rank:].double())
        p = torch.softmax((sc * scale).masked_fill(~visible(r, n, window), float("-inf")), -1)
        o = torch.einsum("hij,jhd->ihd", p, v)
        if gate == "head":
            o = o * torch.sigmoid(g[mine, :H].double())[:, :, None]
        o = o.reshape(r, -1)
        if gate == "full":
            o = o * torch.sigmoid(g[mine].double())
        assert rel(out[mine], o) < 8e-3           # weights and outputs rounded to bfloat16: 2^-9 each
        at += n


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("hd,nh,nkv", [(128, 4, 2), (64, 6, 2), (64, 3, 3)])
@pytest.mark.parametrize("window,chunk", [(None, None), (100, None), (None, 96)])
def test_mixed_heads(lens, hd, nh, nkv, window, chunk):
    from rllm_b200.kernels import hybrid, sm100
    page, long = 16, 128
    cu, cud, kvl, seq, pos, table, pages = batch(lens, page, hd, 1)
    T = cu[-1]
    q = rnd(T, nh * hd + 8, seed=3).bfloat16()[:, : nh * hd]
    kc, vc = rnd(pages, nkv, page, hd, seed=4).bfloat16(), rnd(pages, nkv, page, hd, seed=5).bfloat16()
    mix, sinks, scale = rnd(nh, nh, seed=6), rnd(nh, seed=7), hd ** -0.5
    args = (q, kc, vc, seq, pos, table, cud, len(lens), max(r for r, _ in lens), nh, scale, mix, window, chunk, sinks)
    plain = hybrid.talk_attention_mma(*args)
    parts = torch.full((T, nh, nkv, hd), float("nan"), device=DEV)
    sm100.attention_prefill_tc(q, kc, vc, cud, kvl, table, max(r for r, _ in lens), nh, scale, window, chunk=chunk, sinks=sinks,
                               long_from=long, cross=parts)
    short = max((r for r, _ in lens if r < long), default=0)
    got = hybrid.talk_attention_mma(*args[:8], short, *args[9:], parts=parts, skip_from=long, any_short=short > 0)
    sm100.check_error(torch.device(DEV))
    for s, (r, n) in enumerate(lens):
        mine = slice(cu[s], cu[s + 1])
        k, v = (c[table[s, : (n + page - 1) // page].long()].transpose(1, 2).reshape(-1, nkv, hd)[:n].double()
                .repeat_interleave(nh // nkv, 1) for c in (kc, vc))
        sc = torch.einsum("ihd,jhd->hij", q[mine].double().view(r, nh, hd), k) * scale
        sc = sc.masked_fill(~visible(r, n, window, chunk), float("-inf"))
        p = torch.softmax(torch.cat([sc, sinks.double()[:, None, None].expand(nh, r, 1)], -1), -1)[..., :-1]
        o = torch.einsum("hij,jhd->ihd", torch.einsum("hg,gij->hij", mix.double(), p), v).reshape(r, -1)
        assert rel(got[mine], o) < 8e-3 and rel(got[mine], o) < 1.2 * rel(plain[mine], o) + 1e-4
        if r < long:
            # sixteen rows and fewer have a form of their own, whose sums are grouped otherwise
            assert torch.equal(got[mine], plain[mine]) or (short * (nh // nkv) <= 16 and rel(got[mine], plain[mine].double()) < 4e-3)


@pytest.mark.parametrize("lens", LENS[1:])
@pytest.mark.parametrize("splits", [1, 3])
def test_latents_beside_long_portions(lens, splits):
    """The rows of the short portions when the long ones are another kernel's, in both forms of the kernel."""
    from rllm_b200.kernels import mix
    H, rank, rot, page, long = 8, 128, 64, 16, 128
    cu, cud, kvl, seq, pos, table, pages = batch(lens, page, rank + rot, 1)
    cache, qfull = rnd(pages, page, rank + rot, seed=2).bfloat16(), rnd(cu[-1], H, rank + rot, seed=3).bfloat16()
    scale = (128 + rot) ** -0.5
    few = max(r for r, _ in lens if r < long) <= 2
    got = mix.latent_attention(qfull, cache, seq, pos, table, rank, scale, None, cu_q=cud, num_seqs=len(lens), splits=splits, few=few,
                               skip_from=long)
    for s, (r, n) in enumerate(lens):
        if r >= long:
            continue
        mine = slice(cu[s], cu[s + 1])
        c = cache[table[s, : (n + page - 1) // page].long()].reshape(-1, rank + rot)[:n].double()
        sc = torch.einsum("ihd,jd->hij", qfull[mine].double(), c) * scale
        p = torch.softmax(sc.masked_fill(~visible(r, n, None), float("-inf")), -1)
        assert rel(got[mine], torch.einsum("hij,jd->ihd", p, c[:, :rank])) < 8e-3


@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("hd,nh,nkv", [(128, 8, 2), (48, 3, 1)])
@pytest.mark.parametrize("window", [None, 70])
def test_mixed_heads_of_single_tokens_over_ranges_of_keys(splits, hd, nh, nkv, window):
    """Sequences shorter than a range, ranges that the window empties, one that ends at a tile's edge."""
    from rllm_b200.kernels import hybrid
    lens = [(1, 1), (1, 64), (2, 130), (1, 700)]
    cu, cud, _, seq, pos, table, pages = batch(lens, 16, hd, 1)
    q = rnd(cu[-1], nh * hd, seed=3).bfloat16()
    kc, vc = rnd(pages, nkv, 16, hd, seed=4).bfloat16(), rnd(pages, nkv, 16, hd, seed=5).bfloat16()
    args = (q, kc, vc, seq, pos, table, cud, len(lens), 2, nh, hd ** -0.5, rnd(nh, nh, seed=6), window, None, rnd(nh, seed=7))
    one, got = hybrid.talk_attention_mma(*args), hybrid.talk_attention_mma(*args, splits=splits)
    # the weights of a range are rounded to bfloat16 against its own maximum: 2^-9 each, as the one range's are
    assert rel(got, one.double()) < 6e-3


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("cross", [True, False])
@pytest.mark.parametrize("page", [16, 256])
def test_what_a_page_held_before(hd, cross, page):
    """Keys and values in a sequence's last page beyond its last token are none of its own, whatever is there."""
    from rllm_b200.kernels import sm100
    nh, nkv, lens = 4, 2, ((257, 300), (129, 129), (150, 641))
    cu, cud, kvl, _, _, table, pages = batch(lens, page, hd, 1)
    q = rnd(cu[-1], nh * hd, seed=3).bfloat16()
    kc, vc = rnd(pages, nkv, page, hd, seed=4).bfloat16(), rnd(pages, nkv, page, hd, seed=5).bfloat16()
    got = []
    for left in (0.0, float("inf"), float("nan")):
        for s, (_, n) in enumerate(lens):
            if n % page:
                last = int(table[s, n // page])
                kc[last, :, n % page:] = left
                vc[last, :, n % page:] = left
        kw = dict(cross=torch.empty((cu[-1], nh, nkv, hd), device=DEV)) if cross else {}
        got.append(sm100.attention_prefill_tc(q, kc, vc, cud, kvl, table, 257, nh, hd ** -0.5, None, **kw).clone())
    sm100.check_error(torch.device(DEV))
    assert bool(got[0].isfinite().all()) and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
