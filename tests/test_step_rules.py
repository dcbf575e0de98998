"""Which form of an operation a step takes, by the sizes of its portions alone: the rules that the backend asks on the host, at
sizes where both forms were measured."""
from types import SimpleNamespace

import pytest


def step(lens):
    """A step of [(rows, keys)], as the rules see it."""
    q, n = [r for r, _ in lens], [k for _, k in lens]
    return SimpleNamespace(graph_safe=False, q_lens_host=q, kv_lens_host=n, max_q_len=max(q), max_kv_len=max(n), num_seqs=len(lens),
                           num_tokens=sum(q), per_forward={})


@pytest.mark.parametrize("heads,rank,window,lens,expanded", [
    (16, 512, None, [(512, 512)], False),                       # us over the latents / expanded: 143 / 148
    (16, 512, None, [(2048, 2048)], True),                      # 689 / 149
    (16, 512, None, [(256, 2256)], True),                       # 270 / 148
    (64, 512, None, [(256, 256)], True),                        # 170 / 132
    (16, 64, None, [(512, 512)], False),                        # 112 / 120
    (16, 64, None, [(2048, 2048)], True),                       # 317 / 152
    (16, 512, 128, [(2048, 2048)], True),                       # 203 / 147
    (16, 512, 128, [(512, 512)], False),                        # 113 / 119
    (16, 512, None, [(1, 1001)] * 16 + [(512, 512)], False),    # 173 / 194
    (128, 512, None, [(1, 1001)] * 16 + [(512, 512)], True),    # 617 / 352
    (128, 512, None, [(1, 1001)] * 63 + [(256, 256)], False),   # 470 / 573
    (16, 512, None, [(1, 4001)] * 8 + [(2048, 4048)], True),    # 1,665 / 332
])
def test_latents_are_expanded_where_it_pays(monkeypatch, heads, rank, window, lens, expanded):
    from rllm_b200.kernels.backend import Backend
    monkeypatch.delenv("RLLM_B200_NO_TC_ATTENTION", raising=False)
    be = SimpleNamespace(fast=True, _sm100=SimpleNamespace(prefill_dense_supported=lambda *a: True))
    got = Backend.latent_expanded(be, step(lens), None, None, False, heads, 128, 64, 128, rank, window, 0.1)
    assert (got is not None) == expanded
    if expanded:
        short = [r for r, _ in lens if r < 32]
        assert got[1:] == (sum(n for r, n in lens if r >= 32), (sum(short), len(short)))


@pytest.mark.parametrize("heads,vdim,rows,walked,chunks", [
    (16, 128, [256], True, 4),                      # us row by row / in chunks: 107 / 56
    (64, 128, [256], True, 4),                      # 193 / 117
    (128, 128, [256], True, None),                  # 207 / 235
    (8, 128, [256] * 16, True, None),               # 207 / 238
    (16, 128, [256] * 4, True, 16),                 # 193 / 118
    (32, 64, [256] * 4, True, 16),                  # 175 / 100
    (16, 64, [256] * 16, True, None),               # 159 / 197
    (64, 128, [1] * 63 + [256], True, 4),           # 310 / 278
    (32, 128, [512] * 8, False, 64),                # against three passes: 1,403 / 601
    (16, 128, [255] * 4, True, None),
])
def test_recurrences_run_in_chunks_where_it_pays(heads, vdim, rows, walked, chunks):
    from rllm_b200.engine.context import StepContext
    got = StepContext.long_rows(step([(n, n) for n in rows]), heads, vdim, walked)
    assert got.get("chunks") == chunks
    if got:
        assert got["longs"] == sum(n >= 64 for n in rows) and got["any_short"] == (min(rows) < 64)


@pytest.mark.parametrize("hd,nh,nkv,lens,tcgen05", [
    (128, 16, 4, [(384, 384)], False),                          # us mma.sync / tcgen05: 39 / 41
    (128, 16, 4, [(512, 512)], True),                           # 56 / 40
    (128, 16, 4, [(128, 1200)], True),                          # 76 / 43
    (128, 16, 4, [(256, 256)] * 4, True),                       # 58 / 42
    (128, 16, 4, [(1, 800)] * 17 + [(512, 900)], True),         # 144 / 121
    (128, 4, 1, [(512, 512)], False),                           # 31 / 44
    (128, 4, 1, [(1024, 1024)], True),                          # 51 / 40
    (128, 4, 1, [(256, 256)] * 4, False),                       # 25 / 40
    (128, 4, 1, [(1, 800)] * 17 + [(512, 900)], False),         # 54 / 61
    (128, 32, 4, [(384, 384)], True),                           # 66 / 43
    (64, 16, 4, [(512, 512)], False),                           # 33 / 41
    (64, 16, 4, [(1024, 1024)], True),                          # 85 / 41
    (64, 16, 4, [(1, 800)] * 17 + [(512, 900)], False),         # 77 / 87
    (64, 64, 8, [(384, 384)], True),                            # 112 / 96
    (128, 16, 4, [(127, 4000)], False),
])
def test_mixed_heads_on_tcgen05_where_it_pays(hd, nh, nkv, lens, tcgen05):
    from rllm_b200.kernels.backend import talk_on_tcgen05
    assert talk_on_tcgen05(step(lens), nh, nkv, hd) == tcgen05


def test_scratch_that_did_not_fit_is_not_asked_for_again(monkeypatch):
    import torch
    from rllm_b200.kernels.backend import Backend
    asked = []

    def empty(n, **k):
        asked.append(n)
        if n > 100:
            raise torch.OutOfMemoryError("no")
        return n
    monkeypatch.setattr(torch, "empty", empty)
    be = SimpleNamespace(_no_room=1 << 62)
    be._or_none = lambda *a: Backend._or_none(be, *a)
    got = [Backend.scratch(be, n, "cpu") for n in (50, 400, 500, 400, 200, 300, 100, 200)]
    assert got == [50, None, None, None, None, None, 100, None] and asked == [50, 400, 200, 100]


def test_profile_counts_a_portion_once():
    """Rows over the latents, expansion and attention over what it made: every pair of query and key in one line."""
    import torch
    from rllm_b200.kernels import profile
    lens, window, heads, rank, rot = [(1, 500), (300, 700), (3, 40), (64, 64)], 100, 4, 64, 64
    for q, n in lens:
        for w in (None, 1, 30, 100, 500, 5000):
            assert profile._visible(q, n, w) == sum(min(p + 1, w or p + 1) for p in range(n - q, n))
    ctx, lines = step(lens), []
    prof = profile.OpProfile.__new__(profile.OpProfile)
    prof._be = SimpleNamespace(latent_attention=None, latent_attention_expanded=None, latent_expand=None)
    prof._timed = lambda cls, nbytes, flops, fn, *a, **k: lines.append((cls, nbytes, flops))
    bf = lambda *s: torch.empty(s, dtype=torch.bfloat16)
    pairs = {s: profile._visible(*lens[s], window) for s in range(4)}
    long, rows = (32, 764, (304, 3)), 764
    prof.latent_expand(SimpleNamespace(tensors={"kv": bf(9, 16, rank + rot)}), ctx, bf(heads * 256, rank), rank, long)
    prof.latent_attention(bf(304, heads, rank + rot), None, ctx, rank, 0.1, window, 32, 3)
    prof.latent_attention_expanded(None, None, (bf(rows, rank + rot), bf(rows, heads * 256)), ctx, heads, 128, rot, rank, 0.1, window, long)
    assert [f for _, _, f in lines] == [2 * rows * heads * 256 * rank, 2 * heads * (2 * rank + rot) * (pairs[0] + pairs[2]),
                                        2 * heads * (128 + rot + 128) * (pairs[1] + pairs[3])]
    assert lines[1][1] == 2 * ((100 + 40) * (rank + rot) + 4 * heads * (2 * rank + rot))
    assert lines[2][1] == 2 * (rows * (rank + rot + heads * 256) + 364 * heads * (128 + rot + 128))
