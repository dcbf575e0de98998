"""The native writer of a step's metadata against the same vectors made number by number: portions and single tokens that end on and
beside page edges, new requests and grown ones, two cache groups of which one has given pages back behind its window."""
import numpy as np
import pytest
import torch


def manager(window, page, pages, reqs):
    from rllm_b200.cache import CacheManager
    from rllm_b200.parts.base import KVCacheSpec
    return CacheManager([KVCacheSpec(1, 16, None), KVCacheSpec(1, 16, window)], page, pages, reqs, torch.float32, "cpu", allocate=False)


def by_hand(m, lay, entries, rcs):
    ps, host = m.page_size, np.full(lay.total, -1, dtype=np.int32)
    q0 = r = 0
    lay.view(host, 3, lay.S + 1)[0] = 0
    for s, (e, rc) in enumerate(zip(entries, rcs)):
        for i, t in enumerate(e.tokens):
            p = rc.num_tokens + i
            for v, x in ((0, t), (1, p), (2, s)):
                lay.view(host, v, lay.T)[q0 + i] = x
            for g in range(lay.G):
                lay.view(host, 7 + 2 * g, lay.T)[q0 + i] = rc.pages[g][p // ps] * ps + p % ps
        for g in range(lay.G):
            held = rc.pages[g]
            lay.view(host, 8 + 2 * g, lay.S * lay.P)[s * lay.P: s * lay.P + len(held)] = held
        q0 += len(e.tokens)
        lay.view(host, 3, lay.S + 1)[s + 1] = q0
        lay.view(host, 4, lay.S)[s] = rc.num_tokens + len(e.tokens)
        lay.view(host, 5, lay.S)[s] = rc.state_slot
        for w in e.want:
            lay.view(host, 6, max(lay.n_rows, 1))[r] = q0 - len(e.tokens) + w
            r += 1
    if lay.n_rows == 0:
        lay.view(host, 6, 1)[0] = 0
    return host


@pytest.mark.parametrize("page", [1, 4, 16])
@pytest.mark.parametrize("lens", [[(0, 1)], [(0, 16), (5, 1), (0, 3)], [(15, 1), (16, 1), (17, 33), (0, 64)], [(40, 8), (0, 15), (63, 2), (1, 1)]])
def test_metadata_of_a_step(page, lens):
    from rllm_b200.engine.step import Engine, Entry, MetaLayout, StepError
    m = manager(8, page, 800, len(lens) + 1)
    eng = Engine.__new__(Engine)
    eng.cache = m
    entries, rcs = [], []
    for i, (have, q) in enumerate(lens):
        rc = m.open(i)
        for at in range(have):
            m.reserve(rc, at + 1)
            m.commit(rc, at + 1)
        m.reserve(rc, have + q)
        rcs.append(rc)
        entries.append(Entry(i, [(7 * i + 3 * k) % 50 for k in range(q)], [q - 1] if i % 2 else [0, q - 1][: q]))
    P = max(rc.num_held(g) for rc in rcs for g in range(2))
    for want in (True, False):
        if not want:
            entries = [Entry(e.request_id, e.tokens, []) for e in entries]
        lay = MetaLayout(sum(q for _, q in lens), len(lens), P, sum(len(e.want) for e in entries), 2)
        host = np.full(lay.total, -1, dtype=np.int32)
        eng.fill_meta(host, lay, entries, rcs)
        assert (host == by_hand(m, lay, entries, rcs)).all()
    with pytest.raises(StepError):                      # a token beyond the pages that are held
        more = [Entry(e.request_id, e.tokens + [1] * (page + 1), []) for e in entries]
        lay = MetaLayout(sum(len(e.tokens) for e in more), len(lens), P, 0, 2)
        eng.fill_meta(np.full(lay.total, -1, dtype=np.int32), lay, more, rcs)
