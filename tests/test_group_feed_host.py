"""The block-wise tile order of the D3Q27 AB steps (lbmminiapp_gb300/csrc/
lbm_step_async.cuh), modelled on the CPU: a block's warps take the tiles of a group
together, three groups in a fixed order and then one counter, which the block's
first thread asks one group ahead, the number handed over in one of two slots with
a barrier between.  Blocks and the warps between two barriers are interleaved at
random.  Every tile is processed exactly once, every warp of a block sees the same
groups, and the counters are zero again after the launch."""
import random

import pytest

FEED_MIN_TILES = 16


def launch(ntiles, nblocks, warps, seed):
    rng = random.Random(seed)
    nw = nblocks * warps
    ngroups = -(-ntiles // warps)
    fed = ntiles >= FEED_MIN_TILES * nw
    state = {"counter": 0, "done": 0}
    got = []
    blocks = [{"slots": [None, None], "waiting": 0, "phase": 0, "groups": [[] for _ in range(warps)], "arrived": 0}
              for _ in range(nblocks)]

    def barrier(b):
        """One thread's arrival; yields until every warp has arrived."""
        B = blocks[b]
        phase = B["phase"]
        B["waiting"] += 1
        if B["waiting"] == warps:
            B["waiting"] = 0
            B["phase"] += 1
        while B["phase"] == phase:
            yield

    def warp(b, w):
        B = blocks[b]
        pend = 0
        if fed and w == 0:
            pend = state["counter"]
            state["counter"] += 1
        yield

        def tile(g):
            t = g * warps + w
            return t if g < ngroups and t < ntiles else ntiles

        def clip(g):
            return g if g < ngroups else ngroups

        g, it = b, 0
        if g < ngroups:
            g1, g2 = clip(g + nblocks), clip(g + 2 * nblocks)
            t, t1 = tile(g), tile(g1)
            t2 = tile(g2)
            while True:
                B["groups"][w].append(g)
                if t < ntiles:
                    got.append(t)
                yield
                if g1 >= ngroups:
                    break
                g, g1 = g1, g2
                if g2 < ngroups:
                    if fed:
                        if w == 0:
                            n = 3 * nblocks + pend
                            B["slots"][it & 1] = n if n < ngroups else ngroups
                            if n < ngroups:
                                pend = state["counter"]
                                state["counter"] += 1
                        yield from barrier(b)
                        yield
                        g2 = B["slots"][it & 1]
                    else:
                        g2 = clip(g2 + nblocks)
                        yield from barrier(b)
                it += 1
                t, t1, t2 = t1, t2, tile(g2)
        if fed:
            yield from barrier(b)
            if w == 0:
                state["done"] += 1
                if state["done"] == nblocks:
                    state["counter"] = state["done"] = 0
        yield

    gens = [warp(b, w) for b in range(nblocks) for w in range(warps)]
    live = list(range(len(gens)))
    while live:
        i = rng.choice(live)
        try:
            next(gens[i])
        except StopIteration:
            live.remove(i)
    assert sorted(got) == list(range(ntiles))
    for B in blocks:
        assert all(seen == B["groups"][0] for seen in B["groups"])
    assert state == {"counter": 0, "done": 0}
    return fed


@pytest.mark.parametrize("nblocks,warps", [(1, 4), (3, 4), (5, 2), (4, 1)])
def test_every_tile_once_and_counters_rearmed(nblocks, warps):
    fed = set()
    nw = nblocks * warps
    for ntiles in (1, warps, warps + 1, nw - 1, nw, 3 * nw - 1, 3 * nw + 1, FEED_MIN_TILES * nw - 1,
                   FEED_MIN_TILES * nw, FEED_MIN_TILES * nw + 1, FEED_MIN_TILES * nw + warps + 1, 40 * nw + 3):
        for seed in range(3):
            if ntiles >= 1:
                fed.add(launch(ntiles, nblocks, warps, seed))
    assert fed == {True, False}
