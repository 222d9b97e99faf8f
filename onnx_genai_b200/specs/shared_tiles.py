"""Model of the counters by which products with few rows sum the tiles that several CTAs share (csrc/kernels/gemm_rows.cuh, rows_epilogue).

The (tile, k-block) iterations are cut into one contiguous range per CTA.  A CTA does the tiles that it shares first: the one with the CTA before
it, then the one with the CTA after it, then its whole ones.  For a shared tile it leaves its partial sum in a slot of its own (one for a tile's
head, one for a later part), then arrives on the tile's counter, which belongs to the first CTA of the tile and wraps to zero with the last
arrival; whoever arrives last adds all partials and stores the tile.  Nobody waits, so residency does not matter.  What has to hold, whatever the
order: the last one finds every partial, every tile is stored once, and the next launch (a replayed graph) finds the counters at zero.

``broken="early"`` arrives before the partial is left (no fence between them), ``broken="sticky"`` lets the counters grow on: the checker finds a
tile summed without a partial, and a second launch that leaves a tile unstored.
"""
from __future__ import annotations

from ..utils.model_check import Result, explore


def check(ctas: int = 3, tiles: int = 4, k_blocks: int = 2, launches: int = 2, broken: str = "") -> Result:
    base, rem = divmod(tiles * k_blocks, ctas)
    bounds = [c * base + min(c, rem) for c in range(ctas + 1)]
    holders = {t: [c for c in range(ctas) if max(bounds[c], t * k_blocks) < min(bounds[c + 1], (t + 1) * k_blocks)] for t in range(tiles)}
    plans = []
    for c in range(ctas):
        mine = [t for t in range(tiles) if c in holders[t]]
        shared = [t for t in mine if len(holders[t]) > 1]
        assert len(shared) <= 2 and sum(holders[t][0] == c for t in shared) <= 1, "two slots, one counter per CTA"
        steps = []
        for t in shared:
            left, arrived = ("leave", t), ("arrive", t)
            steps += [arrived, left] if broken == "early" else [left, arrived]
        plans.append(tuple(steps + [("store", t) for t in mine if t not in shared]))
    # state: launch, per-CTA progress, partials left, counters, tiles stored in this launch, a tile that was summed without a partial
    init = (0, (0,) * ctas, frozenset(), (0,) * ctas, frozenset(), -1)

    def step(s):
        launch, prog, left, counters, stored, bad = s
        if launch < launches and all(prog[c] == len(plans[c]) for c in range(ctas)) and len(stored) == tiles:
            yield (f"launch{launch + 1}", (launch + 1, (0,) * ctas, frozenset(), counters, frozenset(), bad))
        if launch == launches:
            return
        for c in range(ctas):
            if prog[c] == len(plans[c]):
                continue
            what, t = plans[c][prog[c]]
            nprog, nleft, ncount, nstored, nbad = prog[:c] + (prog[c] + 1,) + prog[c + 1:], left, counters, stored, bad
            if what == "leave":
                nleft = left | {(c, t)}
            elif what == "store":
                nstored = stored | {t}
            else:
                own, want = holders[t][0], len(holders[t]) - 1
                last = counters[own] == want
                ncount = counters[:own] + (0 if last and broken != "sticky" else counters[own] + 1,) + counters[own + 1:]
                if last:
                    nstored = stored | {t}
                    if not all((x, t) in left for x in holders[t]):
                        nbad = t
            yield (f"cta{c}.{what}{t}", (launch, nprog, nleft, ncount, nstored, nbad))

    return explore(init, step, {"every partial is there": lambda s: s[5] < 0}, lambda s: s[0] == launches and not any(s[3]))
