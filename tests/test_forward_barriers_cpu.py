"""The hand-over between a query tile's softmax warps and its issuer in the forward kernels (rbf_fwd.cu), every schedule of it:
an mbarrier wait names a phase by its parity, so whoever waits for phase k has to look before phase k + 1 completes and not
before phase k - 1 has. One warp that is late by a few hundred clocks - a first instruction fetch, a time slice - would
otherwise stand at the barrier until the wait runs out, or go on with another tile's result."""

import pytest

WARPS = 2          # of a tile: two are enough for one to be late


def overlapping_items(tiles):
    """Head dim 64: a CTA's items one after the other; s = scores and all but the item's last product, p = P stored and scores
    read, o = the item's last product."""
    warp, issuer = [], []
    s = p = 0
    for item, n in enumerate(tiles):
        issuer.append(("commit", "s"))
        warp += [("wait", "s", s), ("arrive", "p")]
        for j in range(n):
            warp += [("wait", "s", s + 1 + j), ("arrive", "p")]
        warp.append(("wait", "o", item))
        for j in range(n + 1):
            issuer += [("wait", "p", p + j), ("commit", "s" if j < n else "o")]
        s, p = s + n + 1, p + n + 1
    return [warp] * WARPS + [issuer]


def one_item(n, rescale):
    """Head dim 128: s = scores, c = scores read, p / o = P stored / its product complete, even and odd tiles apart."""
    warp, issuer = [], [("commit", "s")]
    for j in range(n):
        warp += [("wait", "s", j), ("arrive", "c")]
        if rescale and j > 0:
            warp.append(("wait", f"o{(j - 1) & 1}", (j - 1) >> 1))
        warp.append(("arrive", f"p{j & 1}"))
        if j + 1 < n:
            issuer += [("wait", "c", j), ("commit", "s")]
        issuer += [("wait", f"p{j & 1}", j >> 1), ("commit", f"o{j & 1}")]
    warp.append(("wait", f"o{(n - 1) & 1}", (n - 1) >> 1))
    return [warp] * WARPS + [issuer]


def search(actors):
    """Depth-first over all schedules. Commits complete in order, at any later time. Returns what goes wrong, or None."""
    commits = [op[1] for op in actors[-1] if op[0] == "commit"]
    arrivals = {op[1] for op in actors[0] if op[0] == "arrive"}
    start = ((0,) * len(actors), 0)
    seen, stack = {start}, [start]
    while stack:
        at, landed = stack.pop()
        issued = sum(op[0] == "commit" for op in actors[-1][:at[-1]])

        def arrived(bar):
            return [sum(op == ("arrive", bar) for op in a[:i]) for a, i in zip(actors[:-1], at[:-1])]

        def phase(bar):                         # phases completed so far
            return min(arrived(bar)) if bar in arrivals else commits[:landed].count(bar)

        for bar in arrivals:
            if max(arrived(bar)) > min(arrived(bar)) + 1:
                return f"a warp arrives at {bar} twice within a phase"
        moves = [(at, landed + 1)] if landed < issued else []
        for n, (actor, i) in enumerate(zip(actors, at)):
            if i == len(actor):
                continue
            if actor[i][0] == "wait":
                _, bar, k = actor[i]
                if not k <= phase(bar) <= k + 1:
                    return f"actor {n} waits for phase {k} of {bar}, {phase(bar)} phases are complete"
                if phase(bar) == k:
                    continue
            moves.append((at[:n] + (i + 1,) + at[n + 1:], landed))
        if not moves and any(i < len(a) for a, i in zip(actors, at)):
            return f"all stand still at {at}"
        for move in moves:
            if move not in seen:
                seen.add(move)
                stack.append(move)
    return None


@pytest.mark.parametrize("tiles", [(1,), (2,), (1, 1, 1), (3, 1, 2), (1, 3), (2, 2, 1)])
def test_no_phase_is_skipped_between_overlapping_items(tiles):
    assert search(overlapping_items(tiles)) is None


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("n", range(1, 8))
def test_no_phase_is_skipped_within_an_item(n, rescale):
    assert search(one_item(n, rescale)) is None


def test_the_search_finds_a_skipped_and_an_early_phase():
    # the item's last product on the scores' barrier: the next item's first scores complete the phase behind it
    def shared(ops):
        s, out = 0, []
        for op in ops:
            if op[:2] in (("wait", "s"), ("wait", "o")):
                out.append(("wait", "s", s))
                s += 1
            else:
                out.append(("commit", "s") if op == ("commit", "o") else op)
        return out
    assert "waits for phase" in search([shared(a) for a in overlapping_items((2, 1))])

    # one barrier for the products of all tiles, the last two waited for in turn, or the last one alone
    def single(actor, last_two):
        out = [op[:1] + ("o",) + op[2:] if op[1][0] == "o" else op for op in actor]
        if out[-1][0] == "wait":
            out[-1:] = [("wait", "o", 2), ("wait", "o", 3)] if last_two else [("wait", "o", 3)]
        return out
    *warps, issuer = one_item(4, False)
    for last_two in (True, False):
        assert "waits for phase" in search([single(w, last_two) for w in warps] + [single(issuer, last_two)])

    # one barrier for P of all tiles
    def joined(actor):
        seen, out = 0, []
        for op in actor:
            if op[1][0] == "p":
                op = ("wait", "p", seen) if op[0] == "wait" else ("arrive", "p")
                seen += 1
            out.append(op)
        return out
    assert search([joined(a) for a in one_item(4, False)]) is not None
