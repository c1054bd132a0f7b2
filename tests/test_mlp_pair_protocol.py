"""The barrier protocol of the MLP kernel on CTA pairs (surrogate.cuh), checked over every interleaving of its roles on the
CPU: the scheduler thread, the thread that issues the MMAs, and in each CTA the epilogue warps that also store input rows
and those that do not. How many arrivals complete the input rows' barrier, which warps arrive on it and whether the arrival
is a release are taken from the kernel's source; a state is each role's place in its program plus the barriers' phases and
what was released into them, and a wait passes when the phase of its parity is complete, as the hardware's does.

What has to hold whatever the order: every role sees every tile's index, once and in turn, the first layer's MMA runs after
both CTAs' rows have been released to its issuer, and no role waits for good."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sirius_b200", "csrc", "surrogate.cuh")


def kernel():
    with open(SOURCE) as f:
        text = f.read()
    epi = int(re.search(r"kEpiWarps = (\d+)", text).group(1))
    count = eval(re.search(r"mbar_init\(bar\(kBarX\), ([^;]*)\);", text).group(1), {"kEpiWarps": epi})
    body = re.search(r"auto store_row = \[&\]\(\) \{(.*?)\n        \};", text, re.S).group(1)
    row_warps = 128 * 2 // 32  # two threads a row, 128 rows a CTA
    # warps without rows leave before the arrival, or go on to it
    leave = re.search(r"return;", body)
    all_arrive = not (leave and leave.start() < body.index("mbar_arrive"))
    # a warp's rows: every lane's stores, the warp's barrier, then one lane's arrival, which has to be a release
    store, sync = body.index("kSmX"), body.index("__syncwarp()")
    release = store < sync < body.index("mbar_arrive") and "mbar_arrive_cluster(bar_x)" in body
    with open(os.path.join(os.path.dirname(SOURCE), "tcgen05.cuh")) as f:
        arrive = re.search(r"void mbar_arrive_cluster\(.*?\}", f.read(), re.S).group(0)
    return {"epi": epi, "rows": row_warps, "count": count, "all": all_arrive,
            "release": release and ".release.cluster." in arrive}


def programs(k, tiles):
    """Each role as a list of steps: ("wait", barrier, parity), ("arrive", barrier, n), ("write", cta, index),
    ("read", cta, expected index), ("rows", cta, n) for an arrival that hands rows over, ("use", None, tile) for the MMA
    on them."""
    ctl = []
    for t in range(tiles + 1):
        for r in (0, 1):
            ctl += [("write", r, t), ("arrive", "tile%d" % r, 1)]
        if t < tiles:
            ctl.append(("wait", "first", t & 1))
    mma, ph_a, ph_out = [], 0, 0
    for t in range(tiles):
        mma += [("wait", "tile0", t & 1), ("read", 0, t), ("wait", "x", t & 1), ("use", None, t), ("arrive", "d0", 1),
                ("arrive", "d1", 1), ("arrive", "first", 1)]
        for layer in range(4):
            mma.append(("wait", "a", ph_a))
            ph_a ^= 1
            mma += [("arrive", b + r, 1) for r in "01" for b in (("d",) if layer < 3 else ("out",))]
        mma.append(("wait", "out0", ph_out))
        ph_out ^= 1
    mma += [("wait", "tile0", tiles & 1), ("read", 0, tiles)]
    roles = {"scheduler": ctl, "issuer": mma}
    for r in (0, 1):
        for name, warps, arrives in (("rows", k["rows"], True), ("others", k["epi"] - k["rows"], k["all"])):
            p, ph_d = [("wait", "tile%d" % r, 0), ("read", r, 0)], 0
            x = [("rows" if name == "rows" else "arrive", r if name == "rows" else "x", warps)] if arrives else []
            p += x
            for t in range(tiles):
                for layer in range(4):
                    p += [("wait", "d%d" % r, ph_d), ("arrive", "a", warps)]
                    ph_d ^= 1
                    if layer == 1:
                        p += [("wait", "tile%d" % r, (t + 1) & 1), ("read", r, t + 1)]
                    if layer == 2 and t + 1 < tiles:
                        p += x
                p.append(("wait", "out%d" % r, t & 1))
            roles["%s%d" % (name, r)] = p
    return roles


def explore(k, tiles):
    """Every reachable state, depth first; what went wrong, or None."""
    roles = programs(k, tiles)
    names = list(roles)
    bars = ["tile0", "tile1", "first", "x", "a", "d0", "d1", "out0", "out1"]
    need = {b: 1 for b in bars}
    need["x"], need["a"] = k["count"], 2 * k["epi"]
    # (places, barriers, told index per CTA, tiles of rows released into x per CTA, of those the issuer knows)
    start = (tuple(0 for _ in names), tuple((0, 0) for _ in bars), (-1, -1), (0, 0), (0, 0))
    seen, stack = {start}, [start]
    while stack:
        at, bar, index, put, known = stack.pop()
        moved = False
        for i, n in enumerate(names):
            if at[i] == len(roles[n]):
                continue
            what, who, v = roles[n][at[i]]
            b2, i2, p2, k2 = bar, index, put, known
            if what == "rows":
                if k["release"]:
                    p2 = tuple(put[r] + (r == who) for r in (0, 1))
                what, who = "arrive", "x"
            if what == "wait":
                if (bar[bars.index(who)][0] & 1) == v:
                    continue  # the phase of this parity is not complete
                if who == "x":
                    k2 = put
            elif what == "arrive":
                j = bars.index(who)
                done, got = bar[j][0], bar[j][1] + v
                if got > need[who]:
                    return "%s: more arrivals on %s than it counts" % (n, who)
                if got == need[who]:
                    done, got = done + 1, 0
                b2 = bar[:j] + ((done, got),) + bar[j + 1:]
            elif what == "write":
                i2 = tuple(v if r == who else index[r] for r in (0, 1))
            elif what == "use":
                if known != (v + 1, v + 1):
                    return "the MMA of tile %d: rows of %s tiles were released to its issuer" % (v, known)
            elif index[who] != v:
                return "%s reads the index of tile %d for tile %d" % (n, index[who], v)
            moved = True
            s = (at[:i] + (at[i] + 1,) + at[i + 1:], b2, i2, p2, k2)
            if s not in seen:
                seen.add(s)
                stack.append(s)
        if not moved and any(at[i] < len(roles[n]) for i, n in enumerate(names)):
            return "stuck: " + ", ".join("%s at %s" % (n, roles[n][at[i]]) for i, n in enumerate(names) if at[i] < len(roles[n]))
    return None


@pytest.mark.parametrize("tiles", [1, 2, 3])
def test_every_role_sees_every_tile(tiles):
    assert explore(kernel(), tiles) is None


def test_a_warp_that_is_not_counted_in_can_miss_the_first_index():
    """The model itself: with the row warps alone on the rows' barrier, the others' first index can be overwritten."""
    assert explore({"epi": 16, "rows": 8, "count": 16, "all": False, "release": True}, 2) is not None
    assert explore({"epi": 16, "rows": 8, "count": 32, "all": True, "release": True}, 2) is None


def test_relaxed_arrivals_do_not_hand_rows_over():
    assert "released" in explore({"epi": 16, "rows": 8, "count": 32, "all": True, "release": False}, 1)
