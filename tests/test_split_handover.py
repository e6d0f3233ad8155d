"""Hand-over of partial sums between the warps of a CTA and the ranks of a cluster (csrc/qmv_split.cuh): no buffer, no area of sums and no
description of a chunk is written again before every warp has read it.

The order of a warp's steps for one chunk is taken from the kernel's source, for each of its three forms: activations in f16, in integers, and in
integers once a warp's share has gone over to halves.  Every interleaving of two ranks with two warps each is then walked through, warps of the last two
forms side by side as well.  (With one activation row and 64-row chunks that is the whole protocol: warp w of a rank sends the rows that rank w
finishes, and only warp 0 reads.)"""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_native_b200", "csrc", "qmv_split.cuh")
RANKS, WARPS, CHUNKS, BUFFERS = 2, 2, 8, 4
AREAS = {"f16": 2, "integers": 4, "halves": 4}


def source():
    with open(SRC) as f:
        return f.read()


def in_order(body, patterns):
    found = []
    for step, pattern in patterns:
        at = [m.start() for m in re.finditer(pattern, body)]
        assert len(at) == 1, step
        found.append((at[0], step))
    return [step for _, step in sorted(found)]


def chunk_steps(form):
    """The steps at the end of the chunk loop, in the order of the source."""
    src = source()
    common = (("arrive", r"mbar_arrive\(&sync_bar\[i & 1u\]\)"), ("add", r"!add\(i - 1"), ("finish", r"!finish\(i - 2"))
    if form == "halves":
        body = src[src.index("// The chunks from a share on that digits do not do for"):]
        return in_order(body[:body.index("d2 = d1;")], (("write", r"sp_far_stages<"),) + common)
    body = src[src.index("---- the warps' partial sums go to shared memory"):]
    # (integers do not wait until the area has been read: they have two more)
    steps = in_order(body[:body.index("d2 = d1;")], (("wait_read", r"!INT && i >= 2 && !wait\(sync_bar\[2\]"), ("write", r"const uint32_t part = red \+ \(INT \? i & 3u : i & 1u\)")) + common)
    return [s for s in steps if form == "f16" or s != "wait_read"]


def program(steps):
    """One warp's steps: (name, chunk); waits are steps of their own."""
    p = []
    for i in range(CHUNKS):
        for s in steps:
            if s == "wait_read" and i >= 2:
                p.append(("wait_read", i - 2))
            elif s in ("write", "arrive"):
                p.append((s, i))
            elif s == "add" and i >= 1:
                p += [("add_wait", i - 1), ("send", i - 1), ("added", i - 1)]
            elif s == "finish" and i >= 2:
                p += [("finish_wait", i - 2), ("read", i - 2)]
    p += [("add_wait", CHUNKS - 1), ("send", CHUNKS - 1), ("added", CHUNKS - 1)]
    for j in (CHUNKS - 2, CHUNKS - 1):
        p += [("finish_wait", j), ("read", j)]
    return p


def overwrites(steps, areas, other=None):
    """(what, chunk) of the first write over something that is still to be read, or None; all interleavings.  `other`: the steps of the last warp of each rank."""
    progs = [program(other if other and w == WARPS - 1 else steps) for r in range(RANKS) for w in range(WARPS)]
    where = [{s: n for n, s in enumerate(p)} for p in progs]
    start = (0,) * (RANKS * WARPS)
    seen, todo, ended = {start}, [start], False
    while todo:
        pcs = todo.pop()
        done = lambda r, w, step, c: pcs[r * WARPS + w] > where[r * WARPS + w][(step, c)]
        moved = False
        for n in range(RANKS * WARPS):
            if pcs[n] == len(progs[n]):
                continue
            r, w = divmod(n, WARPS)
            step, c = progs[n][pcs[n]]
            if step == "wait_read" and not all(done(r, o, "added", c) for o in range(WARPS)):
                continue
            if step == "add_wait" and not all(done(r, o, "arrive", c) for o in range(WARPS)):
                continue
            if step == "finish_wait" and not all(done(o, r, "send", c) for o in range(RANKS)):
                continue
            # the rows of rank w are sent by warp w; warp 0 reads there
            if step == "send" and c >= BUFFERS and not done(w, 0, "read", c - BUFFERS):
                return "buffer", c
            # a warp's sums lie where they lay `areas` chunks before: every warp has added those up
            if step == "write" and c >= areas and not all(done(r, o, "added", c - areas) for o in range(WARPS)):
                return "area", c
            moved = True
            nxt = pcs[:n] + (pcs[n] + 1,) + pcs[n + 1:]
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
        if not moved:
            assert all(pc == len(p) for pc, p in zip(pcs, progs)), "the warps wait for one another"
            ended = True
    assert ended
    return None


@pytest.mark.parametrize("form,other", [("f16", None), ("integers", None), ("halves", None), ("integers", "halves"), ("halves", "integers")])
def test_nothing_is_overwritten_before_it_is_read(form, other):
    assert overwrites(chunk_steps(form), AREAS[form], chunk_steps(other) if other else None) is None


def test_the_walk_finds_an_early_arrival():
    """A warp that arrives for chunk i before it has read chunk i - 2 lets the other rank come round to the same buffer."""
    assert overwrites(["wait_read", "write", "arrive", "add", "finish"], 2) == ("buffer", 4)


@pytest.mark.parametrize("form,areas", [("f16", 1), ("integers", 3), ("halves", 3)])
def test_the_walk_finds_an_area_too_few(form, areas):
    assert overwrites(chunk_steps(form), areas)[0] == "area"


def descriptions_overwritten(slots, descriptions, chunks):
    """Whether the producer can write a chunk's description over one that a warp of its CTA still has to read: chunks of one stage each, which is when it is
    furthest ahead.  A warp reads a description with the chunk's first stage, in add one chunk later and in finish two chunks later."""
    warp = []
    for i in range(chunks):
        warp += [("use", i, i), ("release", i, i)]
        if i >= 2:
            warp.append(("use", i, i - 2))           # finish
        warp.append(("arrive", i, i))
        if i >= 1:
            warp += [("add_wait", i, i - 1), ("use", i, i - 1)]
    where = {(s, c): n for n, (s, i, c) in enumerate(warp) if s in ("release", "arrive")}
    last_use = {c: n for n, (s, i, c) in enumerate(warp) if s == "use"}
    start = (0,) * (WARPS + 1)                       # the warps' places, and the chunks that the producer has described
    seen, todo = {start}, [start]
    while todo:
        pcs = todo.pop()
        made = pcs[-1]
        nexts = []
        if made < chunks and (made < slots or all(pcs[w] > where[("release", made - slots)] for w in range(WARPS))):
            old = made - descriptions
            if old >= 0 and any(pcs[w] <= last_use[old] for w in range(WARPS)):
                return True
            nexts.append(pcs[:-1] + (made + 1,))
        for w in range(WARPS):
            if pcs[w] == len(warp):
                continue
            s, i, c = warp[pcs[w]]
            if s == "use" and i == c and made <= c:
                continue
            if s == "add_wait" and not all(pcs[o] > where[("arrive", c)] for o in range(WARPS)):
                continue
            nexts.append(pcs[:w] + (pcs[w] + 1,) + pcs[w + 1:])
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return False


def test_descriptions_outlive_their_readers():
    src = source()
    have = int(re.search(r"__shared__ SpChunk s_chunk\[(\d+)\]", src).group(1))
    slots = int(re.search(r"constexpr int kSpMaxSlots = (\d+);", src).group(1))
    assert "s_chunk[i & %du]" % (have - 1) in src
    beyond = []
    for few in (1, 2, 3, 4):
        enough = next(d for d in range(1, 12) if not descriptions_overwritten(few, d, few + d + 4))
        beyond.append(enough - few)
    assert max(beyond) == min(beyond)                # so many more than there are slots
    assert slots + beyond[0] <= have
    assert not descriptions_overwritten(slots, have, have + 4)
