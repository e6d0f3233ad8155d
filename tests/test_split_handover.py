"""Hand-over of partial sums between the ranks of a cluster (csrc/qmv_split.cuh): no buffer is written again before every warp has read it.

The order of a warp's steps for one chunk is taken from the kernel's source; every interleaving of two ranks with two warps each is then
walked through.  (With one activation row and 64-row chunks that is the whole protocol: warp w of a rank sends the rows that rank w
finishes, and only warp 0 reads.)"""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_native_b200", "csrc", "qmv_split.cuh")
RANKS, WARPS, CHUNKS, BUFFERS = 2, 2, 8, 4


def chunk_steps():
    """The steps at the end of the chunk loop, in the order of the source."""
    with open(SRC) as f:
        src = f.read()
    body = src[src.index("---- the warps' partial sums go to shared memory"):]
    body = body[:body.index("d2 = d1;")]
    found = []
    for step, pattern in (("wait_read", r"wait\(sync_bar\[2\]"), ("arrive", r"mbar_arrive\(&sync_bar\[i & 1u\]\)"), ("add", r"!add\(i - 1"),
                          ("finish", r"!finish\(i - 2")):
        at = [m.start() for m in re.finditer(pattern, body)]
        assert len(at) == 1, step
        found.append((at[0], step))
    return [step for _, step in sorted(found)]


def program(steps):
    """One warp's steps: (name, chunk); waits are steps of their own."""
    p = []
    for i in range(CHUNKS):
        for s in steps:
            if s == "wait_read" and i >= 2:
                p.append(("wait_read", i - 2))
            elif s == "arrive":
                p.append(("arrive", i))
            elif s == "add" and i >= 1:
                p += [("add_wait", i - 1), ("send", i - 1), ("added", i - 1)]
            elif s == "finish" and i >= 2:
                p += [("finish_wait", i - 2), ("read", i - 2)]
    p += [("add_wait", CHUNKS - 1), ("send", CHUNKS - 1), ("added", CHUNKS - 1)]
    for j in (CHUNKS - 2, CHUNKS - 1):
        p += [("finish_wait", j), ("read", j)]
    return p


def overwrites(steps):
    """(chunk, buffer's chunk) of the first write over rows that are still to be read, or None; all interleavings."""
    p = program(steps)
    where = {s: n for n, s in enumerate(p)}
    start = (0,) * (RANKS * WARPS)
    seen, todo, ended = {start}, [start], False
    while todo:
        pcs = todo.pop()
        done = lambda r, w, step, c: pcs[r * WARPS + w] > where[(step, c)]
        moved = False
        for n in range(RANKS * WARPS):
            if pcs[n] == len(p):
                continue
            r, w = divmod(n, WARPS)
            step, c = p[pcs[n]]
            if step == "wait_read" and not all(done(r, o, "added", c) for o in range(WARPS)):
                continue
            if step == "add_wait" and not all(done(r, o, "arrive", c) for o in range(WARPS)):
                continue
            if step == "finish_wait" and not all(done(o, r, "send", c) for o in range(RANKS)):
                continue
            # the rows of rank w are sent by warp w; warp 0 reads there
            if step == "send" and c >= BUFFERS and not done(w, 0, "read", c - BUFFERS):
                return c, c - BUFFERS
            moved = True
            nxt = pcs[:n] + (pcs[n] + 1,) + pcs[n + 1:]
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
        if not moved:
            assert all(pc == len(p) for pc in pcs), "the warps wait for one another"
            ended = True
    assert ended
    return None


def test_no_buffer_is_overwritten_before_it_is_read():
    assert overwrites(chunk_steps()) is None


def test_the_walk_finds_an_early_arrival():
    """A warp that arrives for chunk i before it has read chunk i - 2 lets the other rank come round to the same buffer."""
    assert overwrites(["wait_read", "arrive", "add", "finish"]) is not None
