"""What the MMA of a pair of CTAs reads has happened before it (csrc/qmm_duo.cu).

CTA 0 issues the multiplications, which read both CTAs' shared memory (activations) and tensor memory (weights).  The barriers' counts and
scopes and the barrier that each step waits for or arrives at are taken from the kernel's source; what is then ordered before the MMA is what
reaches it over edges that order that kind of memory: a copy's completion on the barrier that is waited for, an arrival with release and a wait in
the same scope, and, for tensor memory only, an arrival of any kind between the fences of tcgen05."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_native_b200", "csrc", "qmm_duo.cu")


def source():
    with open(SRC) as f:
        return f.read()


def between(src, start, end):
    at = src.index(start)
    return src[at:src.index(end, at)]


def protocol(src):
    acts = between(src, "if (warp == 0) {\n        uint32_t s = 0", "} else if (warp == 1)")
    mma = between(src, "} else if (warp == 1) {", "} else if (warp == 2)")
    weights = between(src, "tmem_st_32x32_x32(a_dst", "} else {")
    arrive = between(src, "void arrive_at_0(", "}\n")
    count = re.search(r"mbar_init\(&full\[s\], ([^;]*)\);", src).group(1)
    m = re.fullmatch(r"rank == 0 \? (\d+) : (\d+)", count)
    counts = (int(m.group(1)), int(m.group(2))) if m else (int(count), int(count))
    # the barrier on which a CTA's copies complete, and the copies that are expected there
    remote = "duo::copy_3d(" in acts and re.search(r"duo::in_cta_0\(&full\[s\]\)\);", acts) is not None and "cta_group::2" in between(src, "void copy_3d(", "}\n")
    both = "if (rank == 0) mbar_expect_tx(&full[s], 2 * b_stage);" in acts
    release = "mbarrier.arrive.release.cluster" in arrive
    peer_wait = between(mma, "if (rank == 0) {", "duo::elect()")
    cluster_wait = "peer_full[s]" in peer_wait and "cluster" in peer_wait
    # weights: store, wait for it, fence, arrive; relay: wait, fence, fence, arrive; MMA: wait, fence
    steps = [weights.index(x) for x in ("tmem_st_wait();", "tc_fence_before();", "mbar_arrive(&full[sa]);")]
    relay = between(mma, "if (!mbar_wait(&full[s]", "__syncwarp();")
    hops = [relay.index(x) for x in ("mbar_wait(&full[s]", "tc_fence_after();", "mbar_wait(&peer_full[s]", "duo::mma(", "tc_fence_before();", "duo::arrive_at_0(&peer_full[s])")]
    fences = steps == sorted(steps) and hops == sorted(hops) and re.search(r"mbar_wait\(&peer_full.*?tc_fence_after\(\);.*?duo::mma\(", relay, re.S) is not None
    return {"counts": counts, "remote": remote, "both": both, "release": release and cluster_wait, "fences": fences}


def ordered(p):
    """What is ordered before CTA 0's MMA."""
    seen = set()
    # copies of CTA 0 complete on its own barrier, for which its MMA warp waits
    seen.add("activations of CTA 0")
    if p["remote"]:
        if p["both"] and p["counts"] == (9, 8):   # eight warps each, and on CTA 0 the arrival that expects both halves
            seen.add("activations of CTA 1")
    elif p["counts"] == (9, 9) and p["release"]:
        seen.add("activations of CTA 1")          # over the relay's arrival
    if p["fences"]:
        seen |= {"weights of CTA 0", "weights of CTA 1"}
    return seen


EVERYTHING = {"%s of CTA %d" % (what, cta) for what in ("activations", "weights") for cta in (0, 1)}


def test_operands_are_ordered_before_the_multiplication():
    assert ordered(protocol(source())) == EVERYTHING


def test_a_relaxed_relay_would_not_order_copies():
    """The same model on forms that order less: copies that complete on their own CTA's barrier behind a relaxed arrival; half of the copies
    expected; a store to tensor memory that is announced before its fence."""
    p = protocol(source())
    assert "activations of CTA 1" not in ordered(dict(p, remote=False, counts=(9, 9)))
    assert "activations of CTA 1" in ordered(dict(p, remote=False, counts=(9, 9), release=True))
    assert "activations of CTA 1" not in ordered(dict(p, both=False))
    late = source().replace("tmem_st_wait();\n                    tc_fence_before();", "tc_fence_before();\n                    tmem_st_wait();")
    assert late != source() and "weights of CTA 1" not in ordered(protocol(late))


def test_no_load_goes_to_both_ctas():
    """A copy goes to the CTA that asks for it; only the message that multiplications have completed goes to both."""
    lines = [l for l in source().splitlines() if ".multicast" in l]
    assert len(lines) == 1 and "tcgen05.commit" in lines[0]
