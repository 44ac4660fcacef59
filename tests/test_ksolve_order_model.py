"""A CPU model of the hand-over of results in k_ksolve (ksolve.cu): which
arrivals of asynchronous stores are certain to come before which sends.

Every block's forward result y_b and later its backward result x_b are sent
to the same shared-memory slot of every CTA of the cluster by st.async, and
two such stores are ordered only if the first one's arrival happens before the
second is sent.  The model builds the happens-before graph from the kernel's
waits (block b belongs to warp b mod 8C, its CTA waits for what b needs) and
asks for every block and CTA whether y_b's arrival comes before x_b's send."""
import os
import re

import numpy as np
import pytest

WARPS = 8
KSOLVE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfls_b200", "csrc", "device",
                      "ksolve.cu")


def unordered(nblk, ctas, barrier):
    """(block, CTA) pairs for which y_b may arrive after x_b was sent; barrier: every CTA waits for every y and the
    cluster meets between the passes, else an owner waits in its own CTA only, for its block's y and the last one."""
    cta = [(b // WARPS) % ctas for b in range(nblk)]
    ids = {}
    node = lambda *k: ids.setdefault(k, len(ids))
    edges = []
    for b in range(nblk):
        for c in range(ctas):
            edges.append((node("send y", b), node("y there", b, c)))
            edges.append((node("send x", b), node("x there", b, c)))
            if barrier:
                edges.append((node("y there", b, c), node("met")))
        edges += [(node("y there", k, cta[b]), node("send y", b)) for k in range(b)]
        edges += [(node("x there", k, cta[b]), node("send x", b)) for k in range(b + 1, nblk)]
        edges.append((node("send y", b), node("send x", b)))
        edges += [(node("met"), node("send x", b))] if barrier else [
            (node("y there", k, cta[b]), node("send x", b)) for k in (b, nblk - 1)]
    n = len(ids)
    reach = np.eye(n, dtype=bool)
    for a, b in edges:
        reach[a, b] = True
    while True:
        r = reach.astype(np.float32)
        more = (r @ r) > 0
        if np.array_equal(more, reach):
            break
        reach = more
    return [(b, c) for b in range(nblk) for c in range(ctas)
            if not reach[ids[("y there", b, c)], ids[("send x", b)]]]


@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
@pytest.mark.parametrize("nblk", [1, 2, 7, 8, 9, 21, 33, 70])
def test_every_y_has_landed_before_its_x_is_sent(nblk, ctas):
    assert unordered(nblk, ctas, barrier=True) == []


def test_waiting_for_the_last_y_alone_leaves_ctas_without_later_blocks():
    # 21 blocks on four CTAs: 0-7, 8-15, 16-20 and none
    last = [7, 15, 20, -1]
    assert unordered(21, 4, barrier=False) == [(b, c) for b in range(21) for c in range(4) if b > last[c]]


def test_kernel_meets_between_its_two_sends():
    src = re.sub(r"//[^\n]*", "", open(KSOLVE).read())
    body = src[src.index("k_ksolve(const SubDev"):]
    sends = [m.start() for m in re.finditer(r"\bsend_block\(xs", body)][:2]
    between = body[sends[0]:sends[1]]
    met = between.index("cluster_sync_all();")
    assert re.search(r"for \(int b = threadIdx\.x; b < nblk[^)]*\) ok = bar_wait_cluster\(&fwd\[b\]\);", between[:met])
