"""A tree of 16,384 leaves whose blocks of 256 leave more subtrees to the last one than that merges in
its shared memory (1,024): codes that share a long prefix on both sides of every block's end."""
import numpy as np
import pytest

from tests.test_lbvh_gpu import _pair, _same_tree

pytestmark = pytest.mark.gpu

BLOCK, BLOCKS = 256, 64


def _codes():
    """Sorted unique 30-bit codes.  Around the end of block k - 1 they are 6 bits of k and 24 alternating
    bits: of the two codes there one ends on 0 and one on 1, and a neighbor leaves that pattern at each
    of its bits, to the left where the bit is 1 and to the right where it is 0."""
    pattern = "01" * 11 + "0"
    left = [pattern[:i] + "0" + "1" * (23 - i) for i, b in enumerate(pattern) if b == "1"]
    left += [pattern + "0"]
    right = [pattern + "1"]
    right += [pattern[:i] + "1" + "0" * (23 - i) for i, b in enumerate(pattern) if b == "0"][::-1]
    bulk = [format((3 << 22) + k, "024b") for k in range(BLOCK)]  # under the first 1, after all of those
    blocks = []
    for k in range(BLOCKS):
        r, nxt = format(k, "06b"), format(k + 1, "06b")
        head = [r + s for s in right] if k else []
        tail = [nxt + s for s in left] if k + 1 < BLOCKS else []
        blocks += head + [r + s for s in bulk[: BLOCK - len(head) - len(tail)]] + tail
    return blocks


def _triangles(codes):
    cell = np.array([[int(c[a::3], 2) for a in range(3)] for c in codes])
    lo, hi = (cell + 0.4) / 1024, (cell + 0.6) / 1024
    lo[0], hi[-1] = 0.0, 1.0  # the first and the last leaf span the unit cube: codes are cells
    return np.stack([lo, hi, np.stack([lo[:, 0], hi[:, 1], lo[:, 2]], 1)], 1)


def _left_over(nodes, n):
    """Subtrees inside one block whose parent is not."""
    parent, left, right = (nodes[:, k].astype(np.int64) for k in range(3))
    first = np.full(2 * n - 1, -1)
    last = np.full(2 * n - 1, -1)
    order, stack = [], [0]
    while stack:
        v = stack.pop()
        order.append(v)
        if v < n - 1:
            stack += [left[v], right[v]]
    for v in reversed(order):
        if v >= n - 1:
            first[v] = last[v] = v - (n - 1)
        else:
            first[v], last[v] = first[left[v]], last[right[v]]
    inside = first // BLOCK == last // BLOCK
    return int((inside[1:] & ~inside[np.where(parent[1:] < n, parent[1:], 0)]).sum())


def test_build_and_refits_match_oracle(xrt):
    codes = _codes()
    codes[0], codes[-1] = "0" * 30, "1" * 30
    assert codes == sorted(set(codes)) and len(codes) == BLOCK * BLOCKS
    rng = np.random.default_rng(5)
    p = _triangles(codes)[rng.permutation(len(codes))].astype(np.float32).reshape(-1, 9)
    g, o = _pair(p)
    t = _same_tree(g, o)
    assert t["unique"] and [int(c, 2) for c in codes] == t["morton"].tolist()
    assert _left_over(t["nodes"], len(codes)) > 1024
    for _ in range(3):
        moved = (p + rng.normal(0, 0.05, p.shape)).astype(np.float32)
        g.refit(moved)
        o.refit(moved)
        _same_tree(g, o)
    g.build(p[: len(p) // 2])  # the same memory, and a tree whose subtrees do fit
    o.build(p[: len(p) // 2], None, 0.0)
    _same_tree(g, o)
