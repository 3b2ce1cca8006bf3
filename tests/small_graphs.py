"""Small graphs in the Edge / ID / Cut formats, for the edge cases of kernels."""


def write(root, n, edges, H):
    """Edge / ID / Cut files of an undirected graph (u, v, w forth, w back);
    the partition halves the vertex range level by level."""
    e, i, c = (str(root / f) for f in ("Edge.txt", "ID.txt", "Cut.txt"))
    with open(e, "w") as f:
        f.write("%d %d\n" % (n, 2 * len(edges)))
        for u, v, w, x in edges:
            f.write("a %d %d %d\na %d %d %d\n" % (u + 1, v + 1, w, v + 1, u + 1, x))
    with open(i, "w") as f:
        f.write("%d\n" % n + "".join("%d 0.0 0.0 %d\n" % (k, k) for k in range(n)))
    with open(c, "w") as f:
        f.write("%d\n" % H)
        cells = [(0, n)]
        for h in range(1, H + 1):
            f.write("".join("%d %d %d\n" % (h, a, b) for a, b in cells))
            cells = [x for a, b in cells for x in ((a, (a + b) // 2), ((a + b) // 2, b))]
    return e, i, c


def path(n):
    return n, [(k, k + 1, 1 + k % 7) for k in range(n - 1)]


def star(leaves):
    return leaves + 1, [(leaves, k, 3 + k % 5) for k in range(leaves)]


def clique(n):
    return n, [(a, b, 5 + (a * 7 + b * 11) % 23) for a in range(n) for b in range(a)]


def clique_with_tails(n, tail):
    """Tails are light subtrees of `tail` nodes hanging off a clique's chain."""
    n0, edges = clique(n)
    edges = list(edges)
    for k in range(n):
        prev = k
        for t in range(tail):
            edges.append((prev, n0, 1 + (k + t) % 9))
            prev = n0
            n0 += 1
    return n0, edges


def grid(r, c):
    e = []
    for y in range(r):
        for x in range(c):
            if x + 1 < c:
                e.append((y * c + x, y * c + x + 1, 1 + (3 * x + 5 * y) % 13))
            if y + 1 < r:
                e.append((y * c + x, (y + 1) * c + x, 1 + (7 * x + 2 * y) % 11))
    return r * c, e
