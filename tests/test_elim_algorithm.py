"""The vertex elimination the GPU closures run (fap_elim.h), restated on the CPU
on random parts: numeric elimination in a least-degree order, the closed
boundary, then every row from N+ of its vertex.  Directed and undirected parts,
zero weights, unreachable vertices and parts without inner or without boundary
vertices give the distances of Floyd-Warshall; the groups' separators give the
rows of vertices outside the part."""
import numpy as np
import pytest

INF = 100000000


def _floyd(m):
    m = m.copy()
    for k in range(m.shape[0]):
        np.minimum(m, m[:, k:k + 1] + m[k:k + 1], out=m)
    return np.minimum(m, INF)


def _part(rng, s, degree, directed, zeros):
    m = np.full((s, s), INF, np.int64)
    for _ in range(int(s * degree / 2)):
        i, j = rng.integers(0, s, 2)
        if i != j:
            m[i, j] = 0 if zeros and rng.random() < 0.3 else rng.integers(1, 100)
            m[j, i] = rng.integers(1, 100) if directed else m[i, j]
    np.fill_diagonal(m, 0)
    return m


def _eliminate(m, b):
    """(order, N+ of every inner vertex, matrix of W): only pairs that elimination joins are lowered."""
    s = m.shape[0]
    w = m.copy()
    adj = [set(np.flatnonzero((m[v] < INF) | (m[:, v] < INF)).tolist()) - {v} for v in range(s)]
    left, order, nplus = set(range(b, s)), [], {}
    while left:
        v = min(left, key=lambda x: (len(adj[x]), x))
        left.remove(v)
        order.append(v)
        nplus[v] = sorted(adj[v])
        for u in nplus[v]:
            adj[u] |= adj[v] - {u}
            adj[u].discard(v)
            for x in nplus[v]:
                w[u, x] = min(w[u, x], w[u, v] + w[v, x])
    return order, nplus, w


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("s,b,degree", [(1, 0, 0.0), (1, 1, 0.0), (7, 7, 3.0), (30, 0, 2.1), (40, 6, 2.1), (40, 12, 3.5),
                                        (60, 5, 1.2)])
def test_elimination_gives_the_closure(s, b, degree, directed):
    rng = np.random.default_rng(s * 100 + b + directed)
    for trial in range(4):
        m = _part(rng, s, degree, directed, zeros=trial % 2 == 1)
        want = _floyd(m)
        order, nplus, w = _eliminate(m, b)
        d = np.full((s, s), INF, np.int64)
        d[:b, :b] = _floyd(np.minimum(w[:b, :b], INF)) if b else 0
        np.fill_diagonal(d, 0)
        placed = list(range(b))
        for v in reversed(order):               # rows and columns of the vertices placed so far
            for x in placed:
                d[v, x] = min([INF] + [w[v, u] + d[u, x] for u in nplus[v]])
                d[x, v] = min([INF] + [d[x, u] + w[u, v] for u in nplus[v]])
            placed.append(v)
        assert np.array_equal(d, want), (s, b, trial)


@pytest.mark.parametrize("directed", [False, True])
def test_separators_give_the_rows_outside(directed):
    """D[v][x] = min over u in N+(v) of F[v][u] + D[u][x] with the part's exact
    distances F, for x outside the part (no inner vertex has an arc out of it)."""
    rng = np.random.default_rng(7 + directed)
    s, b, out = 45, 7, 20
    inside = _part(rng, s, 2.6, directed, zeros=True)
    m = np.full((s + out, s + out), INF, np.int64)
    m[:s, :s] = inside
    m[s:, s:] = _part(rng, out, 3.0, directed, zeros=False)
    for _ in range(12):
        i, j = rng.integers(0, b), s + rng.integers(0, out)
        m[i, j] = rng.integers(1, 50)
        m[j, i] = rng.integers(1, 50) if directed else m[i, j]
    dist = _floyd(m)
    order, nplus, _ = _eliminate(inside, b)
    for v in order:
        rows = [dist[v, u] + dist[u, s:] for u in nplus[v]]
        assert np.array_equal(np.minimum(np.min(rows, axis=0), INF) if rows else np.full(out, INF), dist[v, s:])
