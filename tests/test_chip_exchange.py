"""The index arithmetic of the on-chip PCG (csrc/pcg_chip.cu), restated on the CPU: how a grid is
cut into boxes, which nodes boxes share, where a neighbour's packet lies, which thread writes each
word of the two halves of w, and that the sum over boxes is K u."""
import itertools

import numpy as np
import pytest

from genpipeline_gb300 import bcs


def span(n, P, a):
    q, r = divmod(n, P)
    return a * q + min(a, r), q + (a < r)


def side(i, e, a, P):
    return (1 if a > 0 else 0) if i == 0 else (2 if i == e and a + 1 < P else 0)


def boxes(grid, cuts):
    return list(itertools.product(*(range(P) for P in cuts)))


def plans():
    rng = np.random.default_rng(11)
    out = [((64, 64, 64), (8, 8, 2)), ((5, 1, 1), (5, 1, 1)), ((7, 9, 33), (3, 2, 4)), ((1, 4, 70), (1, 2, 3)),
           ((32, 8, 8), (16, 1, 1)), ((2, 2, 2), (2, 2, 2)), ((40, 6, 17), (1, 1, 1))]
    while len(out) < 40:
        g = tuple(int(v) for v in rng.integers(1, 40, 3))
        c = tuple(int(rng.integers(1, min(n, 6) + 1)) for n in g)
        if -(-g[2] // c[2]) <= 32:
            out.append((g, c))
    return out


@pytest.mark.parametrize("grid,cuts", plans())
def test_packets_of_shared_nodes(grid, cuts):
    """Every shared node's packet offset in direction (dx, dy, dz) is the same grid node in that
    neighbour's box, and exactly one holder counts a node in the sums."""
    ext = [-(-n // P) + 1 for n, P in zip(grid, cuts)]
    SZ, SY, stride = ext[2], ext[1] * ext[2], ext[0] * ext[1] * ext[2]
    at = {b: k for k, b in enumerate(boxes(grid, cuts))}
    counted = np.zeros([n + 1 for n in grid], dtype=int)
    held = np.zeros_like(counted)
    for b, bid in at.items():
        s = [span(n, P, a) for n, P, a in zip(grid, cuts, b)]
        e = [v[1] for v in s]
        for node in itertools.product(*(range(v + 1) for v in e)):
            sd = [side(i, ee, a, P) for i, ee, a, P in zip(node, e, b, cuts)]
            gn = tuple(v[0] + i for v, i in zip(s, node))
            held[gn] += 1
            counted[gn] += 2 not in sd
            o = node[0] * SY + node[1] * SZ + node[2]
            assert o < stride
            order = []
            for m in range(8):  # the order of the partial sums: the boxes' own order
                d, use = [0, 0, 0], True
                for ax in range(3):
                    hi, me = (m >> (2 - ax)) & 1, int(sd[ax] == 1)
                    use = use and not (sd[ax] == 0 and hi)
                    if sd[ax] and hi != me:
                        d[ax] = 1 if hi else -1
                if not use:
                    continue
                nb = tuple(x + y for x, y in zip(b, d))
                order.append(nb)
                if d == [0, 0, 0]:
                    continue
                off = ((d[0] * cuts[1] + d[1]) * cuts[2] + d[2]) * stride
                for ax, st in enumerate((SY, SZ, 1)):
                    if d[ax]:
                        off += (span(grid[ax], cuts[ax], b[ax] - 1)[1] if d[ax] < 0 else -e[ax]) * st
                pos = bid * stride + o + off
                assert pos // stride == at[nb]
                loc = pos % stride
                theirs = (loc // SY, loc % SY // SZ, loc % SZ)
                ns = [span(n, P, a) for n, P, a in zip(grid, cuts, nb)]
                assert all(0 <= i <= v[1] for i, v in zip(theirs, ns))
                assert tuple(v[0] + i for v, i in zip(ns, theirs)) == gn
            assert order == sorted(order) and len(order) == 2 ** sum(v != 0 for v in sd)
    assert (counted == 1).all() and (held >= 1).all()


@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 3, 5), (3, 8, 32), (9, 4, 7), (12, 2, 16), (5, 11, 3)])
def test_march_writes_each_half_once_and_sums_to_K_u(grid):
    """The march of one box: rows packed into warps, G pairs of x slabs; every place of W0 and W1 gets
    one store, both copies of a slab's end the same sum, one copy of each node counts, and the sum of
    the two halves is the product of the oracle."""
    from oracle import oracle as O

    ex, ey, ez = grid
    NX, NY, NZ = ex + 1, ey + 1, ez + 1
    rng = np.random.default_rng(3)
    E, u = rng.uniform(0.1, 1, (ex, ey, ez)), rng.standard_normal((NX, NY, NZ, 3))
    ke = O.ke_quadrature()
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]

    def product(i, j, k):
        v = np.concatenate([u[i + a, j + b, k + c] for a, b, c in corner])
        y = (E[i, j, k] * ke @ v).reshape(8, 3)
        return {corner[n]: y[n] for n in range(8)}

    rpw = 32 // ez
    groups = -(-ey // rpw)
    for G in range(1, max(1, 8 // groups) + 1):
        if 2 * G > ex + 1 or groups * G > 8:
            continue
        # a place: slab pair, plane of the slab, row, column, lane; a slab's last plane is also the first of
        # the next one, whose copy counts
        L = -(-ex // (2 * G))
        shape = (G, L + 1, NY, NZ, 2)
        W, stored = np.zeros((2, *shape, 3)), np.zeros((2, *shape), dtype=int)
        late, seen = [], set()
        for warp, lane, h in itertools.product(range(groups * G), range(32), range(2)):
            gp, jrow, k = warp // groups, (warp % groups) * rpw + lane // ez, lane % ez
            if lane >= rpw * ez or jrow >= ey:
                continue
            slab, carry = gp + h * G, np.zeros((2, 2, 3))
            for t in range(L + 1):
                i = slab * L + t
                out = carry.copy()
                if t < L and i < ex:
                    seen.add((i, jrow, k))
                    y = product(i, jrow, k)
                    for cy, cz in itertools.product((0, 1), (0, 1)):
                        out[cy, cz] += y[0, cy, cz]
                        carry[cy, cz] = y[1, cy, cz]
                else:
                    carry[:] = 0.0
                for cy, cz in itertools.product((0, 1), (0, 1)):
                    at = (cy, gp, t, jrow + cy, k + cz, h)
                    if cz == 0 or k == ez - 1:
                        stored[at] += 1  # the lane above stores node k + 1, with this lane's half from a shuffle
                    if t == L and slab + 1 < 2 * G:
                        late.append((at, out[cy, cz]))
                    else:
                        W[at] += out[cy, cz]
        assert len(seen) == ex * ey * ez
        for (cy, gp, _, j, k, h), val in late:
            # the next slab's first plane takes the sum, and so does this copy
            nxt = (cy, gp + 1, 0, j, k, h) if gp + 1 < G else (cy, 0, 0, j, k, 1)
            W[nxt] += val
        for (cy, gp, t, j, k, h), _ in late:
            nxt = (cy, gp + 1, 0, j, k, h) if gp + 1 < G else (cy, 0, 0, j, k, 1)
            W[cy, gp, t, j, k, h] = W[nxt]
        assert (stored[0][:, :, :ey] == 1).all() and (stored[0][:, :, ey] == 0).all()
        assert (stored[1][:, :, 1:] == 1).all() and (stored[1][:, :, 0] == 0).all()
        y = O.apply(grid, ke, E.reshape(-1), u.reshape(-1)).reshape(NX, NY, NZ, 3)
        counts = np.zeros((NX, NY, NZ), dtype=int)
        for gp, t, h in itertools.product(range(G), range(L + 1), range(2)):
            i = (gp + h * G) * L + t
            if i > ex:
                continue
            counts[i] += t < L or gp + h * G + 1 == 2 * G
            np.testing.assert_allclose(W.sum(0)[gp, t, :, :, h], y[i], rtol=0, atol=1e-12 * np.abs(y).max())
        assert (counts == 1).all()


def test_boxes_cover_the_elements():
    for grid, cuts in plans():
        n = np.zeros(grid, dtype=int)
        for b in boxes(grid, cuts):
            sl = tuple(slice(s, s + e) for s, e in (span(m, P, a) for m, P, a in zip(grid, cuts, b)))
            n[sl] += 1
        assert (n == 1).all() and bcs.n_nodes(*grid) == np.prod([m + 1 for m in grid])
