"""Neighbour sets of the list build where its routes meet: pairs at exactly
the list radius (the packed tile's test hands them to the exact one), light
home cells beside full ones and on the periodic faces, stencils that overflow
the tile, that span the box, and that need more runs than a home cell holds.
The sets equal the all-pairs oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(n, a):
    return np.stack(np.meshgrid(*[np.arange(k) * a for k in n], indexing="ij"), -1).reshape(-1, 3)


def _shape(kind):
    rng = np.random.default_rng(17)
    if kind == "ties":  # every neighbour shell at an exact distance, one of them the list radius
        pos, box, cell, rc = _lattice((16, 16, 32), 1.0), [16.0, 16.0, 32.0], 2.8, [3.0]
    elif kind == "near_ties":  # the same, moved off the ties by a few units in the last place
        pos, box, cell, rc = _lattice((16, 16, 32), 1.0), [16.0, 16.0, 32.0], 2.8, [3.0]
        pos = np.mod(pos + rng.integers(-2, 3, pos.shape) * 2.0 ** -20, box)
    elif kind == "vapour":  # one to a few atoms a cell, some on the faces
        box = [30.0, 28.0, 95.0]
        pos, cell, rc = rng.random((3000, 3)) * box, 2.8, [2.5, 3.0, 4.5, 5.0]
        pos[:40, 2], pos[40:80, 0], pos[80:120, 1] = 0.0, 0.0, np.float32(box[1]) * (1 - 2.0 ** -23)
    elif kind == "drop":  # a dense block in vapour: full and light cells side by side
        box = [22.0, 22.0, 60.0]
        pos = np.concatenate([_lattice((18, 18, 18), 1.1) + [1.0, 1.0, 50.0], rng.random((500, 3)) * box])
        cell, rc = 2.8, [2.5, 4.0, 5.0]
    elif kind == "dense":  # 5,000 candidates a stencil
        box = [17.0, 17.0, 19.0]
        pos, cell, rc = rng.random((11000, 3)) * box, 2.8, [3.0, 3.5]
    elif kind == "small_box":  # the stencil spans every axis
        box = [8.0, 8.5, 9.0]
        pos, cell, rc = rng.random((1500, 3)) * box, 2.0, [2.5, 3.5]
    elif kind == "thin_box":  # and one axis only
        box = [7.0, 20.0, 40.0]
        pos, cell, rc = rng.random((4000, 3)) * box, 2.8, [2.5, 3.0]
    else:  # "fine_cells": 121 columns a stencil
        box = [14.0, 14.0, 15.0]
        pos, cell, rc = rng.random((2500, 3)) * box, 1.0, [4.0, 4.5]
    return pos, np.array(box), cell, rng.choice(np.array(rc, np.float32), len(pos))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", ["ties", "near_ties", "vapour", "drop", "dense", "small_box", "thin_box", "fine_cells"])
def test_neighbour_sets(mdf, orc, kind, prec):
    pos, box, cell, rc = _shape(kind)
    s = mdf.MDSystem(np.mod(pos, box), box, precision=prec)
    s.set_rcut(rc)
    cl = mdf.CellList(s, cell)
    cl.rebuild()
    nl = mdf.NeighborList(s, float(rc.max()), 0.0, expansion=1.5)
    if kind == "fine_cells":  # more runs than a home cell holds: refused
        with pytest.raises(mdf.MDExcptShortNeighborList):
            nl.fit(s, cl)
        return
    nl.fit(s, cl)
    c, p = nl.lists()
    gp, grc = s.positions(), s.rcut()
    if prec == 0:
        oc, op = orc.nlist_allpair_f32(gp.astype(np.float32), grc, 0.0, box.astype(np.float32), cap=2048)
    else:
        oc, op = orc.nlist_allpair_f64(gp, grc.astype(np.float64), 0.0, box, cap=2048)
    assert np.array_equal(c, oc)
    rows = np.repeat(np.arange(s.n, dtype=np.int64), c) * s.n
    assert np.array_equal(np.sort(rows + p), np.sort(rows + op))
