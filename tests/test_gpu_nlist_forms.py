"""GPU: neighbour sets of the list build in the forms that take different builds
-- few and many cells, light cells, stencils of more than 32 columns, stencils
that span the box or hold more atoms than a tile, minimum image and cell shift,
both precisions -- against all pairs by the same operations in torch, with pairs
across the faces and within a few units in the last place of the radius."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {
    # atoms, box, cell, cutoff
    "few_cells": (1500, (12.0, 13.0, 12.5), 2.86, 2.5),      # two blocks an SM
    "spans": (1500, (9.0, 9.5, 14.0), 2.0, 3.5),             # stencil as wide as the box in x and y
    "spans_slab": (3000, (11.0, 11.5, 70.0), 2.2, 4.0),      # the same over 775 cells: binary64 three blocks an SM
    "cells_of_two": (3000, (15.6, 15.0, 16.0), 1.4, 2.5),    # 1,210 cells, most of them light
    "one_to_a_cell": (3000, (20.0, 20.0, 20.0), 1.5, 3.0),   # 2,197 cells
    "wide_stencil": (4000, (17.0, 17.0, 18.0), 1.0, 2.3),    # 49 columns
    "vapour": (1200, (40.0, 41.0, 45.0), 2.86, 5.0),
    "over_the_tile": (14000, (25.0, 26.0, 27.0), 2.86, 7.7),  # 729 atoms times five a stencil
}


def all_pairs(pos, box, rl, real, shift_first):
    import torch
    t = torch.float32 if real == 0 else torch.float64
    x = torch.tensor(pos, device="cuda").to(t)
    L = torch.tensor(box, device="cuda").to(t)
    Li = (1.0 / torch.tensor(box, device="cuda")).to(t)
    r2 = torch.tensor(rl, dtype=torch.float64, device="cuda").to(t) ** 2
    n, out = len(pos), []
    for i0 in range(0, n, 500):
        d2 = None
        for d in range(3):
            xi, xj = x[i0:i0 + 500, d, None], x[None, :, d]
            r = xj - xi
            s = torch.floor(r * Li[d] + 0.5) * L[d]
            e = (xj - s) - xi if shift_first else r - s
            d2 = e * e if d2 is None else d2 + e * e
        m = d2 < r2
        m[torch.arange(len(m)), torch.arange(i0, i0 + len(m))] = False
        out.append((m.nonzero() + torch.tensor([i0, 0], device="cuda")).cpu().numpy())
    return np.concatenate(out)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", ["minimage", "cellshift"])
@pytest.mark.parametrize("form", list(FORMS))
def test_sets_of_every_form(mdf, form, mode, prec):
    n, box, cell, rc = FORMS[form]
    box = np.array(box)
    rng = np.random.default_rng(len(form) + n)
    pos = rng.uniform(0, 1, (n, 3)) * box
    pos[:30, 0] = 0.0
    pos[30:60, 1] = np.float32(box[1]) * (1 - 2.0 ** -23)
    # partners at the radius, a few units in the last place to either side
    rl = float(np.float32(rc) + np.float32(0.3))
    u = rng.normal(size=(200, 3))
    u *= (rl * (1 + rng.integers(-3, 4, 200) * (2.0 ** -23 if prec == 0 else 2.0 ** -52)) / np.sqrt((u ** 2).sum(1)))[:, None]
    pos[200:400] = pos[:200] + u
    pos = np.mod(pos, box)
    if prec == 0:
        pos = pos.astype(np.float32).astype(np.float64)
    pos[pos >= box] = 0.0
    sys = mdf.MDSystem(pos, box, precision=prec)
    sys.set_rcut(np.full(n, rc, np.float32))
    cl = mdf.CellList(sys, cell)
    cl.rebuild()
    shift = mode == "cellshift"
    nl = mdf.NeighborList(sys, rl, 0.0 if shift else 0.3, mode=mdf.NL_CELLSHIFT if shift else mdf.NL_MINIMAGE)
    nl.fit(sys, cl)
    nl.rebuild(sys, cl)
    counts, pairs = nl.lists()
    nc = cl.ncell()
    reach = np.ceil(rl / (box / nc))
    cells_shift = shift and (np.array(nc) >= 4).all() and (2 * reach + 1 <= nc).all()
    if prec == 1:  # the per-atom radius is a binary32 cutoff and the skin added in binary64
        rl = float(np.float32(rc)) + 0.3 if not shift else rl
    want = all_pairs(sys.positions(), box, rl, prec, cells_shift)
    assert np.array_equal(counts, np.bincount(want[:, 0], minlength=n))
    rows = np.repeat(np.arange(n, dtype=np.int64), counts) * n
    assert np.array_equal(np.sort(rows + pairs), np.sort(want[:, 0] * n + want[:, 1]))
