"""The stage kernels' two item lists (lean: no PML cell and no cell outside the
grid; general: the rest) at the edges of their tiles: grids whose layers end
on, before and after tile boundaries (32 cells in x, 8 in y), with and without
a bottom layer of its own z-chunk, and with a few interior planes only.

FP32 storage against the FP64 oracle within the parity bound of the other
tests, 1e-5 relative L2.  16-bit storage against FP32 storage: a store rounds
by at most 2^-11 (FP16) or 2^-8 (BF16) of the value and a step stores each
field five times (W three times, the accumulator, FW), so three steps differ
by at most 15 of those."""
import numpy as np
import pytest

import cases
import cgfd
import models
import pyoracle
from helpers import comp_errors, rel_l2

pytestmark = pytest.mark.gpu

GRIDS = [  # ni, nj, nk, nabs
    (96, 40, 24, (8, 8, 8, 8, 8, 0)),      # lean tiles between layers
    (64, 16, 12, (0, 0, 0, 0, 0, 0)),      # lean tiles only
    (65, 17, 11, (0, 0, 0, 0, 3, 0)),      # one cell past the tiles, thin bottom layer
    (101, 27, 19, (32, 5, 3, 1, 4, 0)),    # layer ends on a tile boundary, uneven sides
    (100, 9, 20, (1, 35, 0, 0, 9, 0)),     # one row past a tile
    (40, 30, 13, (4, 4, 4, 4, 6, 0)),      # seven planes above the bottom layer: no lean item
]


def _model(g):
    ni, nj, nk, nabs = g
    return models.gaussian_hill(ni=ni, nj=nj, nk=nk, nt=4, dz_top=60.0, dz_bot=120.0,
                                hill_h=200.0, hill_w=600.0, con_depth=400.0, src_depth=300.0,
                                corr_len=200.0, nabs=nabs, f0=0.08, t0=0.25, n_side=2,
                                rcv_spacing=300.0)


def _run(m, init, storage):
    s = cgfd.Solver(m.desc(storage=storage))
    m.load(s)
    if storage == cgfd.STORE_F16:  # the fields' magnitudes, not the source's
        s.set_field_scales([0] * 3 + [14] * 6)
    for c in range(9):
        s.set_field(c, init[c])
    s.step(3)
    out = np.stack([s.get_field(c) for c in range(9)])
    s.close()
    return out


@pytest.mark.parametrize("grid", GRIDS)
def test_item_lists_match_the_oracle(grid):
    m = _model(grid)
    init = cases.random_fields(m, 17)
    o = pyoracle.OracleSolver(m.desc(), 0)
    m.load(o)
    for c in range(9):
        o.set_field(c, init[c])
    o.step(3)
    ref = np.stack([o.get_field(c, 0) for c in range(9)])
    o.close()
    got = _run(m, init, cgfd.STORE_F32)
    for c, e in enumerate(comp_errors(got, ref)):
        assert e < 1e-5, (cgfd.COMPONENTS[c], e)
    for store, ulp in ((cgfd.STORE_F16, 2.0 ** -11), (cgfd.STORE_BF16, 2.0 ** -8)):
        w = _run(m, init, store)
        for c in range(9):
            assert rel_l2(w[c], got[c]) < 15 * ulp, (store, cgfd.COMPONENTS[c])
