"""The stage kernels' two item lists (lean: no PML cell and no cell outside the
grid; general: the rest) at the edges of their tiles: grids whose layers end
on, before and after tile boundaries (32 cells in x, 8 in y), with and without
a bottom layer of its own z-chunk, and with a few interior planes only.

Which items each grid has is checked on the CPU (test_work_lists.py).

FP32 storage against the FP64 oracle within the parity bound of the other
tests, 1e-5 relative L2.  16-bit storage against FP32 storage: a store rounds
by at most u = 2^-11 (FP16) or 2^-8 (BF16) of the value and a step stores each
field five times (W three times, the accumulator, FW), so three steps differ
by at most 15 of those.  Four steps, which run each of the four stencil
patterns, alone and in a batch (whose kernels are compilations of their own), are
compared on every plane of cells along each axis by itself, so that an error
confined to one edge shows: there the 20 roundings of a field and those it takes
over from the others are independent, sqrt(20) u in the root mean square, held to
twice that; FP32 to 1e-5."""
import ctypes as C
import itertools

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


def _fields(s):
    return np.stack([s.get_field(c) for c in range(9)])


def _start(s, m, init, storage):
    m.load(s)
    if storage == cgfd.STORE_F16:
        s.set_field_scales([0] * 3 + [14] * 6)
    for c in range(9):
        s.set_field(c, init[c])


def _oracle4(m, init):
    o = pyoracle.OracleSolver(m.desc(), 0)
    m.load(o)
    for c in range(9):
        o.set_field(c, init[c])
    o.step(4)
    ref = np.stack([o.get_field(c, 0) for c in range(9)])
    o.close()
    return ref


def _plane_errors(got, ref):
    """Largest error of a plane of cells along x, y or z, over its values' norm
    (at least a tenth of the component's mean plane and 1% of the largest
    component of the group, as comp_errors)."""
    d, r = (np.asarray(a, np.float64)[:, 3:-3, 3:-3, 3:-3] for a in (got - ref, ref))
    group = [np.sqrt((r[:3] ** 2).sum((1, 2, 3)).max()), np.sqrt((r[3:] ** 2).sum((1, 2, 3)).max())]
    worst = 0.0
    for c in range(9):
        total = max(np.sqrt((r[c] ** 2).sum()), 1e-2 * group[c >= 3])
        for ax in range(3):
            other = tuple(a for a in range(3) if a != ax)
            n = np.sqrt((r[c] ** 2).sum(other))
            n = np.maximum(n, 0.1 * total / np.sqrt(r.shape[1 + ax]))
            worst = max(worst, (np.sqrt((d[c] ** 2).sum(other)) / n).max())
    return worst


BOUND = {cgfd.STORE_F32: 1e-5, cgfd.STORE_F16: 2 * 20 ** 0.5 * 2.0 ** -11,
         cgfd.STORE_BF16: 2 * 20 ** 0.5 * 2.0 ** -8}


@pytest.mark.parametrize("grid", GRIDS)
def test_every_stencil_pattern_plane_by_plane(grid):
    m = _model(grid)
    init = cases.random_fields(m, 23)
    ref = _oracle4(m, init)
    for storage, bound in BOUND.items():
        s = cgfd.Solver(m.desc(storage=storage))
        _start(s, m, init, storage)
        s.step(4)
        e = _plane_errors(_fields(s), ref)
        s.close()
        assert e < bound, (storage, e)


@pytest.mark.parametrize("storage", list(BOUND), ids=["f32", "f16", "bf16"])
def test_every_stencil_pattern_in_a_batch_plane_by_plane(storage):
    ms = [_model(g) for g in GRIDS]
    b = cgfd.Batch([m.desc(storage=storage) for m in ms])
    inits = [cases.random_fields(m, 30 + k) for k, m in enumerate(ms)]
    for m, s, init in zip(ms, b.models, inits):
        _start(s, m, init, storage)
    b.step(4)
    for m, s, init in zip(ms, b.models, inits):
        e = _plane_errors(_fields(s), _oracle4(m, init))
        assert e < BOUND[storage], ((m.ni, m.nj, m.nk), e)
    b.close()


@pytest.mark.parametrize("axis,at", [(0, 40), (1, 20), (2, 15)])
def test_profiles_that_are_not_one_off_the_layers(axis, at):
    """B other than 1 in the interior: such a model has general items only, alone
    and beside a plain one in a batch (the lists are rebuilt when the profiles are
    known, and once more when plain ones replace them)."""
    plain, m = _model(GRIDS[0]), _model(GRIDS[0])
    m.pml[1][axis][3 + at:3 + at + 2] = 1.25
    init = cases.random_fields(m, 41)
    ref, ref_plain = _oracle4(m, init), _oracle4(plain, init)
    assert _plane_errors(ref, ref_plain) > 1e-2
    s = cgfd.Solver(m.desc())
    _start(s, m, init, cgfd.STORE_F32)
    s.step(4)
    assert _plane_errors(_fields(s), ref) < 1e-5
    s.close()
    b = cgfd.Batch([plain.desc(), m.desc()])
    for mm, s in zip((plain, m), b.models):
        _start(s, mm, init, cgfd.STORE_F32)
    b.step(4)
    assert _plane_errors(_fields(b.models[0]), ref_plain) < 1e-5
    assert _plane_errors(_fields(b.models[1]), ref) < 1e-5
    b.close()
    s = cgfd.Solver(m.desc())
    _start(s, m, init, cgfd.STORE_F32)
    s.prepare()
    s.upload_pml(*plain.pml)
    s.step(4)
    assert _plane_errors(_fields(s), ref_plain) < 1e-5
    s.close()


@pytest.mark.parametrize("storage", list(BOUND), ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("grid", [GRIDS[0], GRIDS[3]])
def test_every_direction_in_every_stage(grid, storage):
    """The four stages of a step in each of the eight stencil directions, driven
    one by one: with the batched patterns above these are the kernels of every
    direction, stage kind, item list and storage type.  (A step's five roundings
    of each field, within the bound for four steps.)"""
    m = _model(grid)
    init = cases.random_fields(m, 51)
    s, o = cgfd.Solver(m.desc(storage=storage)), pyoracle.OracleSolver(m.desc(), 0)
    _start(s, m, init, storage)
    m.load(o)
    for d in itertools.product((1, -1), repeat=3):
        for c in range(9):  # (the layers' auxiliaries go on)
            s.set_field(c, init[c])
            o.set_field(c, init[c])
        for rk in range(4):
            s.rk_stage(rk, 0, *d)
            o.rk_stage(rk, 0, *d)
        ref = np.stack([o.get_field(c, 0) for c in range(9)])
        e = _plane_errors(_fields(s), ref)
        assert e < BOUND[storage], (d, e)
    s.close()
    o.close()


def test_planes_past_2_to_the_15():
    """A grid of 33000 planes (z ranges that once overflowed an item's two 16-bit
    halves), both item lists, against the untiled kernel on the same inputs:
    FP32 roundings of one step, 1e-5."""
    ni, nj, nk, nabs = 32, 10, 33000, (0, 0, 1, 1, 8, 0)
    shape = (ni + 6, nj + 6, nk + 6)
    rng = np.random.default_rng(61)
    prof = [[np.full(n, v) for n in shape] for v in (0.0, 1.0, 0.0)]  # APD, B, DB
    for ax, cells in ((1, [3, nj + 2]), (2, list(range(3, 11)))):
        for p, v in zip(prof, (2.0, 1.5, 20.0)):
            p[ax][cells] = v
    # a random block, repeated in z with another amplitude each time
    block = rng.standard_normal((9, ni, nj, 100)).astype(np.float32)
    amp = np.repeat(rng.uniform(0.5, 2.0, nk // 100).astype(np.float32), 100)
    out = []
    for kernel in (cgfd.KERNEL_FUSED, cgfd.KERNEL_SIMPLE):
        s = cgfd.Solver(cgfd.Desc(ni=ni, nj=nj, nk=nk, steph=100.0, stept=0.005, nt=2,
                                  con_index=nk // 2, hybrid_grid=1,
                                  nabs=(C.c_int * 6)(*nabs), kernel=kernel))
        zero, one = np.zeros(shape), np.ones(shape)
        s.upload_metric(zero, zero, one, one)
        s.upload_media(*(np.full(shape, v, np.float32) for v in (6000.0, 3464.0, 2670.0)))
        s.upload_pml(*prof)
        for c in range(9):
            f = np.zeros(shape, np.float32)
            f[3:-3, 3:-3, 3:-3] = np.tile(block[c], nk // 100) * amp * (1.0 if c < 3 else 1e7)
            s.set_field(c, f)
        s.step(1)
        out.append(_fields(s))
        s.close()
    assert _plane_errors(*out) < 1e-5
