"""The stage kernels' work lists and the launch plan around them, on a CUDA
runtime that lives on the host (tests/fakecuda): no GPU, no kernel runs."""
import ctypes as C

import numpy as np
import pytest

import cgfd
import fakecuda
import models

cudaErrorMemoryAllocation = 2


def _model(ni=96, nj=40, nk=24, nabs=(8, 8, 8, 8, 8, 0)):
    return models.gaussian_hill(ni=ni, nj=nj, nk=nk, nt=4, dz_top=60.0, dz_bot=120.0,
                                hill_h=200.0, hill_w=600.0, con_depth=400.0, src_depth=300.0,
                                corr_len=200.0, nabs=nabs, f0=0.08, t0=0.25, n_side=2,
                                rcv_spacing=300.0)


def _launched(h):
    """The stage launches' lists: {GEN_VEL, GEN_STR, LEAN} -> items, checked to
    be the same in every launch."""
    out = {}
    for q in range(h.fake_launches()):
        it = fakecuda.items(h, q)
        assert np.array_equal(out.setdefault(h.fake_list(q), it), it)
    return out


def test_failed_list_rebuild_is_reported_and_tried_again(fake):
    """A model whose profiles are not 1 off the layers has no lean items: its
    lists are rebuilt at prepare.  Whichever allocation of prepare fails, prepare
    reports it, and the next prepare rebuilds the lists instead of taking them
    for built."""
    m = _model()
    m.pml[1][0][50] = 1.5  # B in the interior
    blocks, nth, failed = fake.fake_blocks(), 0, True
    while failed:
        s = cgfd.Solver(m.desc())
        m.load(s)
        fake.fake_fail(b"cudaMalloc", nth, cudaErrorMemoryAllocation)
        try:
            s.prepare()
            failed = False
        except cgfd.CgfdError as e:
            assert "out of memory" in str(e)
        fake.fake_fail(b"cudaMalloc", 1000, 0)
        assert fake.fake_last() == 0  # nothing left for a later call to report
        fake.fake_clear_launches()
        s.prepare()
        if failed:
            assert set(_launched(fake)) == {fakecuda.GEN_VEL, fakecuda.GEN_STR}
        s.close()
        assert fake.fake_blocks() == blocks
        nth += 1
    assert nth > 1


@pytest.mark.parametrize("call", [b"cudaMalloc", b"cudaMemcpy"])
@pytest.mark.parametrize("nth", [0, 1])
def test_failed_work_shape_leaves_the_lists_in_use(fake, call, nth):
    m = _model()
    s = cgfd.Solver(m.desc())
    m.load(s)
    s.prepare()
    before, shape = _launched(fake), s.work_shape
    fake.fake_fail(call, nth, cudaErrorMemoryAllocation)
    with pytest.raises(cgfd.CgfdError, match="out of memory"):
        s.work_shape = (24, 4, 2.0)
    assert s.work_shape == shape and fake.fake_last() == 0
    fake.fake_clear_launches()
    s.step_timed(1, per_stage=True)  # the launch of a freed list fails
    after = _launched(fake)
    assert set(after) == set(before) and all(np.array_equal(after[k], before[k]) for k in after)
    s.close()


@pytest.mark.parametrize("kernel,storage", [(cgfd.KERNEL_FUSED, cgfd.STORE_F32),
                                            (cgfd.KERNEL_FUSED, cgfd.STORE_F16),
                                            (cgfd.KERNEL_FUSED, cgfd.STORE_BF16),
                                            (cgfd.KERNEL_SCALAR, cgfd.STORE_F32)])
def test_kernel_attributes_are_set_on_every_device(fake, kernel, storage):
    """The dynamic shared memory of the tiled kernels is opted into per device:
    solvers of one process on several devices all launch.  An opt-in that fails
    is reported by the solver's creation and tried again by the next."""
    m = _model()
    for device in (0, 1, 2):
        if device == 2:
            fake.fake_fail(b"cudaFuncSetAttribute", 5, cudaErrorMemoryAllocation)
            with pytest.raises(cgfd.CgfdError, match="out of memory"):
                cgfd.Solver(m.desc(kernel=kernel, storage=storage, device=device))
            assert fake.fake_last() == 0
        s = cgfd.Solver(m.desc(kernel=kernel, storage=storage, device=device))
        m.load(s)
        s.prepare()  # captures every launch
        s.close()


TILE_X, TILE_Y, LFD = 32, 8, 3
GRIDS = [  # ni, nj, nk, nabs (the first six are those of test_gpu_lean_tiles.py)
    (96, 40, 24, (8, 8, 8, 8, 8, 0)),
    (64, 16, 12, (0, 0, 0, 0, 0, 0)),
    (65, 17, 11, (0, 0, 0, 0, 3, 0)),
    (101, 27, 19, (32, 5, 3, 1, 4, 0)),
    (100, 9, 20, (1, 35, 0, 0, 9, 0)),
    (40, 30, 13, (4, 4, 4, 4, 6, 0)),
    (1, 1, 4, (0, 0, 0, 0, 0, 0)),
    (200, 300, 4, (20, 20, 20, 20, 2, 0)),
    (40, 12, 33000, (4, 4, 0, 0, 8, 0)),  # planes past 2^15
    (32, 8, 70000, (0, 0, 0, 0, 0, 0)),  # and past 2^16
]


def _covered(it, model):
    """How often the items of one model and part compute each cell."""
    ni, nj, nk, nabs = model
    n = np.zeros((nk, nj, ni), np.int8)
    for i0, j0, z0, z1 in it[:, :4]:
        assert i0 % TILE_X == 0 and i0 < ni and LFD <= z0 < z1 <= nk + LFD
        n[z0 - LFD:z1 - LFD, max(j0, 0):max(j0 + TILE_Y, 0), i0:i0 + TILE_X] += 1
    return n


@pytest.mark.parametrize("plain", [True, False], ids=["plain", "not_plain"])
@pytest.mark.parametrize("grids", [[g] for g in GRIDS] + [GRIDS[:6]],
                         ids=["x".join(map(str, g[:3])) for g in GRIDS] + ["batch"])
def test_items_cover_every_cell_once(fake, grids, plain):
    """Every cell is an item's of each part exactly once; lean items hold cells
    of the grid outside the layers only, and where a model is deep enough they
    hold every whole tile of those."""
    descs = [cgfd.Desc(ni=ni, nj=nj, nk=nk, steph=100.0, stept=0.005, nt=4,
                       con_index=nk // 2 + LFD, hybrid_grid=1, nabs=(C.c_int * 6)(*nabs))
             for ni, nj, nk, nabs in grids]
    b = cgfd.Batch(descs) if len(grids) > 1 else None
    solvers = b.models if b else [cgfd.Solver(descs[0])]
    for s, (ni, nj, nk, _) in zip(solvers, grids):
        shape = (ni + 6, nj + 6, nk + 6)
        one, zero = np.ones(shape), np.zeros(shape)
        s.upload_metric(zero, zero, one, one)
        s.upload_media(*(np.full(shape, v, np.float32) for v in (6000.0, 3464.0, 2670.0)))
        prof = [[np.full(n, v) for n in shape] for v in (0.0, 1.0, 0.0)]
        if not plain:
            prof[1][2][nk // 2 + LFD] = 1.25
        s.upload_pml(*prof)
    if b:  # not the members' own launches
        for s in solvers:
            s.prepare()
        fake.fake_clear_launches()
    (b or solvers[0]).prepare()
    lists = _launched(fake)
    for k, g in enumerate(grids):
        ni, nj, nk, nabs = g
        of = {q: it[it[:, 4] == k] for q, it in lists.items()}
        none = np.zeros((0, 6), np.int32)
        lean = of.get(fakecuda.LEAN, none)
        general = of.get(fakecuda.GEN_VEL, none)
        assert np.array_equal(general, of.get(fakecuda.GEN_STR, none))
        parts = [_covered(lean[lean[:, 5] == p], g) for p in (0, 1)]
        assert np.array_equal(*parts)
        assert np.all(parts[0] + _covered(general, g) == 1)
        for i0, j0, z0, _ in lean[:, :4]:
            assert nabs[0] <= i0 <= ni - nabs[1] - TILE_X
            assert nabs[2] <= j0 <= nj - nabs[3] - TILE_Y and z0 - LFD >= nabs[4]
        whole = max(sum(nabs[0] <= i <= ni - nabs[1] - TILE_X for i in range(0, ni, TILE_X)), 0) * \
            ((nj - nabs[2] - nabs[3]) // TILE_Y) * (nk - nabs[4])
        want = whole * TILE_X * TILE_Y if plain and nk - nabs[4] >= 8 else 0
        assert parts[0].sum(dtype=np.int64) == want
    (b or solvers[0]).close()


@pytest.mark.parametrize("grid,lists", [((28, 24, 20), 1), ((200, 160, 90), 10)])
def test_autotuner_times_a_list_once(fake, grid, lists):
    """On a small grid most shapes cut the same items.  (lists: at least so many
    different ones.)"""
    m = _model(*grid, nabs=(4, 4, 4, 4, 4, 0))
    s = cgfd.Solver(m.desc())
    m.load(s)
    s.prepare()
    fake.fake_clear_launches()
    s.autotune(steps=1)
    # a captured step is four stages, each with the launches of its lists; four
    # steps are captured per shape
    runs = [(fake.fake_list(q), fakecuda.items(fake, q).tobytes())
            for q in range(fake.fake_launches())]
    per = len({k for k, _ in runs})
    shapes = [tuple(runs[k:k + per]) for k in range(0, len(runs), 4 * 4 * per)]
    timed, chosen = shapes[:-1], shapes[-1]
    assert len(timed) == len(set(timed)) >= lists and chosen in timed
    s.close()


@pytest.mark.parametrize("kernel", [cgfd.KERNEL_FUSED, cgfd.KERNEL_SCALAR])
@pytest.mark.parametrize("sms,split", [(148, True), (16, False)])
def test_traction_image_is_split_where_it_does_not_fill_the_device(fake, kernel, sms, split):
    """A thread per component below eight blocks per SM of the device in use:
    3 * 24 * 3 blocks of this grid."""
    fake.fake_sms(sms)
    m = _model(ni=96, nj=96)
    s = cgfd.Solver(m.desc(kernel=kernel))
    m.load(s)
    s.prepare()
    assert fake.fake_grid_z(b"timg_split_kernel") == (9 if split else -1)
    assert fake.fake_grid_z(b"timg_kernel") == (-1 if split else 3)
    s.close()
