"""The stage kernels' work lists and the launch plan around them, on a CUDA
runtime that lives on the host (tests/fakecuda): no GPU, no kernel runs."""
import numpy as np
import pytest

import cgfd
import fakecuda
import models

cudaErrorMemoryAllocation = 2


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    path = fakecuda.build(str(tmp_path_factory.mktemp("fakecuda")))
    if path is None:
        pytest.skip("nvcc and g++ are needed")
    return fakecuda.lib(path)


@pytest.fixture
def fake(fake_lib, monkeypatch):
    fake_lib.fake_reset()
    monkeypatch.setattr(cgfd, "_lib", fake_lib)
    return fake_lib


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
        assert out.setdefault(h.fake_list(q), it) == it
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
    assert _launched(fake) == before
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
