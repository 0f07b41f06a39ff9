"""Device buffers kept between calls -- the staging of uploads, downloads and
snapshots (with the solver up to 64 MB, per call above) and the training
gradient's -- on a CUDA runtime that lives on the host (tests/fakecuda)."""
import numpy as np
import pytest

import cgfd

cudaErrorMemoryAllocation, cudaErrorIllegalAddress = 2, 700


CALLS = {
    "set_field": lambda s: s.set_field(0, np.zeros(s.shape, np.float32)),
    "get_field": lambda s: s.get_field(0),
    "snapshot": lambda s: s.snapshot((3, 3, 3), [n - 6 for n in s.shape]),
    "media": lambda s: s.upload_media(*[np.ones(s.shape, np.float32)] * 3),
}


# below and above the size that is kept (a field of 260^3 cells is 70 MB)
@pytest.mark.parametrize("side", [16, 254])
@pytest.mark.parametrize("error,text", [(cudaErrorMemoryAllocation, "out of memory"),
                                        (cudaErrorIllegalAddress, "illegal")])
@pytest.mark.parametrize("call", list(CALLS))
def test_failed_staging_reports_its_cause(fake, call, error, text, side):
    """An earlier kernel's error comes back from the next allocation: it is that
    error the caller is told, not a lack of memory.  The next call works, and
    nothing is lost or freed twice."""
    blocks = fake.fake_blocks()
    s = cgfd.Solver(cgfd.Desc(ni=side, nj=side, nk=side, steph=100.0, stept=0.005, nt=4,
                              con_index=side // 2, hybrid_grid=1))
    fake.fake_fail(b"cudaMalloc", 0, error)
    with pytest.raises(cgfd.CgfdError, match=text) as e:
        CALLS[call](s)
    assert e.value.status == cgfd.ERR_CUDA and fake.fake_last() == 0
    CALLS[call](s)
    CALLS[call](s)
    s.close()
    assert fake.fake_blocks() == blocks


@pytest.mark.parametrize("what,nth", [(b"cudaMalloc", k) for k in range(5)] +
                         [(b"cudaFuncSetAttribute", 0)])
def test_failed_gradient_buffers_are_tried_again(fake, what, nth):
    """A first gradient call on a device that fails part of the way through its
    buffers leaves the next one to finish them (its launch would be refused
    without them)."""
    w = np.zeros(cgfd.MLP_PARAMS, np.float16)
    x, t = np.zeros((300, 45), np.float32), np.zeros((300, 9), np.float32)
    fake.cudaSetDevice(10 + nth + 10 * (what != b"cudaMalloc"))  # one without buffers yet
    blocks = fake.fake_blocks()
    fake.fake_fail(what, nth, cudaErrorMemoryAllocation)
    with pytest.raises(cgfd.CgfdError, match="out of memory"):
        cgfd.mlp_gradient(w, x, t)
    assert fake.fake_last() == 0
    cgfd.mlp_gradient(w, x, t)
    cgfd.mlp_gradient(w, x, t)
    assert fake.fake_blocks() == blocks + 5
