"""16-bit storage: the order in which the velocity equations add the three
directions' products (cells of Geom::kx0..ky1 contract the sums, the others
round each product first) belongs to the cell, not to the tile or the item list
that computes it.  A 16-bit run follows its roundings, so the fields are held
to the bit: CRC-32 sums of the nine fields after eight steps (each of the four
stencil patterns twice), recorded from the kernels with tiles of 64 x 4 cells
that brought the order in.  The grids: rows of the range that fill no tile of
eight, too few planes above the bottom layer for lean items, a flat model, and
one where range and tiles end together."""
import zlib

import numpy as np
import pytest

import cases
import cgfd
import models

pytestmark = pytest.mark.gpu

STORES = {"f16": cgfd.STORE_F16, "bf16": cgfd.STORE_BF16}
LAYERS = (8, 0, 4, 4, 4, 0)


def _hill(nj, nk):
    return models.gaussian_hill(ni=160, nj=nj, nk=nk, nt=8, dz_top=60.0, dz_bot=120.0,
                                hill_h=200.0, hill_w=600.0, con_depth=400.0, src_depth=300.0,
                                corr_len=200.0, nabs=LAYERS, f0=0.08, t0=0.25, n_side=2,
                                rcv_spacing=300.0)


MODELS = {
    "rows_past_tiles": lambda: _hill(28, 20),
    "shallow": lambda: _hill(28, 11),
    "flat": lambda: models.small_flat(ni=160, nj=28, nk=20, nt=8, nabs=LAYERS),
    "ends_agree": lambda: _hill(24, 20),
}


def fields_crc(m, storage, batch=False):
    """The fields of one model, alone or as the first of two in a batch (whose
    kernels are compilations of their own, with roundings of their own)."""
    init = cases.random_fields(m, 17)
    init[3:] *= 8  # steps that change V by much more than a rounding of it
    b = cgfd.Batch([m.desc(storage=storage)] * 2) if batch else None
    solvers = b.models if batch else [cgfd.Solver(m.desc(storage=storage))]
    for s in solvers:
        m.load(s)
        if storage == cgfd.STORE_F16:  # the fields' magnitudes, not the source's
            s.set_field_scales([0] * 3 + [17] * 6)
        for c in range(9):
            s.set_field(c, init[c])
    (b if batch else solvers[0]).step(8)
    out = [zlib.crc32(np.ascontiguousarray(solvers[0].get_field(c)).tobytes()) for c in range(9)]
    (b if batch else solvers[0]).close()
    return out


RECORDED = {
    ("rows_past_tiles", "f16", "alone"): (0xe1ce0196, 0x4b0227f2, 0x080383c1, 0x7cf3bf2b, 0x4f90dd80,
        0xa584c578, 0x01ff6e9d, 0x72d0821a, 0xeb855249),
    ("rows_past_tiles", "f16", "batch"): (0x9341f7ee, 0x175d393f, 0x79a80bda, 0x6b515cda, 0xb6ac735b,
        0xeb22c102, 0x6e56c319, 0x821b9380, 0x18201749),
    ("rows_past_tiles", "bf16", "alone"): (0xb2725f64, 0x11899224, 0x0e661d56, 0xacb25533, 0x1a83e291,
        0x00d3064a, 0xead53fce, 0x2f6c68c3, 0x9df6ebf7),
    ("rows_past_tiles", "bf16", "batch"): (0xb2725f64, 0x11899224, 0x0e661d56, 0xacb25533, 0x1a83e291,
        0x00d3064a, 0xead53fce, 0x2f6c68c3, 0x9df6ebf7),
    ("shallow", "f16", "alone"): (0x76fb4f4f, 0x64411da0, 0x5cc54f4d, 0xe7bbc521, 0x5a0f5c71,
        0xbd0845ae, 0xa3643b88, 0x89cc3def, 0x9c92dee3),
    ("shallow", "f16", "batch"): (0xce04ff17, 0x79f35da0, 0xec876957, 0xb3ed32bd, 0x24f7c8e3,
        0xd700f82b, 0x4851a2c6, 0x73a80605, 0x17b2ac3e),
    ("shallow", "bf16", "alone"): (0x7174d0dc, 0x4455814a, 0xf92f93c8, 0xbc3ca7a4, 0x633f8389,
        0xb4be75ee, 0xc1bf9eab, 0x1b63a30c, 0xc2fbe9d7),
    ("shallow", "bf16", "batch"): (0x3b44d8ca, 0x47deca43, 0x5d6a7898, 0x5202d28a, 0x72c3e633,
        0x619ea80d, 0x92ca39f3, 0x2d6974f3, 0x3f5dde42),
    ("flat", "f16", "alone"): (0xf3cc06cc, 0xa722379d, 0xec566b7e, 0xaecee29e, 0x12dfc6e6,
        0xa063d3a0, 0xb40bc5bf, 0x63a136a9, 0x3283c7b7),
    ("flat", "f16", "batch"): (0xb5031a40, 0xcb502df7, 0x3669b5a6, 0x7b86cd77, 0x1eb909ed,
        0x19a22fbc, 0x3895594b, 0x75dda73b, 0x5399c9ff),
    ("flat", "bf16", "alone"): (0x9c4d03e7, 0xf91ec35a, 0x3e587cc9, 0xfd6d3a92, 0xad603d16,
        0xf243e7d8, 0x3a620d30, 0x626b9a4b, 0x44761a81),
    ("flat", "bf16", "batch"): (0xe415675d, 0x4ff182af, 0xcb68bb0a, 0xd5417bdd, 0x5f0f127e,
        0x670f3846, 0x4efd8527, 0xcd7487fb, 0x154df4c6),
    ("ends_agree", "f16", "alone"): (0x5a36979b, 0x4a49afd9, 0x61d32685, 0x4495966f, 0xe92964c9,
        0x3506ff11, 0xf83694ed, 0x74637907, 0x459978ea),
    ("ends_agree", "f16", "batch"): (0x757b1293, 0x2259e056, 0x61d32685, 0x57c54b91, 0xe92964c9,
        0x3506ff11, 0x2dff61ec, 0x74637907, 0x3d607b98),
    ("ends_agree", "bf16", "alone"): (0x2d196da8, 0xeb8947c8, 0xc6c060c1, 0xafa21c24, 0xee9ea082,
        0x65262b26, 0xc1941a71, 0xf7210615, 0xdc0f106d),
    ("ends_agree", "bf16", "batch"): (0x2d196da8, 0xeb8947c8, 0xc6c060c1, 0xafa21c24, 0xee9ea082,
        0x65262b26, 0xc1941a71, 0xf7210615, 0xdc0f106d),
}


@pytest.mark.parametrize("name,store,how", list(RECORDED))
def test_rounding_order_belongs_to_the_cell(name, store, how):
    got = fields_crc(MODELS[name](), STORES[store], how == "batch")
    want = RECORDED[name, store, how]
    assert [cgfd.COMPONENTS[c] for c in range(9) if got[c] != want[c]] == []
