"""Macrocell ranges and majorants of volumes whose rows are read as vectors (x
extent a multiple of 8): one macrocell a row, rows that end inside and beyond
a warp's 32 macrocells, and ragged y and z extents, against the oracle."""
import numpy as np
import pytest

import oracle
from barney_b200 import synth
from tests.helpers import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "u8", "u16", "f16", "bf16"])
@pytest.mark.parametrize("shape", [(2, 2, 8), (9, 17, 16), (17, 33, 248), (10, 9, 256), (19, 8, 264), (3, 25, 520), (40, 2, 24)])
def test_vector_rows(dtype, shape):
    import barney_b200 as bn
    rng = np.random.default_rng(sum(shape))
    f = rng.random(shape).astype(np.float32)
    if dtype == "f32":  # signed zeros and infinities are ordinary scalars
        f[rng.random(shape) < 0.02] = -0.0
        f[0, 0, 0], f[-1, -1, -1] = np.inf, -np.inf
    vol = synth.to_storage(f, dtype)
    d = synth.scene(vol, dtype, 8, 8, synth.tf_knots(256, 1), 50.0, synth.DEFAULT_CAMERA)
    r = bn.VolumeRenderer(d)
    ranges, maj = r.macrocells()
    r.close()
    sc = oracle.Scene(d)
    o_ranges = oracle.build_ranges(sc)
    # values: the sign of a zero minimum depends on the order of comparison
    assert np.array_equal(ranges, o_ranges)
    assert_bitexact(maj, oracle.map_majorants(sc, o_ranges), "majorants")
