"""Plain path at the edges of each CTA tile (256 x 32, 128 x 16 and 128 x 8 of the FP32 form, 256 x 8 of
the FP64 form): bit-identical to the reference's arithmetic whichever tile a size takes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MEAS = ["SqrDistance", "SqrDistance_Norm", "AbsDistance", "CrossCorr", "CrossCorr_Norm"]

# (width, height): small images take 128 x 8, 700 x 300 takes 128 x 16, 1024 x 1030 256 x 32.
SIZES = [(9, 9), (127, 16), (129, 9), (257, 33), (700, 300), (1024, 1030)]


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("th,tw", [(7, 5), (9, 8), (1, 9)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_float_tiles_equal_reference(ocip, plain, W, H, th, tw, dtype):
    rng = np.random.default_rng(W * 7 + H + th)
    S = (rng.random((H, W)) - 0.25).astype(dtype)
    T = (rng.random((th, tw)) - 0.25).astype(dtype)
    for m, name in enumerate(MEAS):
        want = O.proximity_refexact(m, S, T, fused=True)
        assert np.array_equal(ocip.match(name, S, T), want, equal_nan=True), name


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.uint16])
def test_integer_tiles_equal_exact_sums(ocip, plain, W, H, dtype):
    rng = np.random.default_rng(W + H)
    info = np.iinfo(dtype)
    S = rng.integers(info.min, info.max + 1, (H, W), dtype=dtype)
    T = rng.integers(info.min, info.max + 1, (6, 7), dtype=dtype)
    for m in (0, 2, 3):
        want = O.proximity_exact(m, S, T).astype(np.float32)
        assert np.array_equal(ocip.match(MEAS[m], S, T), want), MEAS[m]
