"""FP64 form of the plain path on both of its tiles, at their edges: 256 x 16 (template rows too many for
two CTAs of the other on an SM), 256 x 8 (few rows, or an image of a few tiles), and a template too wide
for the tall tile on an image that would take it."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MEAS = ["SqrDistance", "SqrDistance_Norm", "AbsDistance", "CrossCorr", "CrossCorr_Norm"]

# (width, height, template width, template height): 1025 x 449 has 145 tiles of 256 x 16, 285 of 256 x 8.
TALL = [(1025, 449, 5, 60), (1025, 449, 24, 45), (1024, 448, 8, 64)]
LOW = [(1025, 449, 23, 12), (257, 33, 17, 17), (255, 9, 40, 9)]


@pytest.mark.parametrize("W,H,tw,th", TALL + LOW)
def test_f64_equals_reference(ocip, plain, W, H, tw, th):
    rng = np.random.default_rng(W + th)
    S, T = rng.random((H, W)) - 0.25, rng.random((th, tw)) - 0.25
    for m, name in enumerate(MEAS):
        want = O.proximity_refexact(m, S, T, fused=True)
        assert np.array_equal(ocip.match(name, S, T), want, equal_nan=True), name


@pytest.mark.parametrize("W,H,tw,th", TALL + LOW)
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int16])
def test_integers_equal_exact_sums(ocip, plain, W, H, tw, th, dtype):
    rng = np.random.default_rng(H + tw)
    info = np.iinfo(dtype)
    S = rng.integers(info.min, info.max + 1, (H, W), dtype=dtype)
    T = rng.integers(info.min, info.max + 1, (th, tw), dtype=dtype)
    for m in (0, 2, 3):
        want = O.proximity_exact(m, S, T).astype(np.float32)
        assert np.array_equal(ocip.match(MEAS[m], S, T), want), MEAS[m]


def test_template_too_wide_for_the_tall_tile(ocip, plain):
    rng = np.random.default_rng(1)
    S = rng.integers(0, 65536, (208, 1500), dtype=np.uint16)
    T = rng.integers(0, 65536, (17, 1430), dtype=np.uint16)
    rows = [0, 100, 207]
    want = O.proximity_exact_rows(3, S, T, rows).astype(np.float32)
    assert np.array_equal(ocip.match("CrossCorr", S, T)[rows], want)
