"""Templates of many tiles on the tensor path (12 and 36 tiles of at most 64 x 64: eight maps added at a
time, and three launches whose sums pass through an FP64 map), templates wider than 289 columns with
window energies, and prepared batches with more row-energy planes than one launch takes (65535)."""
import numpy as np
import pytest

import bench

pytestmark = pytest.mark.gpu

MEAS = {"SqrDistance": 0, "SqrDistance_Norm": 1, "CrossCorr": 3, "CrossCorr_Norm": 4}


def tensor_map(ocip, ctx, m, S, T):
    ctx.make_current()
    ctx.set_path(ocip.PATH_TENSOR)
    try:
        got = ocip.match(m, S, T)
        assert ctx.last_path() == ocip.PATH_TENSOR
    finally:
        ctx.set_path(ocip.PATH_PLAIN)
    return got


# (template height, width, image height, width, channels)
SHAPES = [(200, 130, 223, 301, 1), (130, 200, 221, 299, 3), (370, 330, 411, 403, 1)]


@pytest.mark.parametrize("th,tw,H,W,nch", SHAPES)
def test_u8_many_tiles_equal_plain(ocip, ctx, th, tw, H, W, nch):
    rng = np.random.default_rng(th + nch)
    S = rng.integers(0, 256, (H, W, nch) if nch > 1 else (H, W), dtype=np.uint8)
    T = S[7:7 + th, 11:11 + tw].copy()
    for m in MEAS:
        ctx.make_current()
        ctx.set_path(ocip.PATH_PLAIN)
        want = ocip.match(m, S, T)
        assert np.array_equal(tensor_map(ocip, ctx, m, S, T), want, equal_nan=True), m


@pytest.mark.parametrize("dtype", [np.float32, np.uint16])
@pytest.mark.parametrize("th,tw,H,W,nch", SHAPES)
def test_split_many_tiles_within_bar(ocip, ctx, dtype, th, tw, H, W, nch):
    """1e-5 against the long-double oracle (SqrDistance[_Norm]: of the scale of their terms)."""
    planes = [bench.blob_field(W, H, nblobs=30, seed=th + c) for c in range(nch)]
    S = np.stack(planes, -1) if nch > 1 else planes[0]
    if dtype == np.uint16:
        S = (S * (65535 / S.max())).astype(np.uint16)
    T = S[9:9 + th, 13:13 + tw].copy()
    rows = [0, H // 2, H - 1]
    for m, i in MEAS.items():
        e = bench.error_rows(i, S, T, tensor_map(ocip, ctx, m, S, T), rows)
        assert e["max_scaled" if i in (0, 1) else "max_rel"] <= 1e-5, (m, e)


def test_batch_with_more_planes_than_a_grid_dimension(ocip, ctx):
    """512 images of 4 channels, templates 1 to 33 columns wide: 67584 row-energy planes."""
    ctx.make_current()
    rng = np.random.default_rng(3)
    N, H, W = 512, 4, 40
    S = rng.integers(0, 256, (N, H, W, 4), dtype=np.uint8)
    T = [rng.integers(0, 256, (2 + w % 2, w, 4), dtype=np.uint8) for w in range(1, 34)]
    images = [ocip.Image(s) for s in S]
    templates = [ocip.Image(t) for t in T]
    out = np.zeros((N, len(T), H, W, 4), np.float32)
    dests = [ocip.Image(out[i, j]) for i in range(N) for j in range(len(T))]
    batch = ocip.prepare_batch("SqrDistance", images, templates, dests)
    ocip.check(batch.run())
    ctx.set_path(ocip.PATH_PLAIN)
    for i in (0, 255, 496, 511):
        for j in range(len(T)):
            got = dests[i * len(T) + j].read()
            assert np.array_equal(got, ocip.match("SqrDistance", S[i], T[j])), (i, j)
    batch.release()
    for r in images + templates + dests:
        r.release()


@pytest.mark.parametrize("th,tw", [(16, 16), (31, 31), (64, 64), (128, 70)])
def test_dark_area_beside_a_bright_one(ocip, ctx, th, tw):
    """Window energies are running sums down the rows: exact, so that a window of zeros has none, while
    the row energies' exponents lie within 2^29 of one another less log2 of the rows."""
    rng = np.random.default_rng(th)
    H, W = 300, 200
    S = rng.integers(1, 256, (H, W)).astype(np.float32)
    S[100:100 + th + 20] *= 2.0 ** -10   # energies 2^-20 of the rows around
    S[100 + th + 20:280, :100] = 0
    T = S[104:104 + th, 20:20 + tw].copy()
    got = tensor_map(ocip, ctx, "CrossCorr_Norm", S, T)
    rows = sorted({0, 100 + th // 2 + 5, 100 + th + 10, min(299, 120 + th + th), 290, 299})
    e = bench.error_rows(4, S, T, got, rows)
    assert e["max_rel"] <= 1e-5, e
    zero = np.array([[not S[max(0, y - th // 2):y - th // 2 + th, max(0, x - tw // 2):x - tw // 2 + tw].any()
                      for x in range(W)] for y in rows])
    assert np.array_equal(np.isnan(got[rows]), zero)
