"""Tensor path at the edges of its tiles: widths around a strip (128 S positions) and a half (S / 2
positions a thread), bands of one and few rows (blocks of 16 / S steps that end early), zero windows,
and maps large enough for 8-bit _Norm scores that lie next to an FP32 rounding boundary (about one in
2^14 is decided by the full FP64 chain)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MEAS = ["SqrDistance", "SqrDistance_Norm", "CrossCorr", "CrossCorr_Norm"]


def both(ocip, ctx, m, S, T, dtype=np.float32, band=0):
    ctx.make_current()
    ctx.set_path(ocip.PATH_PLAIN)
    plain = ocip.match(m, S, T, dtype)
    ctx.set_path(ocip.PATH_TENSOR)
    ctx.set_band_height(band)
    try:
        got = ocip.match(m, S, T, dtype)
        assert ctx.last_path() == ocip.PATH_TENSOR
    finally:
        ctx.set_band_height(0)
        ctx.set_path(ocip.PATH_PLAIN)
    return plain, got


@pytest.mark.parametrize("th", [16, 32, 64])
@pytest.mark.parametrize("dw", [-1, 0, 1, 3])
@pytest.mark.parametrize("band", [0, 1, 7])
def test_u8_edges_equal_plain(ocip, ctx, th, dw, band):
    strip = 128 * (128 // th)
    rng = np.random.default_rng(th + 10 * dw + band)
    S = rng.integers(0, 256, (th + 5, strip + dw), dtype=np.uint8)
    S[:, : strip // 4] = 0  # windows without energy
    T = rng.integers(0, 256, (th - 1, 23), dtype=np.uint8)
    for m in MEAS:
        for dtype in (np.float32, np.float64):
            plain, got = both(ocip, ctx, m, S, T, dtype, band)
            assert np.array_equal(plain, got, equal_nan=True), (m, dtype)


@pytest.mark.parametrize("th", [12, 32, 64])
@pytest.mark.parametrize("H", [190, 255, 700])
def test_u8_tall_bands_equal_plain(ocip, ctx, th, H):
    """One band: its blocks go round the ring of sums in tensor memory (32 blocks of 2, 4 or 8 rows)
    up to ten times."""
    rng = np.random.default_rng(th + H)
    S = rng.integers(0, 256, (H, 300), dtype=np.uint8)
    T = rng.integers(0, 256, (th, 31), dtype=np.uint8)
    for m in MEAS:
        plain, got = both(ocip, ctx, m, S, T, np.float32, H)
        assert np.array_equal(plain, got, equal_nan=True), m


@pytest.mark.parametrize("th,tw", [(17, 17), (40, 48), (64, 64)])
def test_u8_norm_rounding_equals_plain(ocip, ctx, th, tw):
    rng = np.random.default_rng(th)
    S = rng.integers(0, 256, (900, 1100), dtype=np.uint8)
    T = np.clip(S[300:300 + th, 400:400 + tw] + rng.integers(-8, 9, (th, tw)), 0, 255).astype(np.uint8)
    for m in ("SqrDistance_Norm", "CrossCorr_Norm"):
        plain, got = both(ocip, ctx, m, S, T)
        assert np.array_equal(plain, got, equal_nan=True)


@pytest.mark.parametrize("dtype", [np.float32, np.uint16])
@pytest.mark.parametrize("th,tw,nch", [(16, 64, 1), (31, 31, 1), (64, 64, 1), (33, 9, 3)])
def test_split_edges_within_bar(ocip, ctx, dtype, th, tw, nch):
    """1e-5 of the scale of the terms, per output, against the exact oracle."""
    R = 16 if th <= 16 else 32 if th <= 32 else 64
    rng = np.random.default_rng(th + tw)
    shape = (th + 9, 128 * (128 // R) + 5) + ((nch,) if nch > 1 else ())
    S = rng.random(shape)
    S = (S * 65535).astype(np.uint16) if dtype == np.uint16 else S.astype(np.float32)
    T = S[4:4 + th, 6:6 + tw].copy()
    for m in MEAS:
        for band in (0, 1, 5):
            _, got = both(ocip, ctx, m, S, T, np.float32, band)
            ex = O.proximity_exact(["SqrDistance", "SqrDistance_Norm", "AbsDistance", "CrossCorr",
                                    "CrossCorr_Norm"].index(m), S, T)
            ss, _, tt = O.window_terms_exact(S, T)
            tt = tt if S.ndim == 3 else tt[0]
            scale = np.abs(ex)
            if m.startswith("Sqr"):
                scale = ss + tt
                if m.endswith("_Norm"):
                    scale = scale / np.sqrt(ss * tt)
            assert np.max(np.abs(got - ex) / scale) <= 1e-5, (m, band)
