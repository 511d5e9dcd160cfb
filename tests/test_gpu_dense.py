"""Row-major quantised matmul (k_dense_mma) against a float64 product with the dequantised weights:
every format, rows that start at any byte, contractions that end inside a 128-column block, output counts
around the 32-row tile and row counts around the 4-row column sets."""
import numpy as np
import pytest

from colibri_b200.quant import QTensor, quantize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,gs", [(1, 0), (2, 0), (3, 0), (4, 32), (4, 64), (4, 96), (4, 48), (7, 0), (8, 0)])
@pytest.mark.parametrize("I,O", [(16, 1), (128, 31), (130, 33), (272, 64), (1030, 70), (2048 + 16, 160), (77, 5)])
def test_formats_and_shapes(be, fmt, gs, I, O):
    if fmt == 7:
        I = -(-I // 32) * 32               # the container format's own limit
    rng = np.random.default_rng(fmt * 1000 + I + O + gs)
    if fmt == 3:                       # 2-bit codes: value code - 2, four per byte
        codes, sc = rng.integers(0, 4, (O, I)), rng.random(O).astype(np.float32)
        pad = np.zeros((O, -(-I // 4) * 4), np.int64)
        pad[:, :I] = codes
        packed = sum(pad[:, j::4] << (2 * j) for j in range(4)).astype(np.uint8)
        t, w = QTensor(packed, sc, 3, I, O), (codes - 2.0) * sc[:, None].astype(np.float64)
    else:
        t = quantize((rng.standard_normal((O, I)) * 0.02).astype(np.float32), fmt, gs)
        w = t.dequant().astype(np.float64)
    for S in (1, 4, 5, 8, 13, 17, 33):
        x = rng.standard_normal((S, I)).astype(np.float32)
        box = [None]
        ok, y = be.run_matmul(box, x, t.w, t.s, fmt, I, O, gs=gs)
        assert ok
        be.tensor_free(box[0])
        mag = np.abs(x).astype(np.float64) @ np.abs(w).T
        assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30), (S, fmt)
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt", [1, 8])
@pytest.mark.parametrize("I", [1, 3, 15, 17, 63, 66, 127, 250])
def test_runs_of_bytes_that_start_anywhere(be, fmt, I):
    """Byte rows of odd lengths: every start of a row within a word, runs of 16 that end inside one, and a last row that ends with
    the tensor. Same bound as above."""
    rng = np.random.default_rng(fmt * 1000 + I)
    t = quantize((rng.standard_normal((37, I)) * 0.02).astype(np.float32), fmt, 0)
    w = t.dequant().astype(np.float64)
    for S in (1, 8, 9):
        x = rng.standard_normal((S, I)).astype(np.float32)
        box = [None]
        ok, y = be.run_matmul(box, x, t.w, t.s, fmt, I, 37, gs=0)
        assert ok
        be.tensor_free(box[0])
        mag = np.abs(x).astype(np.float64) @ np.abs(w).T
        assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30), S
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt,gs,I", [(1, 0, 272), (1, 0, 130), (2, 0, 130), (3, 0, 272), (4, 64, 192), (7, 0, 160), (8, 0, 272), (8, 0, 130)])
def test_more_tiles_than_sms(be, fmt, gs, I):
    """More than 8 rows over 151 tiles of 32 outputs: the instance for two CTAs per SM. Same bound as above."""
    O, S = 4805, 11
    rng = np.random.default_rng(fmt * 1000 + I)
    if fmt == 3:
        codes, sc = rng.integers(0, 4, (O, I)), rng.random(O).astype(np.float32)
        packed = sum(codes[:, j::4] << (2 * j) for j in range(4)).astype(np.uint8)
        t, w = QTensor(packed, sc, 3, I, O), (codes - 2.0) * sc[:, None].astype(np.float64)
    else:
        t = quantize((rng.standard_normal((O, I)) * 0.02).astype(np.float32), fmt, gs)
        w = t.dequant().astype(np.float64)
    x = rng.standard_normal((S, I)).astype(np.float32)
    box = [None]
    ok, y = be.run_matmul(box, x, t.w, t.s, fmt, I, O, gs=gs)
    assert ok
    be.tensor_free(box[0])
    mag = np.abs(x).astype(np.float64) @ np.abs(w).T
    assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30)
    assert be.kernel_status(0) == 0


@pytest.mark.parametrize("fmt,gs,I", [(1, 0, 272), (1, 0, 130), (2, 0, 130), (3, 0, 272), (4, 64, 192), (7, 0, 160), (8, 0, 272), (8, 0, 130)])
@pytest.mark.parametrize("O,S", [(9601, 4), (14500, 3), (21000, 1), (9601, 9), (14500, 9)])
def test_ctas_that_share_an_sm(be, fmt, gs, I, O, S):
    """Few rows over more tiles than two CTAs per SM hold (three, four, and two waves), and more than 8 rows where three waves of one
    are taken. Same bound as above."""
    rng = np.random.default_rng(fmt * 1000 + I + S)
    if fmt == 3:
        codes, sc = rng.integers(0, 4, (O, I)), rng.random(O).astype(np.float32)
        packed = sum(codes[:, j::4] << (2 * j) for j in range(4)).astype(np.uint8)
        t, w = QTensor(packed, sc, 3, I, O), (codes - 2.0) * sc[:, None].astype(np.float64)
    else:
        t = quantize((rng.standard_normal((O, I)) * 0.02).astype(np.float32), fmt, gs)
        w = t.dequant().astype(np.float64)
    x = rng.standard_normal((S, I)).astype(np.float32)
    box = [None]
    ok, y = be.run_matmul(box, x, t.w, t.s, fmt, I, O, gs=gs)
    assert ok
    be.tensor_free(box[0])
    mag = np.abs(x).astype(np.float64) @ np.abs(w).T
    assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30)
    assert be.kernel_status(0) == 0
