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
