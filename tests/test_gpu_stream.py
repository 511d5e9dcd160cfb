"""The streaming kernel's branches per pass (1, 2, 4, 8 column sets in one launch, several passes of an
expert) and host rows in one or several pieces, against the CPU oracle."""
import numpy as np
import pytest

from tests.test_gpu_grouped import rand_qt
from tests.util import max_rel_err, upload_qt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,gs,half", [(4, 32, True), (4, 64, False), (2, 0, False), (7, 0, False)])
@pytest.mark.parametrize("D,I,rows", [
    (256, 128, [1, 4, 5, 8]),
    (256, 128, [8, 1, 9, 3, 1, 1, 2]),               # one expert above 8 rows: two passes
    (384, 256, [16, 17, 3, 32, 8, 33, 12]),          # every width in one launch
    (4096, 128, [3, 9, 4]),                          # host rows in one piece: up to 512 KB, 32 rows of 16 KB
    (4096, 128, [5, 9, 3]),
    (4096, 128, [20, 1, 11]),                        # exactly one
    (4096, 128, [20, 1, 12]),                        # and a second one of a single row
    (4096, 128, [400, 3, 197]),                      # 9.8 MB: sixteen pieces above 512 KB
])
def test_uneven_group(be, oracle, fmt, gs, half, D, I, rows):
    rng = np.random.default_rng(D + sum(rows) + fmt)
    ex = [(rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, I, D, fmt, gs, half=half), rand_qt(rng, D, I, fmt, gs, half=half))
          for _ in rows]
    hs = [[upload_qt(be, t) for t in e] for e in ex]
    x = ((rng.random((sum(rows), D)) - 0.5) * 2).astype(np.float32)
    be.set_tensor_core(0)
    ok, y = be.run_expert_group([h[0] for h in hs], [h[1] for h in hs], [h[2] for h in hs], rows, x, D)
    be.set_tensor_core(1)
    assert ok and be.kernel_status(0) == 0
    off = 0
    for e, r in zip(ex, rows):
        assert max_rel_err(y[off:off + r], oracle.expert_mlp(x[off:off + r], *e)) <= 1e-3
        off += r
    for h in hs:
        for t in h:
            be.tensor_free(t)


# 16 KB of x a row: pulled by a kernel; one piece; five and ten pieces of 512 KB; sixteen larger ones (above 8 MB)
@pytest.mark.parametrize("S", [1, 17, 130, 300, 512, 513, 600])
def test_matmul_rows_in_pieces(be, S):
    I, O = 4096, 4128
    rng = np.random.default_rng(S)
    t = rand_qt(rng, O, I, 2, 0)
    h = upload_qt(be, t)
    w = t.dequant().astype(np.float64)
    x = rng.standard_normal((S, I)).astype(np.float32)
    ok, y = be.run_matmul([h], x, None, None, 2, I, O, gs=0)
    assert ok
    mag = np.abs(x).astype(np.float64) @ np.abs(w).T
    assert np.all(np.abs(y - x.astype(np.float64) @ w.T) <= 2e-6 * mag + 1e-30)
    be.tensor_free(h)
