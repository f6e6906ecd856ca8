"""The training step's backward pass over batch sizes that fill one tile, several CTAs, all their tile pipelines and
more than one tile per pipeline. Gradients are sums over records, so a batch's gradient is the sum of its chunks'
(chunks of 1,000 use one pipeline per CTA and are checked against the f64 oracle in test_gpu_guide.py)."""
import numpy as np
import pytest

from rtcuda.guide import Guide, LEVELS, TABLE_ENTRIES

pytestmark = pytest.mark.gpu


def _records(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 16), dtype=np.float32)
    r[:, 0:3] = rng.uniform(-1, 1, size=(n, 3))
    for a in (3, 6, 9):
        v = rng.normal(size=(n, 3))
        r[:, a:a + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    r[:, 12] = rng.uniform(0.1, 2.0, size=n)
    return r


@pytest.mark.parametrize("n", [1, 128, 129, 148 * 128 + 1, 4 * 148 * 128 + 500])
def test_batch_gradient_is_the_sum_of_its_chunks(n):
    g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
    t = np.random.default_rng(9).normal(scale=0.5, size=LEVELS * TABLE_ENTRIES * 2)
    g.set_params(table16=np.float16(t).view(np.uint16))
    rec = _records(n, n)
    raw, loss, gm, gt = g.grads(rec)
    sum_m, sum_t, sum_loss, size_m = 0.0, 0.0, 0.0, 0.0
    for k in range(0, n, 1000):
        raw_c, loss_c, m, tb = g.grads(rec[k:k + 1000])
        assert np.array_equal(raw[k:k + 1000], raw_c)
        sum_m, sum_loss, size_m = sum_m + m.astype(np.float64), sum_loss + loss_c, size_m + np.abs(m)
        sum_t = sum_t + tb.astype(np.float64)
    g.close()
    # f32 sums in another order: every partial sum rounds to 2^-24 of itself, over at most 600 rows and 1,000 records.
    assert (np.abs(gm - sum_m) <= 1e-5 * size_m + 1e-4 * np.abs(sum_m).max()).all()
    assert np.linalg.norm(gm - sum_m) <= 1e-5 * np.linalg.norm(sum_m)
    # The table's sums are integers of 2^-24; each chunk's is rounded to f32 once when it is read.
    assert np.abs(gt - sum_t).max() <= 1e-6 * np.abs(sum_t).max() + 2.0 ** -24
    assert abs(loss - sum_loss) <= 1e-5 * abs(sum_loss) + 1e-5


def test_training_is_reproducible():
    """Two networks trained on the same batches agree bit for bit (no sum depends on the order blocks run in)."""
    out = []
    for _ in range(2):
        g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
        for k in range(3):
            g.train_step(_records(65_536, k))
        out.append(g.params())
        g.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
