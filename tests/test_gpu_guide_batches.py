"""The training step's backward pass over batch sizes that fill one tile, several CTAs, all their tile pipelines and
more than one tile per pipeline. Gradients are sums over records, so a batch's gradient is the sum of its chunks'
(chunks of 1,000 use one pipeline per CTA and are checked against the f64 oracle in test_gpu_guide.py)."""
import ctypes
import zlib

import numpy as np
import pytest
import torch

from rtcuda import guide as guide_mod
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


@pytest.mark.parametrize("n", [5, 300 * 128 + 77, 592 * 128, 592 * 128 + 1, 1500 * 128 + 5])
def test_gradient_keeps_its_order_of_summation(n):
    """Row r of two per SM adds tiles (128 records) r, r + rows, r + 2 rows, ... in turn, then the rows are added in
    turn, in f32: bit for bit what the tiles' own gradients give in that order, over batches of one round of the
    backward pass's pipelines, exactly that, and several."""
    g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
    rec = _records(n, n)
    tiles = [g.grads(rec[k:k + 128], table=False)[2] for k in range(0, n, 128)]
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    want = np.zeros_like(tiles[0])
    for r in range(min(rows, len(tiles))):
        row = tiles[r].copy()
        for t in range(r + rows, len(tiles), rows):
            row += tiles[t]
        want += row
    got = g.grads(rec, table=False)[2]
    g.close()
    assert np.array_equal(got, want)


def test_bias_gradient_is_summed_as_a_weight_of_a_constant_input():
    """A bias is the weight of an input that is always 1: where a unit of the layer below is 1 for every record, its
    weights' gradients and the biases' are the same sums, bit for bit."""
    g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
    mlp, t = g.params()
    table = np.random.default_rng(9).normal(scale=0.5, size=t.size)
    shapes = [(64, 48), (64, 64), (64, 64), (48, 64)]
    w_at = np.cumsum([0] + [a * b for a, b in shapes])
    for lv in range(3):   # unit 5 of every hidden layer: no weights, bias 1
        mlp[w_at[lv]:w_at[lv + 1]].reshape(shapes[lv])[5] = 0.0
        mlp[w_at[4] + 64 * lv + 5] = 1.0
    g.set_params(mlp=mlp, table16=np.float16(table).view(np.uint16))
    rec = _records(40_000, 2)
    rec[:, 3:6] = (1.0, 0.0, 0.0)   # input 32 of the first layer
    gm = g.grads(rec, table=False)[2]
    g.close()
    for lv, unit in enumerate((32, 5, 5, 5)):
        o = shapes[lv][0]
        weights = gm[w_at[lv]:w_at[lv + 1]].reshape(shapes[lv])[:, unit]
        biases = gm[w_at[4] + 64 * lv:w_at[4] + 64 * lv + o]
        assert np.abs(biases).max() > 0
        assert np.array_equal(weights, biases), lv


def test_training_gives_the_recorded_network():
    """Four steps on fixed records give the network recorded here: no change of a kernel's shape may move the order of
    a sum or where a product is rounded."""
    g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
    t = np.random.default_rng(9).normal(scale=0.5, size=LEVELS * TABLE_ENTRIES * 2)
    g.set_params(table16=np.float16(t).view(np.uint16))
    for k in range(4):
        g.train_step(_records(60_000, k))
    mlp, table = g.params()
    g.close()
    assert (zlib.crc32(mlp.tobytes()), zlib.crc32(table.tobytes())) == (1770624645, 2885379321)


def test_inference_writes_any_memory_a_copy_reaches():
    """Outputs in device memory of 16-byte and 4-byte alignment and in pinned host memory: the same values."""
    g = Guide((-1, -1, -1), (1, 1, 1), seed=3)
    n = 5000
    rec = torch.from_numpy(_records(n, 4)).cuda()
    want = g.infer(rec.cpu().numpy())
    device = torch.zeros(n * 48 + 4, device="cuda")
    pinned = torch.zeros(n * 48 + 4, pin_memory=True)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for buf in (device, pinned):
        for at in (0, 1, 4):
            buf.zero_()
            torch.cuda.synchronize()
            guide_mod._check(guide_mod._g().rt_guide_infer_device(g.h, rec.data_ptr(), n, buf[at:].data_ptr(),
                                                                  ctypes.c_void_p(st.cuda_stream)))
            st.synchronize()
            assert np.array_equal(buf[at:at + n * 48].cpu().numpy().reshape(n, 48), want)
            assert (buf[:at] == 0).all() and (buf[at + n * 48:] == 0).all()
    g.close()
