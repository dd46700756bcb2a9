"""cospdnn_prune_compact at the edges of its chunks, slices and vector paths,
against numpy (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("hilo", [False, True])
@pytest.mark.parametrize("batch,neuron,keep,offset", [
    (1, 1, 1.0, 0),        # one value
    (127, 63, 0.5, 0),     # no vector loads, rows short of a slice
    (1024, 65, 0.0, 0),    # nothing kept, a row past a slice
    (1025, 8, 1.0, 0),     # a column past a chunk, all kept
    (2052, 130, 0.9, 1),   # vector loads, an output that is not aligned
    (5003, 33, 0.3, 0),    # several chunks, odd batch
])
def test_prune_edges(batch, neuron, keep, offset, hilo):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    rng = np.random.default_rng(batch)
    c = rng.random((neuron, batch)).astype(np.float32) + np.float32(0.001)
    c[rng.random((neuron, batch)) < 0.5] = 0.0
    alive = rng.random(batch) < keep
    c[rng.integers(0, neuron, batch), np.arange(batch)] = 1.0 / 3.0  # at least one output above the threshold
    c[:, ~alive] = np.float32(1e-5)  # exactly at it: pruned
    ids = np.nonzero(alive)[0]
    pad = (batch + 127) // 128 * 128
    dt = torch.float16 if hilo else torch.float32
    buf = torch.full((offset + (2 if hilo else 1) * neuron * pad,), 7.0, dtype=dt, device="cuda")
    map_in = torch.arange(batch, dtype=torch.int32, device="cuda") * 3
    cat, mo = (torch.full((batch,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(cs.prune_workspace_bytes(batch), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        cs.prune_compact(torch.from_numpy(c).cuda(), neuron, batch, 1e-5, buf[offset:], cat, map_in, mo, cnt, ws,
                         flags=cs.PRUNE_OUT_HALF_HILO if hilo else 0)
    torch.cuda.synchronize()
    n = int(cnt.item())
    assert n == len(ids)
    np.testing.assert_array_equal(cat.cpu().numpy()[:n], ids)
    np.testing.assert_array_equal(mo.cpu().numpy()[:n], 3 * ids)
    stride = (n + 127) // 128 * 128
    planes = 2 if hilo else 1
    got = buf.cpu().numpy()[offset:offset + planes * neuron * stride].reshape(planes, neuron, stride)
    want = np.zeros((neuron, stride), np.float32)
    want[:, :n] = c[:, ids]
    if hilo:
        hi = want.astype(np.float16)
        np.testing.assert_array_equal(got[0], hi)
        np.testing.assert_array_equal(got[1], (want - hi.astype(np.float32)).astype(np.float16))
    else:
        np.testing.assert_array_equal(got[0], want)
