"""cospdnn_layer with weights on rows past the matrix (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def run(a, v, fuse, cp, start, batch, neuron, flags, shift=0):
    import cospdnn_b200 as cs
    buf = torch.empty(a.numel() + shift, dtype=a.dtype, device="cuda")
    buf[shift:] = a.reshape(-1).cuda()
    out = torch.full((neuron, batch), -1.0, device="cuda")
    dev = lambda t: torch.as_tensor(t).cuda()
    cs.layer(buf[shift:], dev(v), out, dev(fuse), dev(cp), dev(start), 0.0, batch, neuron, flags=flags)
    torch.cuda.synchronize()
    return out.cpu()


def need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# one, two and four columns per thread; batches that are no multiple of 8 or not aligned
BATCHES = [(64, 1, 0), (64, 219, 0), (64, 700, 0), (4096, 1021, 0), (4096, 1028, 0), (4096, 4097, 0), (1024, 520, 1)]


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("a_float,reference", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("neuron,batch,shift", BATCHES + [(64, 512, 0), (4096, 1024, 0)])
def test_rows_past_the_matrix_are_skipped(neuron, batch, shift, a_float, reference, bad):
    """Whatever the weights on them."""
    need_gpu()
    import cospdnn_b200 as cs
    nbc = neuron // 16
    v = np.zeros((2 * nbc, 16, 16), np.float16)
    at = v.transpose(0, 2, 1) if not reference else v
    at[:, 0, :] = 0.5
    at[0::2, 5:, :] = bad
    cp = (2 * np.arange(nbc + 1)).astype(np.int32)
    start = np.where(np.arange(2 * nbc) % 2 == 0, neuron - 5, 7).astype(np.int32)
    x = torch.arange(batch).remainder(31).float().expand(neuron, batch)
    a = x.contiguous() if a_float else torch.cat([x, torch.zeros_like(x)]).half()
    flags = (cs.LAYER_A_FLOAT if a_float else 0) | (cs.LAYER_REFERENCE_ARITH if reference else 0)
    got = run(a, v, np.arange(neuron, dtype=np.int32), cp, start, batch, neuron, flags, shift)
    assert torch.equal(got, x.clamp(0, 32))
