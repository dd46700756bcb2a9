"""cospdnn_layer on pairs of halves that are no split of one FP32 value, and with
weights on rows past the matrix (GPU)."""
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
BATCHES = [(64, 1, 0), (64, 219, 0), (64, 700, 0), (4096, 1021, 0), (4096, 1028, 0), (4096, 4097, 0), (4096, 2500, 0), (1024, 520, 1)]


@pytest.mark.parametrize("reference", [False, True])
@pytest.mark.parametrize("neuron,batch,shift", BATCHES)
def test_halves_have_a_rounding_each(neuron, batch, shift, reference):
    """-32 and then 32 + lo: what is left is lo, which 32 + lo in FP32 does not hold."""
    need_gpu()
    import cospdnn_b200 as cs
    g = torch.Generator().manual_seed(neuron + batch)
    lo = torch.randint(0, 64, (batch,), generator=g).float() * 2.0 ** -24
    a = torch.zeros((2, neuron, batch))
    a[0, :2] = 32.0
    a[1, 1] = lo
    nbc = neuron // 16
    v = np.zeros((2 * nbc, 16, 16), np.float16)
    at = v.transpose(0, 2, 1) if not reference else v  # [block][input][output]
    at[0::2, 0, :] = -1.0
    at[0::2, 1, :] = 1.0
    cp = (2 * np.arange(nbc + 1)).astype(np.int32)
    start = np.zeros(2 * nbc, np.int32)
    flags = cs.LAYER_REFERENCE_ARITH if reference else 0
    got = run(a.half(), v, np.arange(neuron, dtype=np.int32), cp, start, batch, neuron, flags, shift)
    assert torch.equal(got, lo.expand(neuron, batch))


@pytest.mark.parametrize("neuron,batch,shift", BATCHES)
def test_any_pairs_match_fp64(neuron, batch, shift):
    need_gpu()
    rng = np.random.default_rng(batch)
    nbc = neuron // 16
    counts = np.array([3, 0, 2, 1])[np.arange(nbc) % 4]
    cp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    start = rng.integers(0, neuron - 3, cp[-1]).astype(np.int32)
    v = (rng.integers(-8, 9, (cp[-1], 16, 16)) / 64).astype(np.float16)
    fuse = rng.permutation(neuron).astype(np.int32)
    a = torch.as_tensor(rng.standard_normal((2, neuron, batch)) * np.exp2(rng.integers(-16, 5, (2, neuron, batch)))).half()
    got = run(a, v, fuse, cp, start, batch, neuron, 0, shift).double()
    hi, lo = a.double()
    want, size = torch.zeros((2, neuron, batch), dtype=torch.float64)
    for c in range(nbc):
        for q in range(cp[c], cp[c + 1]):
            r = fuse[np.arange(start[q], min(neuron, start[q] + 16))]
            w = torch.as_tensor(v[q].astype(np.float64))[:, :len(r)]
            want[16 * c:16 * c + 16] += w @ (hi[r] + lo[r])
            size[16 * c:16 * c + 16] += w.abs() @ (hi[r].abs() + lo[r].abs())
    # a rounding per half and weight, each at most 2^-24 of the terms' sum
    assert bool((torch.abs(got - want.clamp(0, 32)) <= (2 * 16 * 3 + 2) * 2.0 ** -24 * size).all())


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
