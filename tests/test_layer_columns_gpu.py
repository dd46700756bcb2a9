"""cospdnn_layer with 16x16 blocks at the edges of its column chunks, block
counts and alignments, against the FP64 product (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("a_float,b_float", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("neuron,batch,counts,shift", [
    (32, 1, (1, 2), 0),          # one column
    (48, 129, (0, 1, 5), 0),     # an empty block column, one column past a CTA
    (64, 4 * 700, (2, 3, 4, 2), 0),   # few CTAs: one column per thread
    (4096, 513, (2,), 0),        # four columns per thread, a column past a chunk, odd rows
    (4096, 516, (3, 1), 0),      # vector loads
    (4096, 516, (2, 4), 1),      # a batch of four columns whose data is not aligned
    (2048, 16388, (2, 5), 0),    # several chunks per CTA
])
def test_columns_match_fp64(neuron, batch, counts, shift, a_float, b_float):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    rng = np.random.default_rng(neuron + batch)
    nbc = neuron // 16
    n = np.array([counts[i % len(counts)] for i in range(nbc)])
    cp = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    # starts up to the end of the matrix: weight rows past it are skipped
    start = rng.integers(0, neuron - 3, cp[-1]).astype(np.int32)
    v = (rng.integers(-8, 9, (cp[-1], 16, 16)) / 64).astype(np.float32)
    fuse = rng.permutation(neuron).astype(np.int32)
    x = torch.rand((neuron, batch), generator=torch.Generator().manual_seed(1), dtype=torch.float32) * 4
    if a_float:
        a, xd = x, x.double()
    else:
        hi = x.half()
        lo = (x - hi.float()).half()
        a, xd = torch.cat([hi, lo]), hi.double() + lo.double()
    dev = lambda t: torch.as_tensor(t).cuda()
    buf = torch.empty(a.numel() + shift, dtype=a.dtype, device="cuda")
    buf[shift:] = a.reshape(-1).cuda()
    out = torch.full((neuron, batch), -1.0, device="cuda")
    b = dev(v) if b_float else dev(v).half()
    flags = (cs.LAYER_A_FLOAT if a_float else 0) | (cs.LAYER_B_FLOAT if b_float else 0)
    cs.layer(buf[shift:], b, out, dev(fuse), dev(cp), dev(start), -0.25, batch, neuron, flags=flags)
    torch.cuda.synchronize()
    want = torch.zeros((neuron, batch), dtype=torch.float64, device="cuda")
    size = torch.zeros_like(want)  # sum of |terms|
    xd, vd, fd = xd.cuda(), dev(v).double(), dev(fuse).long()
    for c in range(nbc):
        for q in range(cp[c], cp[c + 1]):
            r = np.arange(start[q], min(neuron, start[q] + 16))
            w = vd[q][:, :len(r)]
            y = xd[fd[torch.as_tensor(r).cuda()]]
            want[16 * c:16 * c + 16] += w @ y
            size[16 * c:16 * c + 16] += w.abs() @ y.abs()
    want = (want - 0.25).clamp(0, 32)
    # one rounding per term and for the bias, each at most 2^-24 of the terms' sum
    terms = 16 * max(counts) + 2
    assert bool((torch.abs(out.double() - want) <= terms * 2.0 ** -24 * (size + 0.25)).all())
