"""Sums inside the tensor cores (multi-layer tiles of 16-bit networks) against the
engine's bound, layer by layer and row by row: weights that the compute type
does not hold, inputs over many binades (GPU)."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_tiles_gpu import layer

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n,k,w,span", [
    (1024, 32, 0.07, 20),    # terms from 2^-16 to 2^4
    (1024, 32, -0.3, 4),     # negative sums
    (2064, 200, 0.011, 12),  # many steps, too dense for tiles of few rows: on the row-tile kernel
    (512, 200, 0.011, 12),   # in tiles
    (512, 17, 1.7, 24),
])
def test_layers_within_bounds(n, k, w, span, prec):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    rng = np.random.default_rng(n + k)
    layers, rows = 5, 70
    csc = [layer(n, k, w if l % 2 == 0 else 0.05, rng) for l in range(layers)]
    y0 = np.exp2(rng.uniform(4 - span, 4, (rows, n))).astype(np.float32)
    bias = np.float32(3.0 if w < 0 else -0.013)
    eng = cs.Engine(0)
    eng.add_net(n, layers, rows, float(bias), 1e-5, prec, cs.KERNEL_CUDA_CORE)
    for l, c in enumerate(csc):
        eng.set_layer_csc(0, l, *c)
    eng.build()
    eng.set_input(0, y0)
    kept = 0
    for l in range(layers):
        vals, ids, bounds = eng.layer_values(0, l, bounds=True)
        want = po.replay_fp64(csc, y0, bias, ids.astype(np.int64), l)
        assert (np.abs(vals.astype(np.float64) - want).max(1) <= bounds).all()
        kept += len(ids)
    assert kept >= rows and (n == 2064 or eng.net_info(0)["row_tile"] == 8)
    eng.close()
