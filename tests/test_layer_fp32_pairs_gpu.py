"""cospdnn_layer on FP32 data at batches that take two columns per thread in few
registers: a column pair past a round of CTAs, batches that are no multiple of 4,
several chunks per CTA, zero to five blocks per column (GPU)."""
import pytest

from test_layer_columns_gpu import test_columns_match_fp64 as columns_match_fp64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b_float", [True, False])
@pytest.mark.parametrize("neuron,batch,counts,shift", [
    (4096, 514, (2,), 0),
    (4096, 1542, (2, 3), 0),
    (1024, 2306, (2,), 0),
    (1024, 2432, (0, 1, 5), 0),
    (1024, 6918, (4, 2), 2),     # aligned for pairs only
    (256, 28426, (2, 1), 0),
])
def test_fp32_pairs_match_fp64(neuron, batch, counts, shift, b_float):
    columns_match_fp64(neuron, batch, counts, shift, True, b_float)
