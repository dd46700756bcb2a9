"""The FP64 replay of rows in doubt: what it counts, and every way that it takes,
against the FP64 oracle (GPU)."""
import numpy as np
import pytest

from netgen import oracle_run
from test_mixed_kernels_gpu import fading_net

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def engine(net, prec, tau=1e-5):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    csc, y0, b = net
    eng = cs.Engine(0)
    eng.add_net(y0.shape[1], len(csc), y0.shape[0], float(b), tau, prec, cs.KERNEL_CUDA_CORE)
    for l, c in enumerate(csc):
        eng.set_layer_csc(0, l, *c)
    eng.build()
    eng.set_input(0, y0)
    return eng


def test_rechecks_are_counted_at_their_layer():
    """Runs of several layers per iteration report the layers where doubt began.
    Up to the first such layer they have no other history than layer by layer."""
    net = fading_net(1024, 32, 0.0625, -0.02, 900, 22, 5)
    eng = engine(net, 2)
    eng.run()
    runs = eng.result(0)
    eng.profile_layers()  # one layer per iteration
    single = eng.result(0)
    eng.close()
    np.testing.assert_array_equal(runs["alive"], single["alive"])
    first = np.nonzero(single["rechecked"])[0][0]
    assert runs["rechecked"][:first].sum() == 0
    assert runs["rechecked"][first] == single["rechecked"][first]
    # rows die in all of the layers 2 to 16, the more of them in doubt the later
    assert np.count_nonzero(runs["rechecked"]) >= 5
    alive_in = np.concatenate([[900], runs["alive"][:-1]])
    assert (runs["rechecked"] <= alive_in).all()
