"""Engines whose networks run on different layer kernels of one precision
(multi-layer tiles, row tiles), against the FP64 oracle (GPU)."""
import numpy as np
import pytest

from netgen import oracle_run
from test_tiles_gpu import layer

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def fading_net(n, k, w, bias, rows, layers, seed):
    """Random inputs whose rows die one after another over the layers."""
    rng = np.random.default_rng(seed)
    csc = [layer(n, k, w, rng) for _ in range(layers)]
    y0 = (rng.random((rows, n)) * rng.uniform(0.05, 0.6, (rows, 1))).astype(np.float32)
    return csc, y0, np.float32(bias)


@pytest.fixture(scope="module")
def nets():
    """(network, rows per tile by precision): a multi-layer tile network with rows
    dying in every layer of its runs, and two whose tiles are as narrow (8192) or
    are sized for fewer neurons (1000) on the row-tile kernel."""
    out = []
    for n, k, w, rows, layers, seed in [(1024, 32, 0.0625, 900, 22, 5), (8192, 24, 0.08, 70, 5, 6),
                                        (1000, 32, 0.0625, 500, 12, 7)]:
        net = fading_net(n, k, w, -0.02, rows, layers, seed)
        out.append((net, oracle_run(*net, want_final=True)))
    return out


@pytest.mark.parametrize("order", [(0, 1), (1, 0), (2, 0, 1), (0, 2)])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_tile_kernels_in_one_engine(nets, prec, order):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    eng = cs.Engine(0)
    for i in order:
        csc, y0, b = nets[i][0]
        nid = eng.add_net(y0.shape[1], len(csc), y0.shape[0], float(b), 1e-5, prec, cs.KERNEL_CUDA_CORE)
        for l, c in enumerate(csc):
            eng.set_layer_csc(nid, l, *c)
    eng.build()
    for _ in range(3):
        for nid, i in enumerate(order):
            eng.set_input(nid, nets[i][0][1])
        eng.run()
        for nid, i in enumerate(order):
            ref, res = nets[i][1], eng.result(nid)
            np.testing.assert_array_equal(res["alive"], ref["alive"])
            np.testing.assert_array_equal(res["categories"], ref["categories"])
            if i == 0 and prec:
                assert res["rechecked"].sum() > 20  # rows in doubt, most of them inside runs of layers
            if len(res["categories"]):
                got = eng.final_values(nid, len(res["categories"])).astype(np.float64)
                assert np.abs(got - ref["final"][ref["categories"]]).max() <= eng.final_bound(nid)
    eng.close()


@pytest.mark.parametrize("with_other", [False, True])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("rows", [50, 600, 900])
def test_dense_networks_change_kernels(nets, prec, rows, with_other):
    """One weight value and up to 300 entries per output: row tiles layer by layer
    while there are few, several layers per launch while there are many."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200 as cs
    dense = fading_net(1024, 300, 0.0066, -0.02, rows, 22, 3)
    todo = [(dense, oracle_run(*dense, want_final=True))] + ([nets[1]] if with_other else [])
    eng = cs.Engine(0)
    for (csc, y0, b), _ in todo:
        nid = eng.add_net(y0.shape[1], len(csc), y0.shape[0], float(b), 1e-5, prec, cs.KERNEL_CUDA_CORE)
        for l, c in enumerate(csc):
            eng.set_layer_csc(nid, l, *c)
    eng.build()
    for step in range(3):
        for nid, ((_, y0, _), _) in enumerate(todo):
            eng.set_input(nid, y0)
        eng.profile_layers() if step == 1 else eng.run()
        for nid, (_, ref) in enumerate(todo):
            res = eng.result(nid)
            np.testing.assert_array_equal(res["alive"], ref["alive"])
            np.testing.assert_array_equal(res["categories"], ref["categories"])
            if len(res["categories"]):
                got = eng.final_values(nid, len(res["categories"])).astype(np.float64)
                assert np.abs(got - ref["final"][ref["categories"]]).max() <= eng.final_bound(nid)
    if rows == 900:  # the others' row tiles are the row-tile kernel's own
        assert eng.net_info(0)["row_tile"] == (8 if prec else 4)
    eng.close()
