"""The multi-layer tile kernel (networks of one weight value per layer)
at the edges of its range, against the FP64 oracle (GPU)."""
import numpy as np
import pytest

from netgen import oracle_run
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def cs():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cospdnn_b200
    cospdnn_b200.lib()
    return cospdnn_b200


def layer(n, k, w, rng):
    """Output j reads U[0, k] random inputs (the first k, the second none), all of weight w."""
    cp, ri = np.zeros(n + 1, np.int32), []
    for j in range(n):
        c = k if j == 0 else 0 if j == 1 else int(rng.integers(0, k + 1))
        ri.append(np.sort(rng.choice(n, size=min(c, n), replace=False)).astype(np.int32))
        cp[j + 1] = cp[j] + len(ri[-1])
    ri = np.concatenate(ri)
    return cp, ri, np.full(len(ri), w, np.float32)


def check(cs, nets, prec):
    """nets: [(csc, y0, bias)].  Per-layer survivors, categories and final values."""
    eng = cs.Engine(0)
    for csc, y0, b in nets:
        nid = eng.add_net(y0.shape[1], len(csc), y0.shape[0], float(b), 1e-5, prec, cs.KERNEL_CUDA_CORE)
        for l, c in enumerate(csc):
            eng.set_layer_csc(nid, l, *c)
    eng.build()
    for rep in range(2):
        for i, (csc, y0, b) in enumerate(nets):
            eng.set_input(i, y0)
        eng.run()
        for i, (csc, y0, b) in enumerate(nets):
            ref = oracle_run(csc, np.nan_to_num(y0), b, want_final=True)
            res = eng.result(i)
            np.testing.assert_array_equal(res["alive"], ref["alive"])
            np.testing.assert_array_equal(res["categories"], ref["categories"])
            if len(res["categories"]):
                got = eng.final_values(i, len(res["categories"])).astype(np.float64)
                assert np.abs(got - ref["final"][ref["categories"]]).max() <= eng.final_bound(i)
    infos = [eng.net_info(i) for i in range(len(nets))]
    eng.close()
    return infos


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n,rows,k,layers", [
    (16, 1, 3, 6),        # one group of outputs, one row
    (48, 9, 16, 20),      # fewer groups than warps, one block of entries, a tile and a row
    (1040, 8, 17, 9),     # an odd number of groups, two blocks, one full tile
    (1024, 1203, 32, 40), # several iterations of growing runs
    (2064, 40, 33, 5),    # two CTAs per SM, three blocks
    (7008, 25, 20, 4),    # nearly the widest tile
    (7024, 6, 40, 3),     # the widest (16-bit)
])
def test_tiles_match_fp64(cs, n, rows, k, layers, prec):
    rng = np.random.default_rng(n * 31 + rows)
    csc = [layer(n, k, 0.0625 if l % 2 else 0.09375, rng) for l in range(layers)]
    y0 = po.input_binary(5, n, rows, n, 0.3, 0.9)
    (info,) = check(cs, [(csc, y0, np.float32(-0.2))], prec)
    if prec or n % 32 == 0:
        assert info["row_tile"] == (8 if prec else 4)


@pytest.mark.parametrize("prec", [0, 1])
def test_tiles_many_networks(cs, prec):
    """More networks than a CTA holds at a time, of several widths and depths."""
    rng = np.random.default_rng(3)
    nets = []
    for i in range(29):
        n = [32, 64, 1024][i % 3] if i < 28 else 2048
        nets.append(([layer(n, 9, 0.125, rng) for _ in range(2 + i % 5)],
                     po.input_binary(7, i, 3 + 5 * i, n, 0.2, 0.8), np.float32(-0.15)))
    check(cs, nets, prec)


def test_tiles_infinite_inputs(cs):
    """An infinite input reaches only the outputs that read it; rows of finite
    inputs are not touched."""
    rng = np.random.default_rng(11)
    n, rows = 1024, 20
    csc = [layer(n, 8, 0.0625, rng) for _ in range(5)]
    y0 = (rng.random((rows, n)) < 0.5).astype(np.float32)
    y0[3, 17] = np.inf
    y0[12, 900] = 1e6  # infinite in FP16
    check(cs, [(csc, y0, np.float32(-0.05))], 1)


def test_tiles_undecided_rows_between_layers(cs):
    """Rows within the error bound of the threshold in the middle of a run of
    layers: re-decided from there, the counts of all layers exact."""
    rng = np.random.default_rng(23)
    n, rows, layers = 512, 64, 30
    csc = [layer(n, 12, 0.1, rng) for _ in range(layers)]
    y0 = (rng.random((rows, n)) * rng.uniform(0.05, 0.6, (rows, 1))).astype(np.float32)
    check(cs, [(csc, y0, np.float32(-0.02))], 2)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n,rows", [
    (1024, 15013),  # four CTAs per SM
    (2064, 7531),   # two
    (4096, 3557),   # one
])
def test_tiles_several_per_cta_after_pruning(cs, n, rows, prec):
    """CTAs that take several tiles of rows that come through the compaction
    map (two networks of one width and one of another, rows dying layer by layer)."""
    rng = np.random.default_rng(n + rows)
    nets = []
    for i, (m, r) in enumerate([(n, rows), (n, rows // 4), (96, 40)]):
        csc = [layer(m, 24, 0.0625, rng) for _ in range(6)]
        # inputs of some rows too few to live through the first layers
        y0 = po.input_binary(9, i, r, m, 0.02, 0.7)
        nets.append((csc, y0, np.float32(-0.3)))
    check(cs, nets, prec)
