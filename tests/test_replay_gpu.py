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


def shifted_layer(n, kmin, kmax, vals, rng):
    """U[kmin, kmax] inputs per output at random distances, weights from `vals`."""
    r = (np.arange(n)[:, None] + rng.choice(n, kmax, replace=False)[None, :]) % n
    count = rng.integers(kmin, kmax + 1, n)
    r = np.where(np.arange(kmax)[None, :] < count[:, None], r, n)
    r.sort(1)
    cp = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    ri = r[r < n].astype(np.int32)
    return cp, ri, rng.choice(np.asarray(vals, np.float32), len(ri))


# rows in doubt in one layer (between `lo` and `hi`) decide who replays them: one CTA
# per row or a cluster (132 and 33 of them on a B200, or 284 and 71)
@pytest.mark.parametrize("n,rows,layers,k,vals,bias,prec,lo,hi", [
    # weights of several values
    (264, 300, 8, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 1, 300),      # too narrow for a cluster
    (1024, 300, 8, (20, 44), (0.05, 0.07), -0.02, 2, 1, 71),              # clusters, two CTAs per SM
    (4096, 300, 6, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 72, 142),    # two rows per cluster
    (4096, 600, 6, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 143, 284),   # a CTA per row
    (16384, 600, 4, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 1, 33),     # clusters, one CTA per SM
    (16384, 1500, 4, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 67, 132),  # a row in shared memory, one in scratch
    (24576, 130, 4, (0, 32), (0.06, 0.0625, 0.065), -0.02, 2, 1, 33),     # both rows in scratch
    # one weight value
    (1024, 300, 10, (20, 44), (0.07,), -0.02, 2, 143, 284),               # six groups of entries
    (1024, 300, 10, (0, 16), (0.125,), -0.02, 2, 143, 284),               # two, a power of two
    (1024, 300, 10, (0, 32), (0.0625,), -0.02, 2, 1, 300),                # the Graph Challenge's form
    (8192, 40, 5, (0, 32), (0.0625,), -0.02, 2, 1, 33),                   # by clusters
    (8192, 700, 5, (0, 32), (0.0625,), -0.02, 2, 67, 132),                # by CTAs
    (65536, 200, 3, (4, 32), (0.0625,), -0.08, 1, 1, 33),                 # entries counted
    (65536, 200, 3, (32, 32), (0.0625,), -0.3, 1, 1, 33),                 # rows in scratch
])
def test_replay_matches_fp64(n, rows, layers, k, vals, bias, prec, lo, hi):
    rng = np.random.default_rng(n + rows)
    csc = [shifted_layer(n, *k, vals, rng) for _ in range(layers)]
    y0 = (rng.random((rows, n), dtype=np.float32) * rng.uniform(0.05, 0.6, (rows, 1)).astype(np.float32))
    net = (csc, y0, np.float32(bias))
    ref = oracle_run(*net, want_final=True)
    eng = engine(net, prec)
    for step in range(2):
        eng.run() if step == 0 else eng.profile_layers()
        res = eng.result(0)
        np.testing.assert_array_equal(res["alive"], ref["alive"])
        np.testing.assert_array_equal(res["categories"], ref["categories"])
        assert lo <= res["rechecked"].max() <= hi, res["rechecked"]
        if len(res["categories"]):
            got = eng.final_values(0, len(res["categories"])).astype(np.float64)
            assert np.abs(got - ref["final"][ref["categories"]]).max() <= eng.final_bound(0)
    eng.close()


def test_replay_of_vanishing_values():
    """Threshold 0 and no bias: two inputs of weight 1/4 halve every value until
    the products themselves vanish (2^-1075 rounds to 0), a layer before their
    sum would."""
    import cospdnn_b200 as cs
    n, layers = 16, 1080
    cp = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    ri = np.sort((np.arange(n)[:, None] + [0, 5]) % n, 1).reshape(-1).astype(np.int32)
    csc = [(cp, ri, np.full(2 * n, 0.25, np.float32))] * layers
    net = (csc, np.ones((9, n), np.float32), np.float32(0))
    ref = oracle_run(*net, tau=0.0)
    last = np.nonzero(ref["alive"])[0][-1]
    assert 1070 < last + 1 < layers
    eng = engine(net, cs.PREC_FP16, tau=0.0)
    eng.run()
    np.testing.assert_array_equal(eng.result(0)["alive"], ref["alive"])
    eng.close()
