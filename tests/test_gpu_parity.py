"""GPU parity tests: every call goes through the C ABI (libglades_b200.so) and is checked against
the CPU oracle (golden vectors made by the compiled reference, and the C restatement).

Tolerances.  Reference mode keeps the reference's fp32 operation order exactly; the only freedom
is the rounding of expf / tanhf / logf (the kernels round a double-precision result once, glibc's
single-precision functions differ from that by one ulp on a small share of inputs).  So:
  * against the restatement run with the same correctly rounded transcendentals: BIT-EXACT;
  * against the golden vectors of the compiled reference: bit-exact for nets without
    transcendentals, 1e-5 relative at step level, and a stated drift bound on long trajectories.
Batched mode sums in a different order from the reference: 1e-5 relative to the largest magnitude
of the compared tensor (the tolerance the task states for fp32), identical argmax / confusion counts.
"""
import glob
import os

import numpy as np
import pytest

from conftest import GOLDEN, bits, desc_from_meta, libc_srand, load_golden, rel_err

pytestmark = pytest.mark.gpu

TRAJ = sorted(os.path.basename(p)[:-4] for p in glob.glob(os.path.join(GOLDEN, "traj_*.npz")))
RTOL = 1e-5


def tensor_close(a, b, rtol=RTOL):
    """|a-b| <= rtol * max|b| elementwise-max norm: the fp32 tolerance for re-ordered sums."""
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    scale = max(float(np.max(np.abs(b))), 1e-30)
    return float(np.max(np.abs(a - b))) <= rtol * scale, float(np.max(np.abs(a - b))) / scale


@pytest.fixture(autouse=True)
def _need_gpu(g):
    if g.device_count() < 1:
        pytest.fail("no sm_100 device visible: GPU tests cannot fall back to anything else")


@pytest.fixture()
def cr_math(oracle):
    """Runs the restatement with correctly rounded transcendentals (what the kernels compute)."""
    oracle.restate_lib().rs_set_math_mode(1)
    yield
    oracle.restate_lib().rs_set_math_mode(0)


# ------------------------------------------------------------------------------------------------
# reference mode
@pytest.mark.parametrize("name", TRAJ)
def test_reference_mode_trajectory_bit_exact_vs_restatement(g, oracle, cr_math, name):
    meta, z = load_golden(name)
    d = desc_from_meta(g, meta)
    net = g.Net(d)
    net.set_weights(z["w0"], z["b0"])
    net.set_data(z["x"], z["y"])
    S = oracle.Restate(d, z["x"], z["y"], g.Metrics)
    S.set_weights(z["w0"], z["b0"])
    # Each side runs its whole trajectory by itself: with dropout both draw their node flags from the C
    # library's rand(), which is seeded once before a run and must not be shared between two runs.
    if "srand" in meta:
        libc_srand(meta["srand"])
    done = 0
    got = []
    for e in meta["snapshots"]:
        m = net.train_epochs(e - done)
        done = e
        got.append((m, net.get_weights(), net.confusion() if meta["out"] != "regression" else None))
    if "srand" in meta:
        libc_srand(meta["srand"])
    done = 0
    for (m, (w, b), cm), e in zip(got, meta["snapshots"]):
        for _ in range(e - done):
            ms, cms, _ = S.epoch(0)
        done = e
        ws, bs = S.get_weights()
        assert np.array_equal(bits(w), bits(ws)), "weights differ at epoch %d" % e
        assert np.array_equal(bits(b), bits(bs)), "bias differs at epoch %d" % e
        assert m.total_error == ms.total_error and m.total_accuracy == ms.total_accuracy
        if meta["out"] != "regression":
            assert np.array_equal(cm, cms)
            for k in ("class_accuracy", "class_precision", "class_recall", "class_specificity", "class_f1"):
                a, bb = getattr(m, k), getattr(ms, k)
                assert a == bb or (np.isnan(a) and np.isnan(bb)), k
    for q in range(meta["batch"]):
        assert np.array_equal(bits(net.pending_delta(q)), bits(S.pending_delta(q)))
    assert net.epochs() == meta["epochs"]
    if "srand" in meta:
        # the test pass drops nodes too: same flags after the same seed, same outputs bit for bit
        libc_srand(meta["srand"] + 1)
        out_g, am_g, mt = net.forward(0, z["x"].shape[0])
        libc_srand(meta["srand"] + 1)
        mst, cmst, out_s = S.epoch(1, True)
        assert np.array_equal(bits(out_g), bits(out_s))
        assert mt.total_error == mst.total_error and mt.total_accuracy == mst.total_accuracy
        if meta["out"] != "regression":
            assert np.array_equal(net.confusion(), cmst)
    net.close()


# bound against the compiled reference's golden weights, as max|a-b| / max|b| per tensor: 0 (bit-exact)
# where the net has no transcendental function, else the stated fp32 tolerance 1e-5 -- one-ulp libm
# differences grow to about 1.5e-6 over the longest run here (200 epochs of online SGD)
GOLDEN_RTOL = {"traj_relu_6_5_4_2_mb7": 0.0}
# (dropout flags are integers: with them identical, the dropout fixtures keep the same tolerance)


@pytest.mark.parametrize("name", TRAJ)
def test_reference_mode_trajectory_vs_golden(g, name):
    meta, z = load_golden(name)
    d = desc_from_meta(g, meta)
    net = g.Net(d)
    net.set_weights(z["w0"], z["b0"])
    net.set_data(z["x"], z["y"])
    if "srand" in meta:
        libc_srand(meta["srand"])  # the run that made the fixture seeded rand() once, before its first epoch
    done = 0
    for k, e in enumerate(meta["snapshots"]):
        m = net.train_epochs(e - done)
        done = e
        w, b = net.get_weights()
        tol = GOLDEN_RTOL.get(name, RTOL)
        if tol == 0.0:
            assert np.array_equal(bits(w), bits(z["w"][k])) and np.array_equal(bits(b), bits(z["b"][k]))
            assert np.array_equal(bits(np.float32(m.total_accuracy)), bits(z["metrics"][k][1]))
        else:
            ok, err = tensor_close(w, z["w"][k], tol)
            assert ok, "epoch %d: weight error %g > %g" % (e, err, tol)
            assert abs(m.total_accuracy - z["metrics"][k][1]) <= max(1e-3, tol * 100)
            assert abs(m.total_error - z["metrics"][k][0]) <= max(1e-5, 10 * tol) * max(1.0, abs(z["metrics"][k][0]))
        if meta["out"] != "regression":
            assert np.array_equal(net.confusion(), z["confusion"][k]), "confusion counts, epoch %d" % e
    net.close()


def test_reference_mode_goes_nonfinite_on_the_same_step(g):
    meta, z = load_golden("cfg1_lr01_nonfinite")
    d = desc_from_meta(g, meta)
    bad = meta["first_bad_step"]
    assert 0 < bad < 150
    # batch 1: training the first k+1 rows for one epoch is exactly the first k+1 steps
    net = g.Net(d)
    net.set_weights(z["w0"], z["b0"])
    net.set_data(z["x"][:bad], z["y"][:bad])
    m = net.train_epochs(1)
    w, b = net.get_weights()
    assert m.nonfinite == 0 and np.isfinite(w).all()
    ok, err = tensor_close(w, z["w_last_good"], 1e-5)
    assert ok, err
    net.set_weights(z["w0"], z["b0"])
    net.set_data(z["x"][:bad + 1], z["y"][:bad + 1])
    m = net.train_epochs(1)
    w, b = net.get_weights()
    assert m.nonfinite == 1 and not (np.isfinite(w).all() and np.isfinite(b).all())
    net.close()


def test_reference_mode_cfg2_step_level(g, oracle, cr_math):
    meta, z = load_golden("cfg2_step")
    d = desc_from_meta(g, meta)
    idx = np.arange(1024)
    x = ((idx[:, None] >> np.arange(9, -1, -1)) & 1).astype(np.float32)
    y = (x.sum(1) % 2).astype(np.float32)[:, None]
    w0 = oracle.synth_fill(g.weight_count(d), meta["seed"], meta["stream"], 0, meta["scale"], meta["offset"])
    net = g.Net(d)
    for k, r in enumerate(meta["snapshot_rows"]):
        net.set_weights(w0, None)
        net.set_data(x[:r + 1], y[:r + 1])
        net.train_epochs(1)
        w, b = net.get_weights()
        # the hidden error sum carries factors up to 2^31 (doubling accumulation); compare with the
        # golden at the stated 1e-5, and bit for bit with the restatement that rounds tanh the same way
        ok, err = tensor_close(w, z["w_rows"][k], RTOL)
        assert ok, (r, err)
        S = oracle.Restate(d, x[:r + 1], y[:r + 1], g.Metrics)
        S.set_weights(w0, None)
        S.epoch(0)
        ws, bs = S.get_weights()
        assert np.array_equal(bits(w), bits(ws)) and np.array_equal(bits(b), bits(bs)), r
    net.close()


# (the reference's hidden error sum doubles per output node, network.cpp:660-662: a 40-wide head multiplies the
# first node's term by 2^39, so these cases need a tiny learning rate to stay finite)
@pytest.mark.parametrize("sizes,rows,mb,lr", [([6, 9, 40], 23, 1, 2e-13), ([5, 7, 3], 1, 1, 0.05), ([8, 12, 33], 17, 4, 1e-11)])
def test_reference_mode_live_vs_restatement_row_prefetch_and_wide_head(g, oracle, cr_math, sizes, rows, mb, lr):
    """Reference mode, three epochs in one launch, against the restatement bit for bit: the kernel fetches the
    next sample's rows while the current one runs (wrapping to row 0 at an epoch's end; a one-row data set
    prefetches its own row), and keeps an epoch's confusion counts in shared memory up to 1024 cells --
    40 x 40 and 33 x 33 heads take the global-memory path."""
    rng = np.random.default_rng(sum(sizes) + rows)
    d = g.make_desc(sizes, ["relu", "sigmoid"], "classification", batch=mb, lr=lr, momentum=0.5, mode=g.MODE_REFERENCE)
    x = rng.uniform(-1, 1, (rows, sizes[0])).astype(np.float32)
    y = np.full((rows, sizes[-1]), 0.01, np.float32)
    y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 0.99
    w = rng.uniform(-0.3, 0.3, g.weight_count(d)).astype(np.float32)
    b = rng.uniform(-0.1, 0.1, len(sizes) - 2).astype(np.float32)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    m = net.train_epochs(3)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for _ in range(3):
        ms, cms, _ = S.epoch(0)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    assert np.isfinite(ws).all() and not np.array_equal(ws, w), "the case itself must stay finite and must train"
    assert np.array_equal(bits(wg), bits(ws)) and np.array_equal(bits(bg), bits(bs))
    assert m.total_error == ms.total_error and m.total_accuracy == ms.total_accuracy
    assert np.array_equal(net.confusion(), cms)
    net.close()


# (edges of the small networks' sample loop: one node, whole and ragged warps, its largest layers and the first sizes
# beyond them; one and two hidden layers; minibatches that leave deltas pending at an epoch's end; decay; rows around the
# depth of the row ring; biases that cross zero and powers of two)
@pytest.mark.parametrize("sizes,rows,mb,lr,wd,bias", [
    ([1, 1, 1], 1, 1, 1e-2, 0.0, 0.05), ([2, 31, 2], 2, 1, 1e-4, 0.01, 1e-6), ([33, 32, 3], 3, 1, 1e-4, 0.0, -0.25),
    ([64, 64, 4], 50, 1, 1e-4, 0.0, 0.2500001), ([65, 17, 2], 9, 3, 1e-3, 0.0, 0.01), ([7, 33, 3], 37, 8, 1e-4, 0.02, -0.03),
    ([5, 64, 8, 3], 21, 1, 1e-6, 0.0, 0.125), ([9, 40, 5, 2], 23, 4, 1e-5, 0.01, -1e-7), ([3, 256, 2], 6, 1, 1e-5, 0.0, 0.02),
    ([3, 257, 2], 6, 2, 1e-5, 0.0, 0.02)])
def test_reference_mode_small_networks_vs_restatement(g, oracle, cr_math, sizes, rows, mb, lr, wd, bias):
    rng = np.random.default_rng(sum(sizes) + rows)
    layers = len(sizes) - 1
    for out in ("classification", "regression"):
        d = g.make_desc(sizes, ["tanh"] * (layers - 1) + ["sigmoid"], out, batch=mb, lr=lr, momentum=0.9, mode=g.MODE_REFERENCE)
        for l in range(layers):
            d.wd1[l], d.wd2[l] = wd, wd / 2
        x = rng.uniform(-1, 1, (rows, sizes[0])).astype(np.float32)
        y = np.full((rows, sizes[-1]), 0.01, np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 0.99
        w = rng.uniform(-0.3, 0.3, g.weight_count(d)).astype(np.float32)
        b = np.full(layers - 1, bias, np.float32)
        net = g.Net(d)
        net.set_weights(w, b)
        net.set_data(x, y)
        S = oracle.Restate(d, x, y, g.Metrics)
        S.set_weights(w, b)
        for epochs in (2, 1):
            m = net.train_epochs(epochs)
            for _ in range(epochs):
                ms, cms, _ = S.epoch(0)
            wg, bg = net.get_weights()
            ws, bs = S.get_weights()
            assert np.isfinite(ws).all()
            assert np.array_equal(bits(wg), bits(ws)) and np.array_equal(bits(bg), bits(bs))
            assert m.total_error == ms.total_error and m.total_accuracy == ms.total_accuracy
            assert out == "regression" or np.array_equal(net.confusion(), cms)
        net.close()


# (the first two are narrow enough for the tiles at most numbers of rows; all layers of the others go by rows up to 32 rows)
FEW_ROWS = [1, 2, 8, 9, 16, 17, 32, 33, 63, 65, 130]
FEW_ROWS_NETS = [[37, 70, 129, 5], [128, 16, 64, 1], [301, 517, 259, 5], [256, 512, 320, 20]]


@pytest.mark.parametrize("rows", FEW_ROWS)
@pytest.mark.parametrize("sizes", FEW_ROWS_NETS)
def test_forward_of_few_rows_equals_that_of_many(g, oracle, sizes, rows):
    """Small batches take the product by rows where it is the cheaper one (16 nodes x 1, 8, 16 or 32 rows per CTA; widths with
    and without whole 16-byte chunks): every row bit for bit as in a batch of 700 by tiles, and like the restatement."""
    rng = np.random.default_rng(rows)
    d = g.make_desc(sizes, ["relu", "tanh", "softmax" if sizes[-1] > 1 else "linear"], "classification" if sizes[-1] > 1 else "regression",
                    batch=32, mode=g.MODE_BATCHED, gemm=g.GEMM_FFMA)
    x = rng.standard_normal((700, sizes[0])).astype(np.float32)
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    few, am, _ = net.forward_host(x[:rows])
    many, amm, _ = net.forward_host(x)
    if sizes[-2] % 4 or sizes[-1] > 16:  # (the other network's last layer has a kernel of its own from 64 rows on)
        assert np.array_equal(bits(few), bits(many[:rows])) and np.array_equal(am, amm[:rows])
    S = oracle.Restate(d, x, np.zeros((700, sizes[-1]), np.float32), g.Metrics)
    S.set_weights(w, b)
    want = S.forward_block(0, rows)[0]
    ok, err = tensor_close(few, want.reshape(few.shape))
    assert ok, err
    net.close()


# (the layer products by FFMA: whole and half tiles, outputs of at most 16 nodes, output layers read one row or four rows per
# warp, layers whose rows start off 16-byte boundaries, scaled deltas of momentum windows, decay; edges of the tiles; tiles of 32 to
# 128 rows for each kind of product, gradients with and without momentum)
FFMA_WINDOWS = [
    ([33, 65, 31, 2], 63, 0.9, 0.0), ([64, 64, 128, 16], 64, 0.0, 0.0), ([130, 600, 17], 1000, 0.9, 0.001),
    ([97, 640, 700, 10], 333, 0.5, 0.0), ([12, 1024, 96, 1], 4800, 0.9, 0.0), ([784, 1000, 500, 10], 1000, 0.9, 0.0),
    ([784, 1000, 500, 10], 300, 0.0, 0.0), ([1001, 1030, 18], 260, 0.9, 0.0), ([1001, 1030, 18], 131, 0.0, 0.001)]


@pytest.mark.parametrize("sizes,rows,mom,wd", FFMA_WINDOWS)
def test_window_by_ffma_products_vs_restatement(g, oracle, sizes, rows, mom, wd):
    rng = np.random.default_rng(rows)
    layers = len(sizes) - 1
    acts = ["tanh"] * (layers - 1) + ["softmax" if sizes[-1] > 1 else "linear"]
    out = "classification" if sizes[-1] > 1 else "regression"
    d = g.make_desc(sizes, acts, out, batch=rows, lr=0.02, momentum=mom, wd1=wd, wd2=wd, mode=g.MODE_BATCHED, gemm=g.GEMM_FFMA)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = np.zeros((rows, sizes[-1]), np.float32)
    y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for _ in range(2):
        net.train_window(0, rows)
        S.window_apply(S.window_grad(0, rows), rows)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    ok, err = tensor_close(wg, ws, 2e-5)
    assert ok, err
    assert np.allclose(bg, bs, rtol=2e-4, atol=2e-6)
    net.close()


# (groups of 2, 4, 8, 12 and 16 rows, one and several per CTA; layers that give a warp 16, 32 and 64 nodes, of more than 256 nodes, of
# whole and of ragged 32-node tiles; rows on and off 16-byte boundaries, each with each group size; narrow heads of 1 to 4 nodes and a narrow hidden layer; decay;
# windows of whole and of ragged 128-row copies, a short last window)
@pytest.mark.parametrize("sizes,rows,batch,mom,wd", [
    ([57, 200, 90, 7], 625, 250, 0.9, 0.0), ([20, 296, 256, 12], 1600, 1525, 0.5, 0.0), ([24, 300, 33, 3], 2300, 2200, 0.9, 0.001),
    ([33, 65, 129, 1], 1200, 1100, 0.0, 0.0), ([64, 128, 4, 64, 2], 700, 500, 0.9, 0.0), ([32, 64, 4], 129, 128, 0.9, 0.001),
    ([60, 516, 20, 16], 5000, 4900, 0.9, 0.0), ([12, 16, 8], 65, 63, 0.5, 0.002),
    ([24, 300, 32, 3], 2300, 2200, 0.5, 0.0), ([24, 300, 32, 3], 4800, 4700, 0.9, 0.0), ([57, 200, 90, 7], 600, 500, 0.9, 0.0),
    ([57, 200, 90, 7], 1600, 1525, 0.0, 0.001), ([57, 200, 90, 7], 1200, 1000, 0.5, 0.0)])
def test_whole_windows_in_one_launch_vs_restatement(g, oracle, sizes, rows, batch, mom, wd):
    rng = np.random.default_rng(rows + batch)
    layers = len(sizes) - 1
    head, out = ("softmax", "classification") if sizes[-1] > 1 else ("linear", "regression")
    d = g.make_desc(sizes, ["tanh"] * (layers - 1) + [head], out, batch=batch, lr=0.02, momentum=mom, wd1=wd, wd2=wd,
                    mode=g.MODE_BATCHED, gemm=g.GEMM_GRID_FUSED)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = np.zeros((rows, sizes[-1]), np.float32)
    y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    net.train_epochs(2)
    for _ in range(2):
        for r0 in range(0, rows, batch):
            n = min(batch, rows - r0)
            S.window_apply(S.window_grad(r0, n), n)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    ok, err = tensor_close(wg, ws, 2e-5)
    assert ok, err
    assert np.allclose(bg, bs, rtol=2e-4, atol=2e-6)
    net.close()


@pytest.mark.parametrize("inputs", [1048574, 1048575, 1048576, 1572863, 1572870])
def test_weights_cross_host_memory_around_the_copy_threads_sizes(g, inputs):
    """4 MB is the line between one plain copy and the copy threads' 2 MB chunks: whole and ragged last chunks."""
    net = g.Net(g.make_desc([inputs, 1, 1], ["tanh", "linear"], "regression", batch=4, lr=0.1, mode=g.MODE_BATCHED))
    w = np.arange(inputs + 1, dtype=np.float32)
    net.set_weights(w, np.zeros(1, np.float32))
    assert np.array_equal(net.get_weights()[0], w)
    net.close()


# (smooth networks on the fp16-split tensor products: every shape, remainders in m, n and k, the narrowest tiles)
@pytest.mark.parametrize("sizes,rows,mom", [([130, 515, 131, 7], 1029, 0.9), ([64, 128, 256, 33], 128, 0.0), ([31, 300, 65, 1], 257, 0.5)])
def test_smooth_window_by_tensor_products_vs_restatement(g, oracle, sizes, rows, mom):
    rng = np.random.default_rng(rows)
    layers = len(sizes) - 1
    head, out = ("softmax", "classification") if sizes[-1] > 1 else ("linear", "regression")
    d = g.make_desc(sizes, ["tanh"] * (layers - 1) + [head], out, batch=rows, lr=0.02, momentum=mom, mode=g.MODE_BATCHED, gemm=g.GEMM_TCGEN05)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = np.zeros((rows, sizes[-1]), np.float32)
    y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for _ in range(2):
        net.train_window(0, rows)
        S.window_apply(S.window_grad(0, rows), rows)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    ok, err = tensor_close(wg, ws, 2e-5)
    assert ok, err
    assert np.allclose(bg, bs, rtol=2e-4, atol=2e-6)
    net.close()


@pytest.mark.parametrize("name", ["fwd_cfg3_32_256_256_1", "fwd_cfg5_784_2048_2048_10", "fwd_cfg4_1024_4096_4096_1024"])
def test_forward_wide_shapes_vs_golden(g, oracle, name):
    """Forward parity on the wide shapes, sampled rows, against the compiled reference's activations:
    reference mode (exact order) bit for bit on the ReLU layers and within 1 ulp behind a sigmoid;
    batched mode within 1e-5 with the same argmax."""
    meta, z = load_golden(name)
    sizes = meta["sizes"]
    w = oracle.synth_fill(int(np.sum(np.array(sizes[1:]) * np.array(sizes[:-1]))), meta["seed"], meta["stream"], 0,
                          meta["scale"], meta["offset"])
    b = np.array(meta["bias"], np.float32)
    x = z["x"]
    rows = x.shape[0]
    y = np.full((rows, sizes[-1]), 0.01, np.float32)
    hidden = sum(sizes[1:-1])
    d = desc_from_meta(g, meta)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    for r in range(rows):
        a = net.activations(r)
        assert np.array_equal(bits(a[:hidden]), bits(z["acts"][r][:hidden])), "hidden activations, row %d" % r
        last_act = meta["acts"][-1]
        if last_act in ("relu", "linear"):
            assert np.array_equal(bits(a[hidden:]), bits(z["acts"][r][hidden:]))
        else:
            assert np.max(np.abs(a[hidden:].astype(np.float64) - z["acts"][r][hidden:])) <= 1.2e-7
    out, am, _ = net.forward(0, rows)
    ref_out = z["acts"][:, hidden:]
    assert np.max(np.abs(out.astype(np.float64) - ref_out)) <= 1.2e-7 * max(1.0, float(np.max(np.abs(ref_out))))
    net.close()
    # batched arithmetic, native head and softmax head
    db = desc_from_meta(g, meta, mode=g.MODE_BATCHED)
    nb = g.Net(db)
    nb.set_weights(w, b)
    nb.set_data(x, y)
    outb, amb, _ = nb.forward(0, rows)
    ok, err = tensor_close(outb, ref_out)
    assert ok, err
    ref_am = np.array([int(np.argmax(r)) if np.max(r) > 0 else -1 for r in ref_out])
    if sizes[-1] > 1:
        assert np.array_equal(amb, ref_am)
    nb.close()
    if sizes[-1] > 1:
        acts_sm = list(meta["acts"][:-1]) + ["softmax"]
        ds = g.make_desc(sizes, acts_sm, "classification", batch=1, lr=0.0, params=meta.get("params"),
                         mode=g.MODE_BATCHED)
        ns = g.Net(ds)
        ns.set_weights(w, b)
        ns.set_data(x, y)
        outs, ams, _ = ns.forward(0, rows)
        zl = z["z_last"].astype(np.float64)
        sm = np.exp(zl - zl.max(1, keepdims=True))
        sm /= sm.sum(1, keepdims=True)
        ok, err = tensor_close(outs, sm)
        assert ok, err
        assert np.array_equal(ams, np.argmax(zl, 1))
        ns.close()


# ------------------------------------------------------------------------------------------------
# batched mode
def _rand_net(rng, sizes, lo=-0.4, hi=0.4):
    nw = int(np.sum(np.array(sizes[1:]) * np.array(sizes[:-1])))
    return rng.uniform(lo, hi, nw).astype(np.float32), rng.uniform(-0.1, 0.1, len(sizes) - 2).astype(np.float32)


BATCHED_CASES = [
    # sizes, acts, out, rows, momentum, wd1, wd2, bias_rule
    ([16, 32, 24, 4], ["tanh", "relu", "sigmoid"], "regression", 64, 0.5, 0.0, 0.0, 0),
    ([7, 13, 5], ["sigmoid", "sigmoid"], "classification", 33, 0.0, 0.0, 0.0, 0),
    ([5, 9, 11, 3], ["relu", "tanh", "softmax"], "classification", 17, 0.9, 0.0, 0.0, 0),
    ([3, 1, 2], ["leaky", "linear"], "regression", 1, 0.0, 0.001, 0.002, 1),
    ([33, 31, 1], ["relu", "linear"], "regression", 100, 0.9, 0.0, 0.0, 0),
    ([64, 128, 128, 10], ["relu", "relu", "softmax"], "classification", 256, 0.0, 0.0, 0.0, 0),
    ([10, 32, 32, 1], ["tanh", "tanh", "sigmoid"], "regression", 32, 0.0, 0.0, 0.0, 1),
]


GRID_FUSED_EXTRA = [
    # the window regressor's shape, and layers wider than one pass of the kernel's 256 threads
    ([32, 256, 256, 1], ["relu", "relu", "linear"], "regression", 1024, 0.9, 0.0, 0.0, 0),
    ([40, 300, 520, 12], ["tanh", "relu", "softmax"], "classification", 203, 0.5, 0.0005, 0.0, 0),
]


def _cluster_variant_applies(sizes):
    """The whole-window kernel's thread-block-cluster variant takes networks with a hidden layer whose input and
    hidden widths are multiples of 4 and whose per-CTA buffers fit one SM's shared memory (the same arithmetic as
    the library's cf_plan)."""
    H = len(sizes) - 2
    if H < 1 or any(s % 4 for s in sizes[:-1]):
        return False
    r4 = lambda v: (v + 3) & ~3
    sl = [r4((s + 7) // 8) for s in sizes]
    floats = (sum(sizes) + sum(r4(s) for s in sizes[1:])) * 32
    floats += sum(sl[l + 1] * (sizes[l] + 4) for l in range(H + 1))
    floats += sum(sl[j] * (r4(sizes[j + 1]) + 4) for j in range(1, H + 1)) + 64
    return floats * 4 <= 226 * 1024


@pytest.mark.parametrize("engine", ["ffma", "grid_fused", "grid_fused_cluster"])
@pytest.mark.parametrize("case", BATCHED_CASES + GRID_FUSED_EXTRA, ids=lambda c: "-".join(map(str, c[0])) + "_" + str(c[3]))
def test_batched_window_vs_restatement(g, oracle, monkeypatch, case, engine):
    """One minibatch window, per-layer products on the FFMA kernel vs the whole window in one
    cooperative launch (grid_fused, and its opt-in thread-block-cluster variant where the network allows it):
    all against the CPU restatement of the batched arithmetic."""
    sizes, acts, out, rows, mom, wd1, wd2, brule = case
    if engine == "grid_fused_cluster":
        if not _cluster_variant_applies(sizes):
            pytest.skip("the cluster variant does not take this network")
        monkeypatch.setenv("GLADES_GF_CLUSTER", "1")
    else:
        monkeypatch.delenv("GLADES_GF_CLUSTER", raising=False)
    rng = np.random.default_rng(sum(sizes) + rows)
    params = [0.05 if a == "leaky" else 1.0 for a in acts]
    d = g.make_desc(sizes, acts, out, batch=rows, lr=0.05 if rows < 1000 else 0.002, momentum=mom, wd1=wd1, wd2=wd2,
                    params=params, mode=g.MODE_BATCHED, bias_rule=brule,
                    gemm=g.GEMM_FFMA if engine == "ffma" else g.GEMM_GRID_FUSED)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    if acts[-1] == "softmax":
        y = np.zeros((rows, sizes[-1]), np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    else:
        y = rng.uniform(0.05, 0.95, (rows, sizes[-1])).astype(np.float32)
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for step in range(2):  # two steps: the second one starts from updated weights
        l0 = net.kernel_launches()
        m = net.train_window(0, rows)
        if engine.startswith("grid_fused"):
            assert net.kernel_launches() - l0 == 1, "the whole window must be one cooperative launch"
            assert (net.window_cluster_ctas() > 0) == (engine == "grid_fused_cluster"), net.window_cluster_ctas()
        cm = np.zeros((sizes[-1], sizes[-1]), np.int32)
        gr = S.window_grad(0, rows, confusion=cm)
        S.window_apply(gr, rows)
        wg, bg = net.get_weights()
        ws, bs = S.get_weights()
        # the update is compared through the gradient it applied: (w_before - w_after)
        ok, err = tensor_close(wg, ws)
        assert ok, "step %d weights rel err %g" % (step, err)
        assert np.allclose(bg, bs, rtol=1e-4, atol=1e-6), (bg, bs)
        cost, acc = gr[-2], gr[-1]
        assert abs(m.total_error - cost) <= 1e-5 * max(1.0, abs(cost))
        assert abs(m.total_accuracy - acc / (rows * sizes[-1])) <= 1e-3
    net.close()


def test_batched_gradient_tensor_vs_restatement(g, oracle):
    """The applied update, isolated: lr-scaled gradient = (w_before - w_after) * rows, per layer."""
    rng = np.random.default_rng(3)
    sizes = [24, 48, 40, 8]
    rows = 96
    d = g.make_desc(sizes, ["relu", "relu", "sigmoid"], "classification", batch=rows, lr=0.5, momentum=0.0,
                    mode=g.MODE_BATCHED, gemm=g.GEMM_FFMA)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = rng.uniform(0.05, 0.95, (rows, sizes[-1])).astype(np.float32)
    w, b = _rand_net(rng, sizes, -0.2, 0.2)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    net.train_window(0, rows)
    gr = S.window_grad(0, rows)
    wg, _ = net.get_weights()
    upd = (w.astype(np.float64) - wg.astype(np.float64)) * rows
    off = 0
    for l in range(3):
        cnt = sizes[l] * sizes[l + 1]
        ref = gr[off:off + cnt]
        got = upd[off:off + cnt]
        # w - (w - g/rows) loses bits of g relative to |w|; allow for that cancellation
        tol = 1e-5 * np.max(np.abs(ref)) + 2.0 ** -23 * np.max(np.abs(w)) * rows
        assert np.max(np.abs(got - ref)) <= tol, l
        off += cnt
    net.close()


def test_batched_epochs_metrics_and_confusion(g, oracle):
    rng = np.random.default_rng(8)
    sizes = [8, 16, 4]
    rows, mb = 100, 32  # 3 full windows + a 4-row tail
    d = g.make_desc(sizes, ["tanh", "sigmoid"], "classification", batch=mb, lr=0.05, momentum=0.3,
                    mode=g.MODE_BATCHED, gemm=g.GEMM_FFMA)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = np.full((rows, sizes[-1]), 0.01, np.float32)
    y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 0.99
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for ep in range(3):
        m = net.train_epochs(1)
        cm = np.zeros((sizes[-1], sizes[-1]), np.int32)
        cost = acc = 0.0
        for r0 in range(0, rows, mb):
            cnt = min(mb, rows - r0)
            gr = S.window_grad(r0, cnt, confusion=cm)
            S.window_apply(gr, cnt)
            cost += gr[-2]
            acc += gr[-1]
        assert np.array_equal(net.confusion(), cm), ep
        assert abs(m.total_error - cost) <= 1e-5 * max(1.0, abs(cost))
        assert abs(m.total_accuracy - acc / (rows * sizes[-1])) <= 1e-3
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    ok, err = tensor_close(wg, ws, 5e-5)
    assert ok, err
    assert net.epochs() == 3
    net.close()


def test_host_window_equals_resident_window(g):
    rng = np.random.default_rng(12)
    sizes = [12, 20, 6]
    rows = 48
    d = g.make_desc(sizes, ["relu", "sigmoid"], "regression", batch=rows, lr=0.1, mode=g.MODE_BATCHED,
                    gemm=g.GEMM_FFMA)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = rng.uniform(0, 1, (rows, sizes[-1])).astype(np.float32)
    w, b = _rand_net(rng, sizes)
    a, c = g.Net(d), g.Net(d)
    for n in (a, c):
        n.set_weights(w, b)
    a.set_data(x, y)
    a.train_window(0, rows)
    c.train_window_host(x, y)
    wa, ba = a.get_weights()
    wc, bc = c.get_weights()
    assert np.array_equal(bits(wa), bits(wc)) and np.array_equal(bits(ba), bits(bc))
    o1, am1, _ = a.forward(0, rows)
    o2, am2, _ = c.forward_host(x, y)
    assert np.array_equal(bits(o1), bits(o2)) and np.array_equal(am1, am2)
    a.close()
    c.close()


def test_empty_and_bad_arguments(g):
    d = g.make_desc([4, 5, 3], ["sigmoid", "sigmoid"], "classification", mode=g.MODE_BATCHED)
    net = g.Net(d)
    with pytest.raises(g.GladesError):
        net.train_window(0, 4)  # no data yet
    x = np.zeros((4, 4), np.float32)
    y = np.zeros((4, 3), np.float32)
    net.set_data(x, y)
    with pytest.raises(g.GladesError):
        net.train_window(2, 4)  # past the end
    with pytest.raises(g.GladesError):
        net.train_window(0, 0)  # empty window
    bad = g.make_desc([4, 5, 3], ["softmax", "sigmoid"], "classification", mode=g.MODE_BATCHED)
    with pytest.raises(g.GladesError):
        g.Net(bad)  # softmax only on the last layer
    bad2 = g.make_desc([4, 5, 3], ["sigmoid", "softmax"], "classification", mode=g.MODE_REFERENCE)
    with pytest.raises(g.GladesError):
        g.Net(bad2)  # the reference has no softmax
    net.close()


def test_synth_fill_matches_cpu_generator(g, oracle):
    import ctypes as C
    n = 100003
    L = g.lib()
    p = C.c_void_p()
    assert L.gl_device_alloc(C.byref(p), n * 4, 0) == 0
    host = np.empty(n, np.float32)
    assert L.gl_synth_fill(p, n, 0x474C4144, 2, 0, 2.0, -1.0, 0) == 0
    assert L.gl_memcpy_d2h(host.ctypes.data_as(C.c_void_p), p, n * 4, 0) == 0
    cpu = oracle.synth_fill(n, 0x474C4144, 2, 0, 2.0, -1.0)
    assert np.array_equal(bits(host), bits(cpu))  # uniform stream: integer arithmetic, exact
    assert L.gl_synth_fill(p, n, 77, 0, 1, 1.0, 0.0, 0) == 0
    assert L.gl_memcpy_d2h(host.ctypes.data_as(C.c_void_p), p, n * 4, 0) == 0
    cpu = oracle.synth_fill(n, 77, 0, 1, 1.0, 0.0)
    assert np.max(np.abs(host - cpu)) <= 1e-6  # normal stream: double libm on both sides, then one rounding
    assert abs(float(host.mean())) < 0.02 and abs(float(host.std()) - 1.0) < 0.02
    L.gl_device_free(p, 0)


def near_tie_rows(outputs, tol=2e-4):
    """Rows whose two largest outputs lie within `tol` (relative to the larger, floor 1): the only rows on
    which two correct fp32 evaluations with differently ordered sums may predict different classes."""
    if outputs.shape[1] < 2:
        return 0
    top = np.sort(outputs.astype(np.float64), axis=1)[:, -2:]
    return int(np.sum(top[:, 1] - top[:, 0] <= tol * np.maximum(1.0, np.abs(top[:, 1]))))


SMALL_FUSED_CASES = [
    # sizes, acts, out, rows, mb, momentum, wd1, wd2, bias_rule, epochs
    ([10, 32, 32, 1], ["tanh", "tanh", "sigmoid"], "regression", 1024, 32, 0.0, 0.0, 0.0, 0, 3),
    ([4, 16, 3], ["sigmoid", "softmax"], "classification", 150, 1, 0.9, 0.0, 0.0, 0, 2),
    ([7, 9, 5, 4], ["relu", "leaky", "sigmoid"], "regression", 77, 16, 0.7, 0.001, 0.002, 1, 3),
    ([33, 40, 2], ["tanh", "linear"], "regression", 50, 64, 0.5, 0.0, 0.0, 0, 2),
    # edges of the samples per warp (16 | 17, 32 | 33 rows), of quads, of warps and of the lanes per sample at the head
    ([1, 1, 2], ["tanh", "softmax"], "classification", 40, 17, 0.0, 0.0, 0.0, 0, 2),
    ([65, 33, 34, 40], ["tanh", "sigmoid", "softmax"], "classification", 100, 33, 0.9, 0.0, 0.0, 0, 2),
    ([3, 130, 9], ["relu", "softmax"], "classification", 70, 32, 0.0, 0.001, 0.002, 0, 2),
    # windows of 65 to 128 rows, five to eight samples per warp: both ends of the range, a remainder inside a warp's samples, rows that
    # the samples round up; the last one, whose rounded-up rows do not fit shared memory, goes by four in two turns
    ([33, 40, 2], ["tanh", "linear"], "regression", 130, 64, 0.5, 0.0, 0.0, 0, 2),
    ([28, 27, 3], ["relu", "softmax"], "classification", 203, 65, 0.9, 0.0, 0.0, 0, 2),
    ([5, 31, 40], ["tanh", "softmax"], "classification", 181, 81, 0.7, 0.001, 0.002, 0, 2),
    ([24, 50, 36, 9], ["tanh", "relu", "softmax"], "classification", 250, 97, 0.0, 0.001, 0.002, 0, 2),
    ([20, 90, 40, 5], ["sigmoid", "tanh", "softmax"], "classification", 300, 113, 0.9, 0.0, 0.0, 0, 2),
    ([12, 17, 1], ["relu", "linear"], "regression", 300, 128, 0.9, 0.0, 0.0, 0, 2),
    ([64, 64, 64, 4], ["tanh", "tanh", "softmax"], "classification", 240, 113, 0.5, 0.0, 0.0, 0, 2),
    ([12, 17, 2], ["tanh", "softmax"], "classification", 300, 129, 0.9, 0.0, 0.0, 0, 2),  # four again
]


@pytest.mark.parametrize("case", SMALL_FUSED_CASES, ids=lambda c: "-".join(map(str, c[0])) + "_mb%d" % c[4])
def test_small_network_fused_epochs_vs_restatement(g, oracle, case):
    """Batched-mode epochs of a network whose weights fit in shared memory run in the fused
    whole-network kernel (one launch); checked window by window against the restatement."""
    sizes, acts, out, rows, mb, mom, wd1, wd2, brule, epochs = case
    rng = np.random.default_rng(len(sizes) * 1000 + rows)
    params = [0.05 if a == "leaky" else 1.0 for a in acts]
    d = g.make_desc(sizes, acts, out, batch=mb, lr=0.005 if brule else 0.05, momentum=mom, wd1=wd1, wd2=wd2,
                    params=params, mode=g.MODE_BATCHED, bias_rule=brule)
    if sizes == [10, 32, 32, 1]:
        idx = np.arange(1024)
        x = ((idx[:, None] >> np.arange(9, -1, -1)) & 1).astype(np.float32)
        y = (x.sum(1) % 2).astype(np.float32)[:, None]
    else:
        x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
        if acts[-1] == "softmax":
            y = np.zeros((rows, sizes[-1]), np.float32)
            y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
        elif out == "classification":
            y = np.full((rows, sizes[-1]), 0.01, np.float32)
            y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 0.99
        else:
            y = rng.uniform(0.05, 0.95, (rows, sizes[-1])).astype(np.float32)
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    l0 = net.kernel_launches()
    m = net.train_epochs(epochs)
    assert net.kernel_launches() - l0 == 1, "the whole call must be one launch of the fused kernel"
    for ep in range(epochs):
        cm = np.zeros((sizes[-1], sizes[-1]), np.int32)
        cost = acc = 0.0
        ties = 0
        for r0 in range(0, rows, mb):
            cnt = min(mb, rows - r0)
            if out != "regression" and ep == epochs - 1:
                ties += near_tie_rows(S.forward_block(r0, cnt)[0])  # this window's predictions, before its update
            gr = S.window_grad(r0, cnt, confusion=cm)
            S.window_apply(gr, cnt)
            cost += gr[-2]
            acc += gr[-1]
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    assert np.isfinite(ws).all(), "the case itself must stay finite"
    ok, err = tensor_close(wg, ws, 2e-5 if epochs * (rows // mb + 1) > 50 else RTOL)
    assert ok, err
    assert np.allclose(bg, bs, rtol=2e-4, atol=2e-6), (bg, bs)
    assert abs(m.total_error - cost) <= 2e-5 * max(1.0, abs(cost))
    assert abs(m.total_accuracy - acc / (rows * sizes[-1])) <= 2e-3
    if out != "regression":
        # identical counts, except that a row whose two best outputs tie within the tolerance may land in
        # another cell (one count less in one cell, one more in another)
        diff = int(np.abs(net.confusion() - cm).sum())
        assert diff <= 2 * ties, "confusion counts differ by %d with %d near-tie rows" % (diff, ties)
    assert net.epochs() == epochs
    net.close()


GRID_FUSED_EPOCH_CASES = [
    # sizes, acts, out, rows, mb, momentum, bias_rule, epochs
    ([32, 256, 256, 1], ["relu", "relu", "linear"], "regression", 2500, 1024, 0.9, 0, 2),   # ragged last window
    ([20, 64, 48, 5], ["tanh", "relu", "softmax"], "classification", 333, 50, 0.6, 0, 3),
    ([12, 40, 3], ["sigmoid", "sigmoid"], "classification", 90, 7, 0.0, 0, 2),          # windows shorter than a row group
]


@pytest.mark.parametrize("cluster", ["cluster", "plain"])
@pytest.mark.parametrize("case", GRID_FUSED_EPOCH_CASES, ids=lambda c: "-".join(map(str, c[0])) + "_mb%d" % c[4])
def test_grid_fused_epochs_vs_restatement(g, oracle, monkeypatch, case, cluster):
    """Whole training runs (epochs x windows, ragged tail included) of a mid-size network in ONE
    cooperative launch, checked against the restatement walked window by window -- on the cluster variant of
    the kernel and on the plain one."""
    sizes, acts, out, rows, mb, mom, brule, epochs = case
    if cluster == "plain":
        monkeypatch.delenv("GLADES_GF_CLUSTER", raising=False)
    else:
        monkeypatch.setenv("GLADES_GF_CLUSTER", "1")
        assert _cluster_variant_applies(sizes)
    rng = np.random.default_rng(len(sizes) * 100 + rows)
    d = g.make_desc(sizes, acts, out, batch=mb, lr=0.002 if mb > 500 else 0.05, momentum=mom, mode=g.MODE_BATCHED,
                    bias_rule=brule, gemm=g.GEMM_GRID_FUSED)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    if acts[-1] == "softmax":
        y = np.zeros((rows, sizes[-1]), np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    elif out == "classification":
        y = np.full((rows, sizes[-1]), 0.01, np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 0.99
    else:
        y = rng.uniform(0.05, 0.95, (rows, sizes[-1])).astype(np.float32)
    w, b = _rand_net(rng, sizes, -0.15, 0.15)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    l0 = net.kernel_launches()
    m = net.train_epochs(epochs)
    assert net.kernel_launches() - l0 == 1
    assert (net.window_cluster_ctas() > 0) == (cluster == "cluster"), net.window_cluster_ctas()
    for ep in range(epochs):
        cm = np.zeros((sizes[-1], sizes[-1]), np.int32)
        cost = acc = 0.0
        ties = 0
        for r0 in range(0, rows, mb):
            cnt = min(mb, rows - r0)
            if out != "regression" and ep == epochs - 1:
                ties += near_tie_rows(S.forward_block(r0, cnt)[0])  # this window's predictions, before its update
            gr = S.window_grad(r0, cnt, confusion=cm)
            S.window_apply(gr, cnt)
            cost += gr[-2]
            acc += gr[-1]
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    assert np.isfinite(ws).all(), "the case itself must stay finite"
    ok, err = tensor_close(wg, ws, 2e-5)
    assert ok, err
    assert np.allclose(bg, bs, rtol=2e-4, atol=2e-6), (bg, bs)
    assert abs(m.total_error - cost) <= 2e-5 * max(1.0, abs(cost))
    assert abs(m.total_accuracy - acc / (rows * sizes[-1])) <= 2e-3
    if out != "regression":
        diff = int(np.abs(net.confusion() - cm).sum())
        assert diff <= 2 * ties, "confusion counts differ by %d with %d near-tie rows" % (diff, ties)
    assert net.epochs() == epochs and not m.nonfinite
    # the last row's predictions, as the reference's getResults() hands them out
    assert np.all(np.isfinite(net.last_outputs()))
    net.close()


def test_grid_fused_engine_is_refused_where_it_does_not_fit(g):
    with pytest.raises(RuntimeError):
        g.Net(g.make_desc([1024, 4096, 1024], ["relu", "sigmoid"], "regression", batch=64, lr=0.1, mode=g.MODE_BATCHED,
                          gemm=g.GEMM_GRID_FUSED))
    with pytest.raises(RuntimeError):
        g.Net(g.make_desc([4, 8, 2], ["tanh", "sigmoid"], "regression", batch=4, lr=0.1, mode=g.MODE_REFERENCE,
                          gemm=g.GEMM_GRID_FUSED))


def test_pipelined_host_windows_equal_synchronous_ones(g):
    """submit/result keeps two host-buffer windows in flight; the weights and every window's loss
    must equal those of the one-at-a-time entry point, and a third submit must be refused."""
    rng = np.random.default_rng(77)
    sizes = [12, 24, 5]
    rows, steps = 40, 5
    d = g.make_desc(sizes, ["tanh", "softmax"], "classification", batch=rows, lr=0.1, momentum=0.3, mode=g.MODE_BATCHED,
                    gemm=g.GEMM_FFMA)
    xs = [rng.standard_normal((rows, sizes[0])).astype(np.float32) for _ in range(steps)]
    ys = []
    for _ in range(steps):
        y = np.zeros((rows, sizes[-1]), np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
        ys.append(y)
    w, b = _rand_net(rng, sizes)
    a, c = g.Net(d), g.Net(d)
    a.set_weights(w, b)
    c.set_weights(w, b)
    sync_losses = [a.train_window_host(xs[i], ys[i]).total_error for i in range(steps)]
    pipe_losses = []
    c.submit_window_host(xs[0], ys[0])
    for i in range(1, steps):
        c.submit_window_host(xs[i], ys[i])
        if i == 1:
            with pytest.raises(g.GladesError):
                c.submit_window_host(xs[i], ys[i])  # two already in flight
        pipe_losses.append(c.window_result().total_error)
    pipe_losses.append(c.window_result().total_error)
    with pytest.raises(g.GladesError):
        c.window_result()  # nothing left in flight
    assert pipe_losses == sync_losses
    wa, ba = a.get_weights()
    wc, bc = c.get_weights()
    assert np.array_equal(bits(wa), bits(wc)) and np.array_equal(bits(ba), bits(bc))
    a.close()
    c.close()


def test_pipelined_inference_batches_equal_synchronous_ones(g):
    """gl_forward_host_submit / _result keep two host batches in flight: classes and metric sums of every
    batch must equal those of the one-at-a-time entry point; a third submit is refused, and a training
    result call must not collect an inference batch."""
    rng = np.random.default_rng(91)
    sizes = [20, 48, 7]
    d = g.make_desc(sizes, ["relu", "softmax"], "classification", batch=64, lr=0.05, mode=g.MODE_BATCHED)
    w, b = _rand_net(rng, sizes)
    net = g.Net(d)
    net.set_weights(w, b)
    batches = []
    for rows in (64, 33, 64, 5):
        x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
        y = np.zeros((rows, sizes[-1]), np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
        batches.append((x, y))
    want = [net.forward_host(x, y) for x, y in batches]
    got = []
    net.submit_forward_host(*batches[0])
    net.submit_forward_host(*batches[1])
    with pytest.raises(RuntimeError):
        net.submit_forward_host(*batches[2])          # two in flight already
    with pytest.raises(RuntimeError):
        net.window_result()                           # the oldest call in flight is not a training window
    got.append(net.forward_result(batches[0][0].shape[0]))
    net.submit_forward_host(*batches[2])
    got.append(net.forward_result(batches[1][0].shape[0]))
    net.submit_forward_host(batches[3][0], None)      # no expected rows: classes only
    got.append(net.forward_result(batches[2][0].shape[0]))
    got.append(net.forward_result(batches[3][0].shape[0]))
    with pytest.raises(RuntimeError):
        net.forward_result(1)                         # nothing in flight
    for k, ((_, am_w, m_w), (am_g, m_g)) in enumerate(zip(want, got)):
        assert np.array_equal(am_w, am_g), k
        if k < 3:
            assert abs(m_w.total_error - m_g.total_error) <= 1e-6 * max(1.0, abs(m_w.total_error)), k
            assert abs(m_w.total_accuracy - m_g.total_accuracy) <= 1e-4, k
    net.close()
