"""GPU tests of the tensor-core (TMA + tcgen05) layer products, through the C ABI: 3xFP16 (gl_matmul, networks without jumps,
backward products of large windows) and 3xTF32 in a fixed order (networks whose activations jump).

Tolerance: both splits keep at least 21 mantissa bits per operand and accumulate in fp32, so
each output must agree with a float64 product within 4e-6 * sum_k |a_mk||b_nk| (the fp32 tolerance
1e-5 of the task with margin; plain TF32 would be ~1e-3 and fail)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(L, a):
    p = C.c_void_p()
    assert L.gl_device_alloc(C.byref(p), a.nbytes + 64, 0) == 0
    assert L.gl_memcpy_h2d(p, a.ctypes.data_as(C.c_void_p), a.nbytes, 0) == 0
    return p


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1), (1, 0)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 32), (256, 256, 64), (128, 384, 96), (384, 256, 160), (256, 512, 1024),
                                   (128, 128, 48), (256, 256, 784)])
def test_tc_matmul_all_layouts(g, a_mn, b_mn, M, N, K):
    L = g.lib()
    rng = np.random.default_rng(M + 3 * N + 7 * K + a_mn + 2 * b_mn)
    A = rng.standard_normal((M, K)).astype(np.float32)   # logical A(m,k)
    B = rng.standard_normal((N, K)).astype(np.float32)   # logical B(n,k)
    A_mem = np.ascontiguousarray(A.T) if a_mn else A      # MN-major: stored [k][m]
    B_mem = np.ascontiguousarray(B.T) if b_mn else B
    a_sm, a_sk = (1, M) if a_mn else (K, 1)
    b_sn, b_sk = (1, N) if b_mn else (K, 1)
    dA, dB = _dev(L, A_mem), _dev(L, B_mem)
    out = np.zeros((M, N), np.float32)
    dC = _dev(L, out)
    ref = A.astype(np.float64) @ B.astype(np.float64).T
    bound = np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T
    for engine in (g.GEMM_TCGEN05, g.GEMM_FFMA):
        st = L.gl_matmul(dA, a_sm, a_sk, dB, b_sn, b_sk, dC, N, M, N, K, engine, 0)
        assert st == 0, L.gl_last_error()
        assert L.gl_memcpy_d2h(out.ctypes.data_as(C.c_void_p), dC, out.nbytes, 0) == 0
        err = float(np.max(np.abs(out.astype(np.float64) - ref) / bound))
        assert err <= 4e-6, "engine %d: error %.3g of sum|a||b|" % (engine, err)
    for p in (dA, dB, dC):
        L.gl_device_free(p, 0)


def _matmul_case(g, M, N, K, a_mn, b_mn, seed, positive=False):
    """One gl_matmul on the tensor-core engine against the float64 product; returns the worst error in
    units of sum_k |a||b| and the change of the per-variant launch counters."""
    L = g.lib()
    rng = np.random.default_rng(seed)
    draw = (lambda s: rng.random(s, dtype=np.float32) + 0.25) if positive else \
        (lambda s: rng.standard_normal(s, dtype=np.float32))
    A = draw((M, K))
    B = draw((N, K))
    A_mem = np.ascontiguousarray(A.T) if a_mn else A
    B_mem = np.ascontiguousarray(B.T) if b_mn else B
    a_sm, a_sk = (1, M) if a_mn else (K, 1)
    b_sn, b_sk = (1, N) if b_mn else (K, 1)
    dA, dB = _dev(L, A_mem), _dev(L, B_mem)
    out = np.full((M, N), np.nan, np.float32)
    dC = _dev(L, out)
    before = g.tc_variant_counts()
    st = L.gl_matmul(dA, a_sm, a_sk, dB, b_sn, b_sk, dC, N, M, N, K, g.GEMM_TCGEN05, 0)
    assert st == 0, L.gl_last_error()
    after = g.tc_variant_counts()
    assert L.gl_memcpy_d2h(out.ctypes.data_as(C.c_void_p), dC, out.nbytes, 0) == 0
    for p in (dA, dB, dC):
        L.gl_device_free(p, 0)
    ref = A.astype(np.float64) @ B.astype(np.float64).T
    bound = np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T
    err = float(np.max(np.abs(out.astype(np.float64) - ref) / bound))
    return err, [a - b for a, b in zip(after, before)]


# The variant the wide-MLP and inference steps run on: 256-wide tiles, persistent CTAs that walk several
# tiles each in bands of 16 row tiles, pipeline and accumulator barriers that keep counting across tiles,
# deep K.  (M, N, K, A MN-major, B MN-major, all-positive operands)
WIDE_CASES = [
    # 320 wide tiles on 148 CTAs, all four operand layouts, shallow K: the tile walk and the barrier
    # phases across tiles (2 to 3 tiles per CTA, a partial last band: 32 row tiles = 2 bands of 16)
    (4096, 2560, 256, 0, 0, False), (4096, 2560, 256, 0, 1, False), (4096, 2560, 256, 1, 1, False),
    (4096, 2560, 256, 1, 0, False),
    # row-tile count that is not a multiple of the band (24 = 16 + 8): the short last band
    (3072, 1536, 272, 0, 0, False),
    # the layer products of the wide-MLP window step at 2048 rows: forward (K-major x K-major), error
    # propagation (weights read MN-major), weight gradient (both operands MN-major, K = rows)
    (2048, 4096, 4096, 0, 0, False), (2048, 4096, 4096, 0, 1, False), (4096, 4096, 2048, 1, 1, False),
    # the first layer's gradient at the full 8192-row window: K = 8192, 128 wide tiles
    (4096, 1024, 8192, 1, 1, False),
    # all-positive operands: the worst case for the tensor core's truncating accumulation at deep K
    (2048, 2560, 4096, 0, 0, True),
    # one tile per CTA but 256 wide and deep: 80 wide tiles
    (2048, 1280, 4096, 0, 0, False),
]


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,positive", WIDE_CASES)
def test_tc_matmul_wide_persistent_variant(g, M, N, K, a_mn, b_mn, positive):
    err, dc = _matmul_case(g, M, N, K, a_mn, b_mn, seed=M + 3 * N + 7 * K + a_mn + 2 * b_mn, positive=positive)
    assert err <= 4e-6, "error %.3g of sum|a||b|" % err
    tiles = (M // 128) * (N // 256)
    assert dc[1] == 1 and dc[0] == 0, "the 256-wide instantiation did not run: %r" % (dc,)
    assert len(dc) == 5
    if tiles > 148:
        assert dc[2] == 1, "%d tiles but no CTA walked more than one" % tiles


# Shapes whose last wave of tiles leaves SMs idle: the kernel deals the k-blocks of those tiles out over all CTAs, a CTA that holds the tail of a tile stores its partial accumulators and the CTA
# that holds the head adds the partials in a fixed order and runs the epilogue.  (M, N, K, A MN-major, B MN-major)
SPLIT_CASES = [
    (1024, 4096, 1024, 0, 0),   # 128 wide tiles on 148 SMs: every CTA gets 0.86 of a tile
    (1024, 4096, 1024, 1, 1),   # the same as a weight-gradient product
    (1024, 1024, 4096, 0, 0),   # 32 wide tiles, deep k: a tile is shared by four or five CTAs
    (1024, 1024, 4096, 0, 1),
    (4096, 4096, 1024, 1, 1),   # 512 tiles: three whole waves, then 68 tiles split
    (1024, 2048, 272, 0, 0),    # 64 wide tiles, 17 k-blocks each: shares that end inside a chunk of 8 k-blocks
    (1792, 1152, 784, 0, 0),    # 128-wide tiles (1152 is no multiple of 256): 126 tiles, 49 k-blocks
]


# By default only a last wave that leaves a quarter of the SMs idle is split; these cases lower the threshold to
# a tenth so that the geometries with 0.86 of a tile per CTA (most tiles shared by two CTAs) stay covered.
@pytest.mark.parametrize("M,N,K,a_mn,b_mn", SPLIT_CASES)
def test_tc_matmul_split_last_wave(g, monkeypatch, M, N, K, a_mn, b_mn):
    monkeypatch.setenv("GLADES_TC_SPLITK_IDLE", "10")
    err, dc = _matmul_case(g, M, N, K, a_mn, b_mn, seed=5 * M + 3 * N + K + a_mn + 2 * b_mn)
    assert err <= 4e-6, "error %.3g of sum|a||b|" % err
    assert dc[4] == 1, "the last wave was not split along k: %r" % (dc,)
    # all-positive operands: partial sums of one sign, the worst case for a lost or doubled partial
    err, dc = _matmul_case(g, M, N, K, a_mn, b_mn, seed=7, positive=True)
    assert err <= 4e-6 and dc[4] == 1


def test_tc_matmul_split_rule_default(g, monkeypatch):
    """Default rule: 128 tiles on 148 SMs (13 % idle) stay whole, 32 and 68-tile last waves are split."""
    monkeypatch.delenv("GLADES_TC_SPLITK_IDLE", raising=False)
    monkeypatch.delenv("GLADES_TC_SPLITK", raising=False)
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the tile counts of this test are chosen for 148 SMs")
    for (M, N, K), split in (((1024, 4096, 1024), 0), ((1024, 1024, 4096), 1), ((4096, 4096, 512), 1)):
        err, dc = _matmul_case(g, M, N, K, 0, 0, seed=11)
        assert err <= 4e-6
        assert dc[4] == split, "M=%d N=%d K=%d: split %d, expected %d" % (M, N, K, dc[4], split)


# (M, N, K, ranks): an owner's band of 2, 1 and 8 row tiles; owners without rows; bands that do not divide the rows; 160 wide
# tiles (several per CTA) and one tile in all; a K that ends inside a chunk.
BAND_CASES = [(512, 384, 256, 2), (512, 384, 272, 4), (384, 128, 1024, 2), (128, 128, 16, 8), (2048, 2560, 512, 2), (2048, 2560, 144, 8),
              (1152, 256, 4096, 3), (256, 512, 640, 1)]


@pytest.mark.parametrize("fixed_order", [0, 1])
@pytest.mark.parametrize("M,N,K,ranks", BAND_CASES)
def test_gradient_stored_in_bands(g, M, N, K, ranks, fixed_order):
    """The data-parallel gradient of both tensor-core kernels: every row band reaches its owner's memory, whichever rank stores
    it, and nothing else is written there.  (All owners' memory is this GPU's; no rank waits for another.)"""
    L = g.lib()
    rng = np.random.default_rng(M + 3 * N + 7 * K + ranks)
    A, B = rng.standard_normal((K, M), dtype=np.float32), rng.standard_normal((K, N), dtype=np.float32)
    col, alpha = rng.standard_normal(N, dtype=np.float32), np.float32(0.05)
    band = ((M + ranks - 1) // ranks + 127) // 128 * 128
    dA, dB, dcol = _dev(L, A), _dev(L, B), _dev(L, col)
    guard = np.full((band + 1, N), np.nan, np.float32)  # a row behind every band
    bands = [_dev(L, guard) for _ in range(ranks)]
    ptrs = (C.c_void_p * ranks)(*[b.value for b in bands])
    ref = float(alpha) * (A.T.astype(np.float64) @ B.astype(np.float64)) + col
    # (the last roundings: of alpha times the sum, and of the sum with the column term)
    bound = float(alpha) * (np.abs(A).T.astype(np.float64) @ np.abs(B).astype(np.float64)) * 4e-6 + 2.0 ** -23 * (np.abs(ref) + np.abs(col))
    first = None
    for self_rank in range(ranks):
        for b in bands:
            assert L.gl_memcpy_h2d(b, guard.ctypes.data_as(C.c_void_p), guard.nbytes, 0) == 0
        before = g.tc_variant_counts()
        assert L.gl_matmul_bands(dA, 1, M, dB, 1, N, ptrs, ranks, self_rank, float(alpha), dcol, M, N, K, fixed_order, 0) == 0, L.gl_last_error()
        assert [a - b for a, b in zip(g.tc_variant_counts(), before)][3] == 1
        out = []
        for o, b in enumerate(bands):
            got = np.empty_like(guard)
            assert L.gl_memcpy_d2h(got.ctypes.data_as(C.c_void_p), b, got.nbytes, 0) == 0
            rows = max(0, min(band, M - o * band))
            assert np.all(np.isnan(got[rows:])), "owner %d: rows behind the band were written" % o
            out.append(got[:rows])
        out = np.concatenate(out)
        assert np.all(np.abs(out - ref) <= bound), "rank %d: %g of the bound" % (self_rank, float(np.max(np.abs(out - ref) / bound)))
        first = out if first is None else first
        assert np.array_equal(out.view(np.uint32), first.view(np.uint32)), "rank %d's walk over the bands gives other sums" % self_rank
    for p in [dA, dB, dcol] + bands:
        L.gl_device_free(p, 0)


@pytest.mark.parametrize("M", [32 * 65535, 32 * 65535 + 1, 64 * 65535, 64 * 65535 + 1, 96 * 65535, 96 * 65535 + 1, 128 * 65535])
def test_ffma_product_of_millions_of_rows(g, M):
    """As many rows as a grid of 32-, 64-, 96- and 128-row tiles can have, and one more, which the next larger tile takes: exact
    products of one term each."""
    L = g.lib()
    a = np.arange(M, dtype=np.float32)
    b = np.array([0.5, -3.0], np.float32)
    dA, dB, dC = _dev(L, a), _dev(L, b), _dev(L, np.zeros((M, 2), np.float32))
    assert L.gl_matmul(dA, 1, 1, dB, 1, 1, dC, 2, M, 2, 1, g.GEMM_FFMA, 0) == 0, L.gl_last_error()
    out = np.empty((M, 2), np.float32)
    assert L.gl_memcpy_d2h(out.ctypes.data_as(C.c_void_p), dC, out.nbytes, 0) == 0
    assert np.array_equal(out, a[:, None] * b[None, :])
    for p in (dA, dB, dC):
        L.gl_device_free(p, 0)


# (each tile of the fp32 product: 32, 64, 96 and 128 rows; remainders of rows, columns and k; one stage of 32 k to the four of the ring,
# one more, and many turns of it; both ways a matrix can lie, rows on and off 16-byte boundaries)
CHAIN_K = [1, 15, 17, 33, 64, 127, 129, 160, 161, 255, 784]
CHAIN_SHAPES = [(33, 65, 0), (1000, 500, 0), (999, 501, 3), (1000, 784, 0), (961, 833, 1), (1024, 1024, 0), (1025, 999, 2)]


@pytest.mark.parametrize("K", CHAIN_K)
@pytest.mark.parametrize("M,N,pad", CHAIN_SHAPES)
def test_ffma_product_is_one_chain_whatever_the_tile(g, M, N, K, pad):
    """A product against 64 bits -- a chain of K fused multiply-adds is off by at most K roundings of its partial sums -- and bit
    for bit against the same rows taken 32 at a time, which run on other tiles."""
    L = g.lib()
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = rng.standard_normal((N, K)).astype(np.float32)
    ref = A.astype(np.float64) @ B.astype(np.float64).T
    bound = K * 2.0 ** -24 * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T) + 1e-30
    for a_mn, b_mn in ((0, 0), (0, 1), (1, 1), (1, 0)):
        def lay(x, mn):
            x = x.T if mn else x
            m = np.full((x.shape[0], x.shape[1] + pad), np.nan, np.float32)
            m[:, :x.shape[1]] = x
            return m, m.shape[1]
        A_mem, lda = lay(A, a_mn)
        B_mem, ldb = lay(B, b_mn)
        dA, dB, dC = _dev(L, A_mem), _dev(L, B_mem), _dev(L, np.full((M, N), np.nan, np.float32))
        strides = ((1, lda) if a_mn else (lda, 1)) + ((1, ldb) if b_mn else (ldb, 1))

        def product(r0, rows):
            a = C.c_void_p(dA.value + 4 * r0 * strides[0])
            assert L.gl_matmul(a, strides[0], strides[1], dB, strides[2], strides[3], dC, N, rows, N, K, g.GEMM_FFMA, 0) == 0, L.gl_last_error()
            out = np.empty((rows, N), np.float32)
            assert L.gl_memcpy_d2h(out.ctypes.data_as(C.c_void_p), dC, out.nbytes, 0) == 0
            return out
        whole = product(0, M)
        assert np.all(np.abs(whole - ref) <= bound), float(np.max(np.abs(whole - ref) / bound))
        for r0 in (0, 32, M - M % 32 if M % 32 else M - 32):
            rows = min(32, M - r0)
            assert np.array_equal(product(r0, rows), whole[r0:r0 + rows])
        for p in (dA, dB, dC):
            L.gl_device_free(p, 0)


# (operands that are contiguous neither way, and one contiguous way beside one that is not; a single row or term at any stride)
@pytest.mark.parametrize("M,N,K", [(33, 65, 17), (1, 70, 130), (130, 1, 33), (70, 40, 1), (1000, 500, 300), (1024, 1024, 161)])
@pytest.mark.parametrize("steps", [(2, 3), (1, 5), (4, 1), (4, 4)])
def test_ffma_product_of_any_strides(g, M, N, K, steps):
    """Every steps[0]-th / steps[1]-th element of what lies in memory, k or m / n outermost: bit for bit the product of the same operands
    laid out densely."""
    L = g.lib()
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)

    def product(a, sa, b, sb):
        dA, dB, dC = _dev(L, a), _dev(L, b), _dev(L, np.full((M, N), np.nan, np.float32))
        assert L.gl_matmul(dA, sa[0], sa[1], dB, sb[0], sb[1], dC, N, M, N, K, g.GEMM_FFMA, 0) == 0, L.gl_last_error()
        out = np.empty((M, N), np.float32)
        assert L.gl_memcpy_d2h(out.ctypes.data_as(C.c_void_p), dC, out.nbytes, 0) == 0
        for p in (dA, dB, dC):
            L.gl_device_free(p, 0)
        return out

    def lay(x, step, turned):
        x = x.T if turned else x
        m = np.full((x.shape[0], x.shape[1] * step + 1), np.nan, np.float32)
        m[:, :x.shape[1] * step:step] = x
        return m, (step, m.shape[1]) if turned else (m.shape[1], step)

    dense = product(np.ascontiguousarray(A.T), (1, M), np.ascontiguousarray(B.T), (1, N))
    bound = K * 2.0 ** -24 * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64).T) + 1e-30
    assert np.all(np.abs(dense - A.astype(np.float64) @ B.astype(np.float64).T) <= bound)
    for a_turned in (False, True):
        for b_turned in (False, True):
            out = product(*lay(A, steps[0], a_turned), *lay(B, steps[1], b_turned))
            assert np.array_equal(out.view(np.uint32), dense.view(np.uint32)), (a_turned, b_turned)


def test_gradient_bands_refuse_what_cannot_be_stored(g):
    L = g.lib()
    a = _dev(L, np.zeros((256, 256), np.float32))
    ptrs = (C.c_void_p * 2)(a.value, a.value)
    for ranks, self_rank, M, N, K in ((2, 2, 256, 128, 32), (9, 0, 256, 128, 32), (0, 0, 256, 128, 32), (2, 0, 200, 128, 32), (2, 0, 256, 100, 32),
                                      (2, 0, 256, 128, 24)):
        for fixed_order in (0, 1):
            assert L.gl_matmul_bands(a, 1, M, a, 1, N, ptrs, ranks, self_rank, 1.0, None, M, N, K, fixed_order, 0) != 0
    L.gl_device_free(a, 0)


def test_tc_matmul_rejects_odd_shapes(g):
    L = g.lib()
    a = np.zeros((100, 32), np.float32)
    dA, dB, dC = _dev(L, a), _dev(L, a), _dev(L, np.zeros((100, 100), np.float32))
    assert L.gl_matmul(dA, 32, 1, dB, 32, 1, dC, 100, 100, 100, 32, g.GEMM_TCGEN05, 0) != 0
    assert L.gl_matmul(dA, 32, 1, dB, 32, 1, dC, 100, 100, 100, 32, g.GEMM_FFMA, 0) == 0
    for p in (dA, dB, dC):
        L.gl_device_free(p, 0)


@pytest.mark.parametrize("momentum,head", [(0.0, "softmax"), (0.9, "sigmoid")])
def test_batched_window_on_tensor_cores_vs_restatement(g, oracle, momentum, head):
    """A whole window step (forward, error propagation, weight gradient, update) with every layer
    product on the tcgen05 kernel, against the double-accumulating CPU restatement."""
    rng = np.random.default_rng(17)
    sizes = [128, 256, 384, 128]
    rows = 256
    out_type = "classification"
    d = g.make_desc(sizes, ["relu", "tanh", head], out_type, batch=rows, lr=0.05, momentum=momentum,
                    mode=g.MODE_BATCHED, gemm=g.GEMM_TCGEN05)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    if head == "softmax":
        y = np.zeros((rows, sizes[-1]), np.float32)
        y[np.arange(rows), rng.integers(0, sizes[-1], rows)] = 1.0
    else:
        y = rng.uniform(0.05, 0.95, (rows, sizes[-1])).astype(np.float32)
    nw = sum(sizes[i] * sizes[i + 1] for i in range(3))
    w = (rng.standard_normal(nw) * 0.05).astype(np.float32)
    b = np.array([0.02, -0.03], np.float32)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    for step in range(2):
        m = net.train_window(0, rows)
        gr = S.window_grad(0, rows)
        S.window_apply(gr, rows)
        wg, bg = net.get_weights()
        ws, bs = S.get_weights()
        err = float(np.max(np.abs(wg.astype(np.float64) - ws)) / np.max(np.abs(ws)))
        assert err <= 1e-5, "step %d: weights rel err %g" % (step, err)
        assert np.allclose(bg, bs, rtol=1e-4, atol=1e-6)
        assert abs(m.total_error - gr[-2]) <= 1e-5 * max(1.0, abs(gr[-2]))
    # 3 forward + 2 error-propagation + 3 gradient products per step, all on tensor cores
    assert net.tensor_core_launches() == 16
    # inference from identical weights (the two sides' weights differ by the step tolerance above)
    wg, bg = net.get_weights()
    S.set_weights(wg, bg)
    out_g, am_g, _ = net.forward(0, rows)
    out_s, am_s = S.forward_block(0, rows)
    assert np.max(np.abs(out_g - out_s)) <= 1e-5 * max(1.0, float(np.max(np.abs(out_s))))
    assert np.array_equal(am_g, am_s)
    net.close()


def _rows_clear_of_relu_threshold(rng, draw, x, W0, W1, b1, margin=1e-5):
    """The reference's ReLU is discontinuous: 0 below 0.046, the identity above (GMath/gmath.cpp:62-68).  A
    hidden pre-activation within fp32 rounding of 0.046 may fall on either side in two correct fp32
    evaluations, and the two then differ by far more than any rounding tolerance.  So that the comparisons
    below measure the kernels and not that coin toss, rows with a pre-activation of either hidden layer
    within `margin` of the threshold (float64 evaluation) are drawn again until none is left."""
    W0 = W0.astype(np.float64)
    W1 = W1.astype(np.float64)
    todo = np.arange(x.shape[0])
    for _ in range(100):
        z1 = x[todo].astype(np.float64) @ W0.T
        z2 = np.where(z1 < 0.046, 0.0, z1) @ W1.T + float(b1)
        bad = np.any(np.abs(z1 - 0.046) < margin, axis=1) | np.any(np.abs(z2 - 0.046) < margin, axis=1)
        todo = todo[bad]
        if todo.size == 0:
            return x
        x[todo] = draw(todo.size)
    raise AssertionError("could not clear the rows of the ReLU threshold")


def _onehot(rows, n, labels):
    y = np.zeros((rows, n), np.float32)
    y[np.arange(rows), labels] = 1.0
    return y


@pytest.mark.parametrize("sizes,acts,window,grad,bands", [
    # jumps, from 4096 rows of the WINDOW on: 3xFP16 backward products
    ([1024, 4096, 4096, 1024], "relu", 8192, 2, 1), ([1024, 4096, 4096, 1024], "relu", 4096, 2, 1), ([784, 1000, 500, 10], "relu", 8192, 2, 0),
    # below: the fixed order, whose gradients leave in bands too
    ([1024, 4096, 4096, 1024], "relu", 3968, 1, 1), ([1024, 4096, 4096, 1024], "relu", 3072, 1, 1), ([512, 2560, 2048, 256], "relu", 1024, 1, 1),
    # no jumps: 3xFP16 at any size
    ([1024, 4096, 4096, 1024], "tanh", 1024, 2, 1)])
def test_engines_of_a_window_do_not_depend_on_the_number_of_gpus(g, sizes, acts, window, grad, bands):
    net = g.Net(g.make_desc(sizes, [acts] * (len(sizes) - 2) + ["softmax"], "classification", batch=window, mode=g.MODE_BATCHED))
    one = net.plan_window(window, window)
    assert np.all(one[:, 2] == grad) and np.all(one[1:, 1] == grad) and one[0, 1] == -1 and np.all(one[:, 3] == bands), one
    for ranks in (2, 4, 8):
        if window % (128 * ranks) == 0:
            assert np.array_equal(net.plan_window(window // ranks, window), one), ranks
    net.close()


@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_windows_on_inputs_off_16_byte_boundaries(g, oracle, momentum):
    """Inputs that begin off a 16-byte boundary keep the first layer's products off the bulk-copy kernels: training windows on
    them, then inference on an aligned copy under the weights they left, against the restatement."""
    rng = np.random.default_rng(29)
    sizes, rows = [128, 256, 128], 256
    d = g.make_desc(sizes, ["relu", "softmax"], "classification", batch=rows, lr=0.05, momentum=momentum, mode=g.MODE_BATCHED,
                    gemm=g.GEMM_TCGEN05)
    w = np.concatenate([rng.uniform(-1, 1, sizes[i] * sizes[i + 1]).astype(np.float32) / np.float32(np.sqrt(sizes[i])) for i in range(2)])
    b = np.array([0.02], np.float32)
    W0 = w[:sizes[0] * sizes[1]].reshape(sizes[1], sizes[0])
    x = _rows_clear_of_relu_threshold(rng, lambda k: rng.standard_normal((k, sizes[0]), dtype=np.float32),
                                      rng.standard_normal((rows, sizes[0]), dtype=np.float32), W0, np.zeros((1, sizes[1])), 1.0)
    y = _onehot(rows, sizes[-1], rng.integers(0, sizes[-1], rows))
    L = g.lib()
    aligned, dy = _dev(L, x), _dev(L, y)
    off = _dev(L, np.concatenate([np.zeros(1, np.float32), x.ravel()]))
    net = g.Net(d)
    net.set_weights(w, b)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    net.set_data_device(off.value + 4, dy.value, rows)
    net.train_window(0, rows)
    S.window_apply(S.window_grad(0, rows), rows)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    assert np.max(np.abs(wg - ws)) <= 1e-5 * np.max(np.abs(ws)) and np.allclose(bg, bs, rtol=1e-4, atol=1e-6)
    net.set_data_device(aligned.value, dy.value, rows)
    out_g, am_g, _ = net.forward(0, rows)
    S.set_weights(wg, bg)
    out_s, am_s = S.forward_block(0, rows)
    assert np.max(np.abs(out_g - out_s)) <= 1e-5 and np.array_equal(am_g, am_s)
    net.close()
    S.close()
    for p in (aligned, dy, off):
        L.gl_device_free(p, 0)


def test_wide_mlp_small_window_vs_restatement(g, oracle):
    """One batched-mode window of the wide-MLP student itself (1024-4096-4096-1024, ReLU/ReLU/softmax,
    cross-entropy, lr 1e-2, weights U(+-1/sqrt(n_in))) on 1024 rows, against the double-accumulating CPU
    restatement: loss, every updated weight within 1e-5 of the largest weight, identical predicted
    classes.  At this size every layer product runs on the 3xTF32 kernel, on 256-wide persistent tiles, several
    tiles per CTA for the 4096 x 4096 gradient.  The rows are drawn so that no hidden pre-activation lies
    within 1e-5 of the discontinuity of the reference's ReLU."""
    sizes = [1024, 4096, 4096, 1024]
    rows = 1024
    rng = np.random.default_rng(404)
    x = rng.standard_normal((rows, sizes[0]), dtype=np.float32)
    y = _onehot(rows, sizes[-1], rng.integers(0, sizes[-1], rows))
    w = np.concatenate([rng.uniform(-1, 1, sizes[i] * sizes[i + 1]).astype(np.float32) / np.float32(np.sqrt(sizes[i]))
                        for i in range(3)])
    b = np.array([0.01, -0.02], np.float32)
    n01, n12 = sizes[0] * sizes[1], sizes[1] * sizes[2]
    x = _rows_clear_of_relu_threshold(rng, lambda k: rng.standard_normal((k, sizes[0]), dtype=np.float32), x,
                                      w[:n01].reshape(sizes[1], sizes[0]), w[n01:n01 + n12].reshape(sizes[2], sizes[1]), b[0])
    d = g.make_desc(sizes, ["relu", "relu", "softmax"], "classification", batch=rows, lr=1e-2, mode=g.MODE_BATCHED)
    net = g.Net(d)
    net.set_weights(w, b)
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, b)
    before, engines = g.tc_variant_counts(), g.tc_engine_counts()
    m = net.train_window(0, rows)
    dc = [a - c for a, c in zip(g.tc_variant_counts(), before)]
    assert dc[1] >= 6 and dc[2] >= 1, "expected the 256-wide persistent variant, saw %r" % (dc,)
    assert [a - c for a, c in zip(g.tc_engine_counts(), engines)] == [0, 8]
    gr = S.window_grad(0, rows)
    S.window_apply(gr, rows)
    wg, bg = net.get_weights()
    ws, bs = S.get_weights()
    lo = 0
    for l in range(3):
        hi = lo + sizes[l] * sizes[l + 1]
        scale = float(np.max(np.abs(ws[lo:hi])))
        assert np.max(np.abs(wg[lo:hi].astype(np.float64) - ws[lo:hi])) <= 1e-5 * scale, "layer %d weights" % l
        # the update itself (new - old) carries the whole gradient: within 1e-3 of its largest entry plus the
        # rounding of the stored weight on both sides (the update is 1e-4 of the weight), 1e-4 on average
        ug = wg[lo:hi].astype(np.float64) - w[lo:hi]
        us = ws[lo:hi].astype(np.float64) - w[lo:hi]
        ulp = float(np.spacing(np.float32(scale)))
        assert np.max(np.abs(ug - us)) <= 1e-3 * np.max(np.abs(us)) + 2 * ulp, "layer %d update" % l
        assert np.mean(np.abs(ug - us)) <= 1e-4 * np.max(np.abs(us)) + ulp, "layer %d update, mean" % l
        lo = hi
    assert np.allclose(bg, bs, rtol=1e-4, atol=1e-7)
    assert abs(m.total_error - gr[-2]) <= 1e-5 * max(1.0, abs(gr[-2]))
    # predictions from identical weights: same classes for every row
    S.set_weights(wg, bg)
    out_g, am_g, _ = net.forward(0, rows)
    out_s, am_s = S.forward_block(0, rows)
    assert np.max(np.abs(out_g - out_s)) <= 1e-5 * max(1.0, float(np.max(np.abs(out_s))))
    assert np.array_equal(am_g, am_s)
    net.close()
    S.close()


# (rows of the window, products on 3xFP16 and on 3xTF32): the last window of whole tiles whose every product keeps the fixed
# order, the first with 3xFP16 backward products, and the next; rows that are no whole tile, whose hidden layers run on fp32
# multiply-adds, on both sides of that line.
RELU_WINDOWS = [(3968, 0, 8), (4096, 6, 2), (4224, 6, 2), (4095, 0, 0), (4100, 6, 0)]


@pytest.mark.parametrize("momentum", [0.0, 0.9])
@pytest.mark.parametrize("rows,f16,tf32", RELU_WINDOWS)
def test_relu_windows_around_the_3xfp16_line_vs_restatement(g, oracle, rows, f16, tf32, momentum):
    """Windows of a network with jumps around the size from which their backward products run on the 3xFP16 kernel.  On that
    side: forward products on 3xTF32 that leave fp16 parts, error propagation through ReLU bits, momentum-weighted deltas, updates
    that leave the new weights' fp16 and low TF32 parts -- which the second window starts from.  Both windows against the
    double-accumulating restatement from the weights that the device holds; rows clear of the ReLU's jump."""
    sizes = [128, 256, 384, 128]
    rng = np.random.default_rng(rows)
    draw = lambda k: rng.standard_normal((k, sizes[0]), dtype=np.float32)  # noqa: E731
    y = _onehot(rows, sizes[-1], rng.integers(0, sizes[-1], rows))
    w = np.concatenate([rng.uniform(-1, 1, sizes[i] * sizes[i + 1]).astype(np.float32) / np.float32(np.sqrt(sizes[i])) for i in range(3)])
    b = np.array([0.01, -0.02], np.float32)
    d = g.make_desc(sizes, ["relu", "relu", "softmax"], "classification", batch=rows, lr=1e-2, momentum=momentum, mode=g.MODE_BATCHED,
                    gemm=g.GEMM_TCGEN05)
    net = g.Net(d)
    net.set_weights(w, b)
    n01, n12 = sizes[0] * sizes[1], sizes[1] * sizes[2]
    for step in range(2):
        x = _rows_clear_of_relu_threshold(rng, draw, draw(rows), w[:n01].reshape(sizes[1], sizes[0]), w[n01:n01 + n12].reshape(sizes[2], sizes[1]), b[0])
        net.set_data(x, y)
        S = oracle.Restate(d, x, y, g.Metrics)
        S.set_weights(w, b)
        before = g.tc_engine_counts()
        m = net.train_window(0, rows)
        assert [a - c for a, c in zip(g.tc_engine_counts(), before)] == [f16, tf32]
        gr = S.window_grad(0, rows)
        S.window_apply(gr, rows)
        wg, bg = net.get_weights()
        ws, bs = S.get_weights()
        S.close()
        lo = 0
        for l in range(3):
            hi = lo + sizes[l] * sizes[l + 1]
            scale = float(np.max(np.abs(ws[lo:hi])))
            assert np.max(np.abs(wg[lo:hi].astype(np.float64) - ws[lo:hi])) <= 1e-5 * scale, "step %d, layer %d weights" % (step, l)
            ug, us = wg[lo:hi].astype(np.float64) - w[lo:hi], ws[lo:hi].astype(np.float64) - w[lo:hi]
            ulp = float(np.spacing(np.float32(scale)))
            assert np.max(np.abs(ug - us)) <= 1e-3 * np.max(np.abs(us)) + 2 * ulp, "step %d, layer %d update" % (step, l)
            lo = hi
        assert np.allclose(bg, bs, rtol=1e-4, atol=1e-7)
        assert abs(m.total_error - gr[-2]) <= 1e-5 * max(1.0, abs(gr[-2]))
        w, b = wg, bg
    net.close()


def test_wide_mlp_window_on_the_benchmarked_variant_vs_64_bits(g):
    """One 8192-row window of the wide-MLP student, the benchmark's step (forward products on 3xTF32, the others on 3xFP16, 256-wide
    persistent tiles), against the same step in 64 bits: every updated weight within 1e-5 of its layer's largest, the update itself
    as in the small window's test.  Rows clear of the ReLU's jump."""
    import torch
    dev, f64 = "cuda:0", torch.float64
    sizes, rows, lr, th = [1024, 4096, 4096, 1024], 8192, 1e-2, float(np.float32(0.046))
    gen = torch.Generator(device=dev).manual_seed(606)
    w = [(torch.rand(o, i, generator=gen, device=dev) * 2 - 1) / float(np.sqrt(i)) for i, o in zip(sizes, sizes[1:])]
    b = torch.tensor([0.01, -0.02], device=dev)
    W, B = [a.to(f64) for a in w], b.to(f64)
    x = torch.randn(rows, sizes[0], generator=gen, device=dev)
    labels = torch.randint(0, sizes[-1], (rows,), generator=gen, device=dev)
    todo = torch.arange(rows, device=dev)
    for _ in range(100):
        z1 = x[todo].to(f64) @ W[0].T
        z2 = torch.where(z1 < th, 0.0, z1) @ W[1].T + B[0]
        todo = todo[((z1 - th).abs() < 1e-5).any(1) | ((z2 - th).abs() < 1e-5).any(1)]
        if todo.numel() == 0:
            break
        x[todo] = torch.randn(todo.numel(), sizes[0], generator=gen, device=dev)
    assert todo.numel() == 0
    y = torch.nn.functional.one_hot(labels, sizes[-1]).to(torch.float32)
    d = g.make_desc(sizes, ["relu", "relu", "softmax"], "classification", batch=rows, lr=lr, mode=g.MODE_BATCHED)
    net = g.Net(d)
    w0 = torch.cat([a.reshape(-1) for a in w])
    net.set_weights(w0.cpu().numpy(), b.cpu().numpy())
    net.set_data_device(x.data_ptr(), y.data_ptr(), rows)
    torch.cuda.synchronize()
    before, engines = g.tc_variant_counts(), g.tc_engine_counts()
    m = net.train_window(0, rows)
    dc = [a - c for a, c in zip(g.tc_variant_counts(), before)]
    assert dc[1] == 8 and dc[2] >= 6, "expected 256-wide persistent tiles, saw %r" % (dc,)
    assert [a - c for a, c in zip(g.tc_engine_counts(), engines)] == [6, 2]
    wg, bg = net.get_weights()
    net.close()
    A = [x.to(f64)]
    for l in range(3):
        z = A[l] @ W[l].T + (B[l - 1] if l else 0.0)
        A.append(torch.where(z < th, 0.0, z) if l < 2 else torch.softmax(z, 1))
    loss = float(-torch.log(A[3].gather(1, labels[:, None])).sum() / (rows * sizes[-1]))
    D = A[3] - y
    at = w0.numel()
    for l in (2, 1, 0):
        G = lr / rows * (D.T @ A[l])
        if l:
            assert abs(float(bg[l - 1] - (B[l - 1] - lr / rows * D.sum()))) <= 1e-7 + 1e-4 * abs(float(bg[l - 1]))
        new = (W[l] - G).reshape(-1)
        got = torch.from_numpy(wg[at - new.numel():at]).to(dev).to(f64)
        scale, big = float(new.abs().max()), float(G.abs().max())
        ulp = float(np.spacing(np.float32(scale)))
        assert float((got - new).abs().max()) <= 1e-5 * scale, "layer %d weights" % l
        assert float((got - new).abs().max()) <= 1e-3 * big + 2 * ulp and float((got - new).abs().mean()) <= 1e-4 * big + ulp, "layer %d update" % l
        at -= new.numel()
        D = (D @ W[l]) * (A[l] != 0)
    assert abs(m.total_error - loss) <= 1e-5 * max(1.0, loss)


def test_inference_net_forward_on_the_benchmarked_variant_vs_restatement(g, oracle):
    """Forward pass of the batched-inference net (784-2048-2048-10, ReLU/ReLU/softmax, weights
    U(-0.05, 0.05), rows U(0,1)) on 2048 rows against the restatement: probabilities within 1e-5 and the
    same predicted class for every row.  The two hidden products run on the 256-wide tiles.  Rows are drawn
    clear of the discontinuity of the reference's ReLU (see _rows_clear_of_relu_threshold)."""
    sizes = [784, 2048, 2048, 10]
    rows = 2048
    rng = np.random.default_rng(505)
    x = rng.random((rows, sizes[0]), dtype=np.float32)
    y = np.full((rows, sizes[-1]), 0.01, np.float32)
    nw = sum(sizes[i] * sizes[i + 1] for i in range(3))
    w = rng.uniform(-0.05, 0.05, nw).astype(np.float32)
    n01, n12 = sizes[0] * sizes[1], sizes[1] * sizes[2]
    x = _rows_clear_of_relu_threshold(rng, lambda k: rng.random((k, sizes[0]), dtype=np.float32), x,
                                      w[:n01].reshape(sizes[1], sizes[0]), w[n01:n01 + n12].reshape(sizes[2], sizes[1]), 0.01)
    d = g.make_desc(sizes, ["relu", "relu", "softmax"], "classification", batch=rows, lr=0.0, mode=g.MODE_BATCHED)
    net = g.Net(d)
    net.set_weights(w, np.array([0.01, 0.02], np.float32))
    net.set_data(x, y)
    S = oracle.Restate(d, x, y, g.Metrics)
    S.set_weights(w, np.array([0.01, 0.02], np.float32))
    before = g.tc_variant_counts()
    out_g, am_g, _ = net.forward(0, rows)
    dc = [a - c for a, c in zip(g.tc_variant_counts(), before)]
    assert dc[1] == 2, "the two hidden products should run on 256-wide tiles, saw %r" % (dc,)
    out_s, am_s = S.forward_block(0, rows)
    assert np.max(np.abs(out_g - out_s)) <= 1e-5
    diff = np.nonzero(am_g != am_s)[0]
    # a row may only differ where its two best classes tie within the tolerance
    for r in diff:
        top = np.sort(out_s[r])[-2:]
        assert top[1] - top[0] <= 2e-5, "row %d: classes differ with a margin of %g" % (r, top[1] - top[0])
    assert diff.size == 0 or diff.size <= 2
    net.close()
    S.close()
