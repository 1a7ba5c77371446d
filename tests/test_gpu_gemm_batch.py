"""The tensor-core GEMM of decode batches (17 to 64 rows, and fewer when the mode is asked for): clusters of one to six
CTAs that share a K loop, one and several rounds of 128-row tiles, rings of an odd and an even number of slots, short
last units, and calls whose weights differ in type and in cluster size."""
import numpy as np
import pytest

import oracle
import plan_shim

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SEED = 299792458
# Both operands are rounded to f16 (relative error <= 2^-11 per element, about 2^-11 / sqrt(3) rms each),
# the sub-block scale and min of the weight once more: about 2^-11 in the result, 4 x that allowed.
TOL = 4 * 2.0 ** -11


@pytest.fixture(scope="module")
def tq():
    import tur_b200
    return tur_b200


def make_weight(dt, n, k, seed):
    rng = np.random.default_rng(seed)
    rows = (rng.standard_normal((min(n, 2048), k)) * 0.02).astype(np.float32)
    w = oracle.quantize(dt, rows).reshape(len(rows), -1)
    return np.ascontiguousarray(w[np.arange(n) % len(rows)]).reshape(-1), rows.shape[0]


# (type, rows, columns, CTAs per cluster on a B200)
SHAPES = [(oracle.Q4_K, 19000, 256, 1), (oracle.Q8_0, 24300, 320, 1), (oracle.Q4_K, 12200, 4096, 2), (oracle.Q5_K, 700, 1024, 2),
          (oracle.Q6_K, 5000, 6144, 3), (oracle.Q5_K, 8100, 5120, 4), (oracle.Q8_0, 300, 2624, 4), (oracle.Q4_K, 3130, 6400, 5),
          (oracle.Q6_K, 2560, 8192, 6), (oracle.Q8_0, 130, 6208, 5), (oracle.Q8_0, 130, 6464, 6)]


@pytest.mark.parametrize("dt,n,k,c", SHAPES)
def test_clusters_share_the_k_loop(tq, dt, n, k, c):
    """Sums of every cluster size against the f64 product; the bits do not depend on the batch, nor on what ran before."""
    assert plan_shim.cluster(n, k) == c
    w, base = make_weight(dt, n, k, SEED + 8000 + n + k)
    rng = np.random.default_rng(SEED + 8001 + n)
    x = (rng.standard_normal((64, k)) * 2.0 ** rng.integers(-8, 9, (64, 1))).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))
    xd = torch.from_numpy(x).cuda()
    y = mm.forward(xd, mode=tq.Mode.TENSOR_CORE)
    ref = oracle.matmul_f64(dt, w[: w.size // n * base], base, k, x)
    got = y.cpu().numpy().astype(np.float64)
    idx = np.arange(n) % base
    err = np.linalg.norm(got - ref[:, idx], axis=1) / np.linalg.norm(ref[:, idx], axis=1)  # row by row: the magnitudes differ
    assert err.max() < TOL, (int(err.argmax()), err.max())
    for m in (1, 16, 17, 24, 33, 48, 56, 63):
        assert torch.equal(mm.forward(xd[:m], mode=tq.Mode.TENSOR_CORE), y[:m]), m
    assert torch.equal(mm.forward(xd, mode=tq.Mode.TENSOR_CORE), y)
    tq.context().poll_status()


@pytest.mark.parametrize("m", [20, 64])
def test_one_call_of_several_types_and_cluster_sizes(tq, m):
    """Q4_K, Q5_K and Q6_K weights whose items share a launch, and one that wants another cluster size: the bits of the separate calls."""
    k = 2048
    shapes = [(oracle.Q4_K, 2048), (oracle.Q6_K, 520), (oracle.Q5_K, 1000), (oracle.Q4_K, 9000)]
    mms = [tq.QMatMul.from_arc(tq.QTensor.new(make_weight(t, n, k, SEED + 8100 + n)[0], tq.GgmlDType(t), (n, k))) for t, n in shapes]
    x = torch.from_numpy(np.random.default_rng(SEED + 8101).standard_normal((m, k)).astype(np.float32)).cuda()
    bias = torch.from_numpy(np.random.default_rng(SEED + 8102).standard_normal(520).astype(np.float32)).cuda()
    want = [mm.forward(x, bias=bias if i == 1 else None, mode=tq.Mode.TENSOR_CORE) for i, mm in enumerate(mms)]
    for _ in range(3):
        got = tq.QMatMul.forward_multi(mms, x, biases=[None, bias, None, None], mode=tq.Mode.TENSOR_CORE)
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    l0 = tq.context().launch_count()
    tq.QMatMul.forward_multi(mms[:3], x, mode=tq.Mode.TENSOR_CORE)
    assert tq.context().launch_count() - l0 == 2          # one conversion, one GEMM
    tq.context().poll_status()


@pytest.mark.parametrize("k,dtype", [(256, torch.float32), (5120, torch.bfloat16), (16640, torch.float32), (33024, torch.bfloat16)])
def test_one_call_of_both_k_orders(tq, k, dtype):
    """Q6_K (in an order of its own where K is cut, which 256 columns are not) beside Q4_K: rows converted by one CTA and by several."""
    rng = np.random.default_rng(SEED + 8200 + k)
    ws = [(t, *make_weight(t, n, k, SEED + 8201 + n)) for t, n in ((oracle.Q4_K, 150), (oracle.Q6_K, 130))]
    mms = [tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(t), (n, k))) for t, w, n in ws]
    x = torch.from_numpy(rng.standard_normal((33, k)).astype(np.float32)).to(dtype).cuda()
    got = tq.QMatMul.forward_multi(mms, x, mode=tq.Mode.TENSOR_CORE)
    for (t, w, n), mm, y in zip(ws, mms, got):
        ref = oracle.matmul_f64(t, w, n, k, x.float().cpu().numpy())
        assert np.linalg.norm(y.double().cpu().numpy() - ref) / np.linalg.norm(ref) < TOL
        assert torch.equal(mm.forward(x, mode=tq.Mode.TENSOR_CORE), y)
    tq.context().poll_status()


# (type, rows, columns, activation rows, rows of a tile): tiles of 16 to 128 rows, whole and ragged, narrow and wide accumulators,
# one item per CTA and several, a last unit of one, two and three 64-k blocks
TILED = [(oracle.Q4_K, 700, 256, 1024, 48), (oracle.Q8_0, 300, 320, 67, 16), (oracle.Q8_0, 5000, 448, 300, 112), (oracle.Q4_K, 4000, 4096, 65, 32),
         (oracle.Q5_K, 3000, 5120, 129, 32), (oracle.Q6_K, 5000, 6144, 300, 112), (oracle.Q8_0, 130, 2624, 96, 16), (oracle.Q6_K, 2560, 1024, 700, 112),
         (oracle.Q8_0, 8200, 704, 255, 128), (oracle.Q4_K, 12288, 512, 128, 128)]


@pytest.mark.parametrize("dt,n,k,m,rows", TILED)
def test_short_prompts_in_tiles(tq, dt, n, k, m, rows):
    """65 to 1024 rows in tiles: against the f64 product, and with the bits of a call that is too large for tiles."""
    assert plan_shim.tile([n], m) == rows and plan_shim.kernel([n], 1024 // m * m + m) == "pairs"
    w, base = make_weight(dt, n, k, SEED + 8300 + n + k)
    rng = np.random.default_rng(SEED + 8301 + n)
    x = (rng.standard_normal((m, k)) * 2.0 ** rng.integers(-8, 9, (m, 1))).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))
    xd = torch.from_numpy(x).cuda()
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    y = mm.forward(xd, mode=tq.Mode.TENSOR_CORE)
    ref = oracle.matmul_f64(dt, w[: w.size // n * base], base, k, x)[:, np.arange(n) % base]
    err = np.linalg.norm(y.double().cpu().numpy() - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < TOL, (int(err.argmax()), err.max())
    assert torch.equal(mm.forward(torch.cat([xd] * (1024 // m + 1)), mode=tq.Mode.TENSOR_CORE)[:m], y)
    a, b = tq.QMatMul.forward_multi([mm, mm], xd, biases=[None, bias], mode=tq.Mode.TENSOR_CORE)
    assert torch.equal(a, y) and torch.equal(b, y + bias)
    tq.context().poll_status()


@pytest.mark.parametrize("k,few,many", [(16640, 140, 150), (33024, 70, 1100)])
def test_long_rows_convert_alike_by_clusters_and_alone(tq, k, few, many):
    """Few rows are converted by clusters of CTAs, many by a CTA each: the same f16 operand and the same bits, into images of
    tiles (up to 1024 rows) and into rows."""
    w, _ = make_weight(oracle.Q4_K, 130, k, SEED + 8400 + k)
    rng = np.random.default_rng(SEED + 8401 + k)
    x = (rng.standard_normal((many, k)) * 2.0 ** rng.integers(-8, 9, (many, 1))).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(oracle.Q4_K), (130, k)))
    xd = torch.from_numpy(x).cuda()
    y = mm.forward(xd, mode=tq.Mode.TENSOR_CORE)
    assert torch.equal(mm.forward(xd[:few], mode=tq.Mode.TENSOR_CORE), y[:few])
    rows = np.r_[0:20, many - 20:many]
    ref = oracle.matmul_f64(oracle.Q4_K, w, 130, k, x[rows])
    err = np.linalg.norm(y.cpu().numpy()[rows] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < TOL, (int(err.argmax()), err.max())
    tq.context().poll_status()
