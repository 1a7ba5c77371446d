"""The tensor-core GEMMs at the sizes where their tiling can go wrong: weight rows around the 256-row
pair tile, activation rows around the 16-row granularity and the limits of 64 and 1024 rows, K loops of
one to a few 256-wide units with a short last one, decode batches of one and several rounds, and calls of several weights
that run side by side. Which kernel a case reaches is asked of the launch plan, so that a rule that moves does not take
a kernel's cases along unnoticed."""
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
    w = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    return oracle.quantize(dt, w)


K_QUANT = [(oracle.Q4_K, 256), (oracle.Q5_K, 512), (oracle.Q6_K, 768)]


@pytest.mark.parametrize("n", [1, 16, 255, 257, 400])
@pytest.mark.parametrize("m,kernel", [(17, "batch"), (48, "batch"), (64, "batch"), (65, "tiles"), (129, "tiles"), (257, "tiles"),
                                      (1025, "pairs"), (1300, "pairs")])
@pytest.mark.parametrize("dt,k", K_QUANT + [(oracle.Q8_0, 64), (oracle.Q8_0, 320), (oracle.Q8_0, 704)])
def test_edges_of_the_pair_tile(tq, dt, k, n, m, kernel):
    assert plan_shim.kernel([n], m) == kernel
    w = make_weight(dt, n, k, SEED + 7000 + n + k)
    rng = np.random.default_rng(SEED + 7001 + m)
    x = rng.standard_normal((m, k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))
    y = mm.forward(torch.from_numpy(x).cuda(), bias=torch.from_numpy(bias).cuda(), mode=tq.Mode.TENSOR_CORE)
    assert oracle.rel_fro(y.cpu().numpy(), oracle.matmul_f64(dt, w, n, k, x) + bias) < TOL
    tq.context().poll_status()


@pytest.mark.parametrize("dt,n,k", [(oracle.Q4_K, 10000, 768), (oracle.Q6_K, 19000, 256), (oracle.Q8_0, 9700, 320),
                                    (oracle.Q8_0, 40000, 64), (oracle.Q5_K, 300, 8192), (oracle.Q8_0, 512, 4160)])
def test_decode_batches_share_the_k_loop(tq, dt, n, k):
    """One and several rounds of tiles, K loops of one unit and cut ones; a second call has the same bits, and a row's bits do not
    depend on the batch."""
    w = make_weight(dt, n, k, SEED + 7100 + n + k)
    x = np.random.default_rng(SEED + 7101).standard_normal((64, k)).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))
    xd = torch.from_numpy(x).cuda()
    y = mm.forward(xd, mode=tq.Mode.TENSOR_CORE)
    assert oracle.rel_fro(y.cpu().numpy(), oracle.matmul_f64(dt, w, n, k, x)) < TOL
    assert torch.equal(mm.forward(xd, mode=tq.Mode.TENSOR_CORE), y)
    assert torch.equal(mm.forward(xd[:21], mode=tq.Mode.TENSOR_CORE), y[:21])
    tq.context().poll_status()


@pytest.fixture(scope="module")
def four_weights(tq):
    """Weights of different types and sizes that share x, in an order in which the number of CTAs falls and rises."""
    k = 1024
    shapes = [(oracle.Q4_K, 4096), (oracle.Q6_K, 272), (oracle.Q5_K, 16), (oracle.Q4_K, 1000)]
    ws = [make_weight(t, n, k, SEED + 7200 + n) for t, n in shapes]
    return k, shapes, ws, [tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(t), (n, k))) for w, (t, n) in zip(ws, shapes)]


def rows_of_all_magnitudes(m, k, seed):
    """Every row by its own power of two, so that the row scales of one x are not those of another."""
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((m, k)) * 2.0 ** rng.integers(-8, 9, (m, 1))).astype(np.float32)


ONE_CALL = [(33, "batch"), (300, "tiles"), (1100, "pairs")]  # 1100 rows: pair tiles of 192, the last one of 140


@pytest.mark.parametrize("m,kernel", ONE_CALL)
def test_weights_of_one_call_run_side_by_side(tq, four_weights, m, kernel):
    """The later weights of a call start beside the first one, whatever follows the call waits for all
    of them, and none of them reads the operand, the row scales or the partial sums of another call:
    calls on different x are issued back to back, with no other kernel between them."""
    k, shapes, ws, mms = four_weights
    assert plan_shim.kernel([n for _, n in shapes], m) == kernel
    xs = [rows_of_all_magnitudes(m, k, SEED + 7201 + i) for i in range(4)]
    some = np.unique(np.r_[0:m:max(1, m // 100), m - 17:m])  # rows compared with the oracle
    xd = [torch.from_numpy(x).cuda() for x in xs]
    want = [[mm.forward(x, mode=tq.Mode.TENSOR_CORE) for mm in mms] for x in xd]
    for x, ys in zip(xs, want):
        for y, w, (t, n) in zip(ys, ws, shapes):
            ref = oracle.matmul_f64(t, w, n, k, x[some])
            scale = np.linalg.norm(ref, axis=1, keepdims=True)         # row by row: the magnitudes differ
            assert oracle.rel_fro(y.cpu().numpy()[some] / scale, ref / scale) < TOL
    for order in (slice(None), slice(None, None, -1)):
        outs = [[torch.full((m, n), float("nan"), device="cuda") for _, n in shapes[order]] for _ in range(20)]
        for i, o in enumerate(outs):
            tq.QMatMul.forward_multi(mms[order], xd[i % 4], outs=o, mode=tq.Mode.TENSOR_CORE)
        got = [torch.cat([y.flatten() for y in o]) for o in outs]      # launches of another kind behind the last call
        for i, g in enumerate(got):
            assert torch.equal(g, torch.cat([y.flatten() for y in want[i % 4][order]])), i
    tq.context().poll_status()


@pytest.mark.parametrize("m,kernel", ONE_CALL)
def test_captured_call_of_several_weights_on_changing_rows(tq, four_weights, m, kernel):
    k, shapes, _, mms = four_weights
    assert plan_shim.kernel([n for _, n in shapes], m) == kernel
    xs = [torch.from_numpy(rows_of_all_magnitudes(m, k, SEED + 7301 + i)).cuda() for i in range(3)]
    want = [[mm.forward(x, mode=tq.Mode.TENSOR_CORE) for mm in mms] for x in xs]
    x = xs[0].clone()
    tq.context().reserve(m, k, 4096)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            outs = [torch.empty((m, n), device="cuda") for _, n in shapes]
            tq.QMatMul.forward_multi(mms, x, outs=outs, mode=tq.Mode.TENSOR_CORE)
            tq.QMatMul.forward_multi(mms, x, outs=outs, mode=tq.Mode.TENSOR_CORE)
        for i in range(9):
            x.copy_(xs[i % 3])
            graph.replay()
            for o, w in zip(outs, want[i % 3]):
                assert torch.equal(o, w), i
    torch.cuda.current_stream().wait_stream(stream)
    tq.context().poll_status()


def test_contexts_on_streams_of_their_own(tq, four_weights):
    """Decode batches, whose clusters exchange partial sums, short prompts and prefill, in calls of several weights, from
    two threads with a context and a stream each: neither waits for or disturbs the other."""
    import threading
    k, shapes, ws, mms = four_weights
    xs = {m: torch.from_numpy(rows_of_all_magnitudes(m, k, SEED + 7400 + m)).cuda() for m in (17, 64, 300, 1100)}
    assert [plan_shim.kernel([n for _, n in shapes], m) for m in xs] == ["batch", "batch", "tiles", "pairs"]
    want = {m: [mm.forward(x, mode=tq.Mode.TENSOR_CORE) for mm in mms] for m, x in xs.items()}
    torch.cuda.synchronize()
    errors = []

    def worker():
        try:
            ctx = tq.new_context()
            mine = [tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(t), (n, k), ctx=ctx)) for w, (t, n) in zip(ws, shapes)]
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for it in range(30):
                    got = {m: tq.QMatMul.forward_multi(mine, x, mode=tq.Mode.TENSOR_CORE) for m, x in xs.items()}
                    stream.synchronize()
                    if not all(torch.equal(g, w) for m in xs for g, w in zip(got[m], want[m])):
                        errors.append(it)
                ctx.poll_status()
        except Exception as e:  # reported to the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=worker) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("k", [320, 384, 576, 1728, 2624])
@pytest.mark.parametrize("m,height", [(2048, 192), (2771, 256), (2999, 224)])
def test_prefill_pairs_with_several_tiles_and_a_short_last_unit(tq, k, m, height):
    """Q8_0 in-features that are no multiple of 256 with tall tiles, several for every pair: at 256 rows the set-up with
    three weight stages, two raw slots and three activation stages, a unit of one or two stages followed
    by the next tile, and the accumulators' hand-over there. Every activation row, weight rows all over the tiles."""
    n = 5000
    assert plan_shim.kernel([n], m) == "pairs" and plan_shim.pair_rows([n], m) == height
    w = make_weight(oracle.Q8_0, n, k, SEED + 7500 + k)
    x = rows_of_all_magnitudes(m, k, SEED + 7501 + m)
    rows = np.unique(np.r_[0:n:41, 255:n:256, 256:n:256, n - 1])
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(oracle.Q8_0), (n, k)))
    xd = torch.from_numpy(x).cuda()
    y = mm.forward(xd, mode=tq.Mode.TENSOR_CORE)
    assert torch.equal(mm.forward(xd, mode=tq.Mode.TENSOR_CORE), y)
    got = y[:, torch.from_numpy(rows).cuda()].cpu().numpy().astype(np.float64)
    ref = oracle.matmul_f64(oracle.Q8_0, np.ascontiguousarray(w.reshape(n, -1)[rows]).reshape(-1), len(rows), k, x)
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)      # row by row: the magnitudes differ
    # 123 or more outputs a row: a row's error stays within a few of the whole matrix' standard deviations
    assert err.max() < TOL, (int(err.argmax()), err.max())
    tq.context().poll_status()
