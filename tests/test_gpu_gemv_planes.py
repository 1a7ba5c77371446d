"""The integer-scheme GEMV's activation planes at the row counts, types and plane routes whose order differs: every number of rows of
one and two row groups, quants read from shared memory, from wide CTAs and from global memory, quantized in the kernel,
by a launch of their own and by the RMSNorm prologue (which writes both orders), and mixed launches, whose Q6_K tiles read
the order of the Q4_K / Q5_K ones."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SEED = 299792458
# integer sums are exact; the f32 sums over the blocks are ordered freely: k / 32 additions of 2^-24 each at most
TOL = 1e-5
TYPES = [oracle.Q8_0, oracle.Q4_K, oracle.Q5_K, oracle.Q6_K]


@pytest.fixture(scope="module")
def tq():
    import tur_b200
    return tur_b200


def weight(tq, dt, n, k, seed):
    w = oracle.quantize(dt, (np.random.default_rng(seed).standard_normal((n, k)) * 0.02).astype(np.float32))
    return w, tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))


@pytest.mark.parametrize("dt", TYPES)
@pytest.mark.parametrize("n,k", [(40, 512), (48, 4096), (4096, 12288)])  # in-kernel and staged, staged and wide, wide and global
def test_rows_of_every_count_against_the_oracle_and_alone(tq, dt, n, k):
    w, mm = weight(tq, dt, n, k, SEED + 8200 + n + k)
    x = np.random.default_rng(SEED + 8201 + k).standard_normal((37, k)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    rows = np.r_[0:min(n, 24), max(0, n - 24):n]
    sample = np.ascontiguousarray(w.reshape(n, -1)[rows]).reshape(-1)
    want = oracle.qmatmul(dt, sample, len(rows), k, x[:17])
    alone = torch.cat([mm.forward(xd[r:r + 1], mode=tq.Mode.INT8_ACT) for r in range(17)])
    assert oracle.rel_fro(alone.cpu().numpy()[:, rows], want) < TOL
    for m in (2, 3, 5, 7, 8, 9, 10, 13, 15, 16, 17):
        assert torch.equal(mm.forward(xd[:m], mode=tq.Mode.INT8_ACT), alone[:m]), m
    for m in (18, 23, 24, 25, 31):  # four groups of rows, the last ones empty, in part or but for a row
        assert torch.equal(mm.forward(xd[:m], mode=tq.Mode.INT8_ACT)[:17], alone), m
    y = mm.forward(xd, mode=tq.Mode.INT8_ACT)  # two passes: 32 rows and five
    assert torch.equal(y[:17], alone) and torch.equal(y[32:33], mm.forward(xd[32:33], mode=tq.Mode.INT8_ACT))
    assert torch.equal(mm.forward(xd[:9].to(torch.bfloat16), mode=tq.Mode.INT8_ACT),
                       mm.forward(xd[:9].to(torch.bfloat16).float(), mode=tq.Mode.INT8_ACT))
    tq.context().poll_status()


@pytest.mark.parametrize("other", [oracle.Q4_K, oracle.Q5_K])
@pytest.mark.parametrize("k", [512, 4096])
def test_mixed_launches_and_the_prologue_read_the_same_planes(tq, other, k):
    shapes = [(other, 272), (other, 48), (oracle.Q6_K, 80)]
    mms = [weight(tq, t, n, k, SEED + 8300 + n + t)[1] for t, n in shapes]
    x = torch.from_numpy(np.random.default_rng(SEED + 8301).standard_normal((20, k)).astype(np.float32)).cuda()
    norm = torch.from_numpy((1 + 0.1 * np.random.default_rng(SEED + 8302).standard_normal(k)).astype(np.float32)).cuda()
    for m in (1, 2, 3, 7, 8, 9, 12, 16, 20):
        got = tq.QMatMul.forward_multi(mms, x[:m], mode=tq.Mode.INT8_ACT)
        assert all(torch.equal(g, mm.forward(x[:m], mode=tq.Mode.INT8_ACT)) for g, mm in zip(got, mms)), m
        y = tq.QMatMul.rmsnorm_forward_multi(mms, x[:m], norm, 1e-6, mode=tq.Mode.INT8_ACT)
        h = tq.QMatMul.rmsnorm_forward_multi(mms[2:], x[:m], norm, 1e-6, mode=tq.Mode.INT8_ACT)[0]  # Q6_K alone: the other order
        assert torch.equal(y[2], h), m
    tq.context().poll_status()


@pytest.mark.parametrize("k", [32, 96, 224, 1056, 4192, 8256])
def test_q8_0_groups_of_one_to_four_tiles(tq, k):
    """Whole groups of four tiles take a path of their own, a last group of one to three the other: in-kernel, staged and global
    planes, one, two and four groups of rows. The bits of a row alone, which are the oracle's up to the order of the sums."""
    n = 48
    w, mm = weight(tq, oracle.Q8_0, n, k, SEED + 8400 + k)
    x = np.random.default_rng(SEED + 8401 + k).standard_normal((32, k)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    alone = torch.cat([mm.forward(xd[r:r + 1], mode=tq.Mode.INT8_ACT) for r in range(32)])
    assert oracle.rel_fro(alone.cpu().numpy(), oracle.qmatmul(oracle.Q8_0, w, n, k, x)) < TOL
    for m in (3, 8, 9, 16, 17, 25, 32):
        assert torch.equal(mm.forward(xd[:m], mode=tq.Mode.INT8_ACT), alone[:m]), m
    tq.context().poll_status()
