"""Integer-scheme launches whose activation planes are shared by two sets of warps of one CTA per SM:
the row counts and in-feature counts at which a CTA's half of the shared memory is too small for them
and, on either side, those at which they stay in global memory; an odd number of shares, row-tiles
cut between shares, one hand-over buffer (8 rows of 12288 values), mixed types. A row's bits are those
it has alone, and a weight is streamed once."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SEED = 299792458


@pytest.fixture(scope="module")
def tq():
    import tur_b200
    return tur_b200


def make_weight(dt, n, k, seed):
    rng = np.random.default_rng(seed)
    return oracle.quantize(dt, (rng.standard_normal((n, k)) * 0.02).astype(np.float32))


@pytest.mark.parametrize("dt", [oracle.Q8_0, oracle.Q4_K, oracle.Q5_K, oracle.Q6_K])
@pytest.mark.parametrize("n,k", [(37, 12288), (1, 4096), (5000, 4096), (300, 8192), (16, 16384)])
def test_rows_keep_their_bits(tq, dt, n, k):
    w = make_weight(dt, n, k, SEED + 8000 + n)
    x = np.random.default_rng(SEED + 8001 + k).standard_normal((16, k)).astype(np.float32)
    mm = tq.QMatMul.from_arc(tq.QTensor.new(w, tq.GgmlDType(dt), (n, k)))
    xd = torch.from_numpy(x).cuda()
    rows = torch.cat([mm.forward(xd[r:r + 1], mode=tq.Mode.INT8_ACT) for r in range(16)])
    for m in (3, 8, 9, 13, 16):
        assert torch.equal(mm.forward(xd[:m], mode=tq.Mode.INT8_ACT), rows[:m])
    few = rows[:2].cpu().numpy()
    # the integers are exact; f32 sums over k / 32 blocks in another order: sqrt(512) * 2^-24 at most
    assert oracle.rel_fro(few, oracle.qmatmul(dt, w, n, k, x[:2])) < 2e-6
    tq.context().poll_status()


@pytest.mark.parametrize("dt", [oracle.Q8_0, oracle.Q4_K, oracle.Q5_K, oracle.Q6_K])
@pytest.mark.parametrize("n,k,rows", [(9600, 4096, (13, 16)), (4096, 12288, (4, 8, 9, 16)), (5120, 8192, (8, 12, 16))])
def test_rows_keep_their_bits_in_large_weights(tq, dt, n, k, rows):
    """9600 rows: every type runs wide with row-tiles cut between shares; 5120: cut, where only Q8_0 and Q6_K run wide."""
    from tur_b200.workloads import random_blocks
    mm = tq.QMatMul.from_arc(tq.QTensor.new(random_blocks(dt, n, k, SEED + 8200 + n, torch.device("cuda", 0)), tq.GgmlDType(dt), (n, k)))
    xd = torch.from_numpy(np.random.default_rng(SEED + 8201 + k).standard_normal((16, k)).astype(np.float32)).cuda()
    alone = torch.cat([mm.forward(xd[r:r + 1], mode=tq.Mode.INT8_ACT) for r in range(16)])
    for m in rows:
        l0 = tq.context().launch_count()
        y = mm.forward(xd[:m], mode=tq.Mode.INT8_ACT)
        assert tq.context().launch_count() - l0 == 2, "one quantization of x, one pass over the weight"
        assert torch.equal(y, alone[:m])
    tq.context().poll_status()


def test_mixed_types_beyond_eight_rows(tq):
    k, shapes = 4096, [(oracle.Q4_K, 1000), (oracle.Q4_K, 272), (oracle.Q6_K, 272)]
    mms = [tq.QMatMul.from_arc(tq.QTensor.new(make_weight(t, n, k, SEED + 8100 + n + t), tq.GgmlDType(t), (n, k))) for t, n in shapes]
    xd = torch.from_numpy(np.random.default_rng(SEED + 8101).standard_normal((16, k)).astype(np.float32)).cuda()
    for m in (9, 16):
        got = tq.QMatMul.forward_multi(mms, xd[:m], mode=tq.Mode.INT8_ACT)
        for g, mm in zip(got, mms):
            assert torch.equal(g, mm.forward(xd[:m], mode=tq.Mode.INT8_ACT))
    tq.context().poll_status()
