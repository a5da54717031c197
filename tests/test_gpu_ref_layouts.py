"""The reference's three stream layouts at the sizes where the kernels' rings, rounds and groups change: one row or
stripe, more rows than a round of warps, the shortest rows, the densest streams (every refill word of the format's
worst case), streams that start off the 16-byte grid.  Bit-exact against the CPU oracle's matvec."""
import numpy as np
import pytest

from conftest import cuda_ok
import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]

if cuda_ok():
    import torch
    from matvans_b200 import codec, ops


def weights(rng, kind, shape):
    if kind == "dense":  # nearly uniform: the most words a symbol
        return rng.integers(-60, 61, size=shape).astype(np.int8)
    if kind == "tails":  # lanes whose streams run at very different rates
        W = np.zeros(shape, np.int8)
        W[:, ::3] = rng.integers(-60, 61, size=W[:, ::3].shape)
        return W
    return np.clip(np.round(rng.normal(0, 3.0, size=shape)), -60, 60).astype(np.int8)


def check(M, W, rng, batches):
    for B in batches:
        x = rng.integers(-128, 128, size=(B, W.shape[1])).astype(np.int8)
        s = rng.uniform(1e-3, 1e-2, size=W.shape[0]).astype(np.float32)
        y, ys = M.matvec(torch.from_numpy(x), scales=s)
        ref = oracle.matvec_i8(W, x)
        assert np.array_equal(y.cpu().numpy(), ref), B
        assert np.array_equal(ys.cpu().numpy(), (ref.astype(np.float32) * s[None, :]).astype(np.float32)), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("kind", ["gauss", "dense", "tails"])
@pytest.mark.parametrize("rows,cols", [(1, 512), (150, 1536), (4200, 512)])
def test_wpr(kind, rows, cols):
    rng = np.random.default_rng(rows + cols)
    W = weights(rng, kind, (rows, cols))
    check(ops.WprMatrix.encode(W), W, rng, (1, 3, 9, 17))


def test_wpr_stream_off_the_grid():
    rng = np.random.default_rng(3)
    W = weights(rng, "gauss", (70, 1024))
    cm = codec.encode_matrix(W)
    cm.payload = np.concatenate([np.full(3, 0xABCD, np.uint16), cm.payload])
    cm.cursors = cm.cursors + np.uint32(3)
    check(ops.WprMatrix(cm), W, rng, (1, 4))


@pytest.mark.parametrize("kind", ["gauss", "dense", "tails"])
@pytest.mark.parametrize("rows,cols", [(1, 128), (150, 640), (4200, 256), (33, 4096)])
def test_awr(kind, rows, cols):
    rng = np.random.default_rng(rows + cols)
    W = weights(rng, kind, (rows, cols))
    check(ops.AwrMatrix.encode(W), W, rng, (1, 3, 9, 17))


@pytest.mark.parametrize("kind", ["gauss", "dense", "tails"])
@pytest.mark.parametrize("rows,cols", [(32, 4), (64, 36), (96, 1000), (4800, 64)])
def test_aws(kind, rows, cols):
    rng = np.random.default_rng(rows + cols)
    W = weights(rng, kind, (rows, cols))
    M = ops.AwsMatrix.encode(W)
    check(M, W, rng, (1, 3, 9, 17))
    # the launcher that does not know the stream's length reads no further than the words it takes
    x = rng.integers(-128, 128, size=cols).astype(np.int8)
    out = torch.empty(rows, dtype=torch.int8, device="cuda")
    assert ops.mat_vec_mul_coalesced_stripes(torch.from_numpy(x).cuda(), out, cols, rows, 2e-3, M.compressed, M.offsets,
                                             M.ppf, M.ppf_cum, M.ppf_prob) is not None
    torch.cuda.synchronize()
    ref = np.clip(np.rint(oracle.matvec_i8(W, x[None, :])[0].astype(np.float32) * np.float32(2e-3)), -128, 127)
    assert np.array_equal(out.cpu().numpy(), ref.astype(np.int8))


@pytest.mark.parametrize("n", [1, 31, 1025, 4096, 4097, 8193, 70000, 8 * 1024 * 16, 8 * 1024 * 16 + 1])
def test_requant_absmax(n):
    # one CTA, clusters of 2, 4 and 8, the last element a thread holds, and the three-launch form behind them; fp32
    # arithmetic of the reference, rounded half to even: equal, not close
    rng = np.random.default_rng(n)
    for y in (rng.integers(-5000000, 5000001, size=n).astype(np.int32), np.where(np.arange(n) == n - 1, -127, 3).astype(np.int32)):
        out8, delta = ops.requant_absmax(torch.from_numpy(y).cuda())
        d = np.float32(np.abs(y.astype(np.int64)).max()) / np.float32(127.0)
        assert delta.item() == d
        assert np.array_equal(out8.cpu().numpy(), np.rint(y.astype(np.float32) / d).astype(np.int8))
    assert ops.device_status() == 0


@pytest.mark.parametrize("n", [4097, 9000, 8 * 1024 * 16])
def test_requant_absmax_every_cta_counts(n):
    # clusters of 2, 4 and 8 whose CTAs write their maxima to each other: the maximum moves over all of them, many launches
    # behind one another
    rng = np.random.default_rng(n)
    base = rng.integers(-1000, 1001, size=n).astype(np.int32)
    got, want = [], []
    for i in range(64):
        y = base.copy()
        y[(i * 1024 + 7 * i) % n] = 5000 + i
        got.append(ops.requant_absmax(torch.from_numpy(y).cuda()))
        d = np.float32(5000 + i) / np.float32(127.0)
        want.append((np.rint(y.astype(np.float32) / d).astype(np.int8), d))
    for (out8, delta), (ref, d) in zip(got, want):
        assert delta.item() == d and np.array_equal(out8.cpu().numpy(), ref)


@pytest.mark.parametrize("batch", [1, 16])
def test_aws_blocks_come_round(batch):
    # dense streams of many more blocks than the ring holds, so that each is overwritten while the decode runs on; the
    # same sums every time
    rng = np.random.default_rng(batch)
    W = weights(rng, "dense", (160, 4096))
    M = ops.AwsMatrix.encode(W)
    x = torch.from_numpy(rng.integers(-128, 128, size=(batch, 4096)).astype(np.int8)).cuda()
    ref = oracle.matvec_i8(W, x.cpu().numpy())
    ys = [M.matvec(x) for _ in range(50)]
    for y in ys:
        assert np.array_equal(y.cpu().numpy(), ref)
    assert ops.device_status() == 0
