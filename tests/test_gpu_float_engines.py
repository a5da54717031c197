"""The float form with engine 1: fp32 on the CUDA cores for any number of vectors, as exact as one vector is, where engine 0
takes tensor-core sums and s . dy as two bf16 terms."""
import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]

if cuda_ok():
    import torch
    from matvans_b200 import ops


def gauss(rng, shape):
    return np.clip(np.round(rng.normal(0, 4.0, size=shape)), -127, 127).astype(np.int8)


def bf16(rng, shape):
    return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda().to(torch.bfloat16)


def scales(rng, rows):
    return torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()


@pytest.mark.parametrize("rows,cols,seg_quads,local", [
    (33, 16, 0, True), (64, 1040, 4, False), (64, 2048, 68, True), (50, 1520, 36, True), (64, 4096, 128, False)])
@pytest.mark.parametrize("B", [2, 3, 5, 8, 9, 17])
def test_engine_1_gives_each_vector_what_it_is_alone(rows, cols, seg_quads, local, B):
    # up to two stripes: a column's two parts add up the same in either order, so both directions are equal bit for bit
    rng = np.random.default_rng(rows + cols + B)
    M = ops.Q8Matrix.encode(gauss(rng, (rows, cols)), local=local, seg_quads=seg_quads)
    s, x, dy = scales(rng, rows), bf16(rng, (B, cols)), bf16(rng, (B, rows))
    t = (2, 1, 1, 0, 1, 1)
    y, dx = M.matvec_bf16(x, s, tuning=t), M.matvec_t_bf16(dy, s, tuning=t)
    for b in range(B):
        assert torch.equal(y[b], M.matvec_bf16(x[b], s, tuning=t)), b
        assert torch.equal(dx[b], M.matvec_t_bf16(dy[b], s, tuning=t)), b
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 2, 4, 8, 33])
@pytest.mark.parametrize("engine", [1])
def test_engine_1_backward_keeps_s_dy_in_fp32(B, engine):
    # one row of weights in a matrix of zeros: dX is w (s dy), two fp32 roundings of 2^-24 each (the other terms are zero);
    # s dy as two bf16 terms would be off by up to 2^-18
    rng = np.random.default_rng(B)
    W = np.zeros((96, 1024), np.int8)
    W[41] = rng.integers(1, 128, size=1024)
    M = ops.Q8Matrix.encode(W)
    s, dy = scales(rng, 96), bf16(rng, (B, 96))
    dx = M.matvec_t_bf16(dy, s, tuning=(0, 0, 0, 0, 0, engine))
    ref = (dy.double() * s.double()) @ torch.from_numpy(W).cuda().double()
    assert ((dx.double() - ref).abs() / ref.abs()).max().item() <= 2.0 ** -23 * (1 + 1e-6)
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols", [(1504, 1040), (4800, 512)])
def test_engine_1_bounds(rows, cols):
    # sums of n fp32 terms: a lane's chain of at most cols terms and the warps' sums forward; 32 rows by 9 additions, and one
    # atomic addition a stripe, backward; each rounding 2^-24 of the sum of the magnitudes
    rng = np.random.default_rng(rows)
    W = gauss(rng, (rows, cols))
    M = ops.Q8Matrix.encode(W)
    W64 = torch.from_numpy(W).cuda().double()
    s = scales(rng, rows)
    for B in (2, 7, 16, 64):
        x, dy = bf16(rng, (B, cols)), bf16(rng, (B, rows))
        t = (0, 0, 0, 0, 0, 1)
        y, dx = M.matvec_bf16(x, s, tuning=t), M.matvec_t_bf16(dy, s, tuning=t)
        mag = (x.double().abs() @ W64.abs().T) * s.double()
        assert ((y.double() - (x.double() @ W64.T) * s.double()).abs() / mag).max().item() < 2.0 ** -24 * (cols + 20)
        g = dy.double() * s.double()
        err = (dx.double() - g @ W64).abs() / (g.abs() @ W64.abs())
        assert err.max().item() < 2.0 ** -24 * (11 + rows / 32 + 1)
        assert torch.equal(y, M.matvec_bf16(x, s, tuning=t)), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("B", [1, 3, 8, 20])
def test_infinities_and_nan_stay_where_they_belong(engine, B):
    # one element of one vector: its outputs are infinite or NaN as in fp32 arithmetic, every other vector's are untouched
    rng = np.random.default_rng(B)
    rows, cols = 96, 1040
    W = gauss(rng, (rows, cols))
    W[:, 5] = rng.integers(1, 100, size=rows)  # (no zero weight meets the infinity)
    W[7] = rng.integers(1, 100, size=cols)
    M = ops.Q8Matrix.encode(W)
    s = scales(rng, rows)
    t = (4, 1, 1, 0, 0, engine)
    for val in (float("inf"), float("-inf"), float("nan")):
        x, dy = bf16(rng, (B, cols)), bf16(rng, (B, rows))
        y0, d0 = M.matvec_bf16(x, s, tuning=t), M.matvec_t_bf16(dy, s, tuning=t)
        b = B // 2
        x[b, 5], dy[b, 7] = val, val
        y, dx = M.matvec_bf16(x, s, tuning=t), M.matvec_t_bf16(dy, s, tuning=t)
        for got, ref0 in ((y, y0), (dx, d0)):
            want = torch.full_like(got[b], val)
            assert torch.equal(got[b].isnan(), want.isnan()) and (val != val or torch.equal(got[b], want)), (engine, B, val)
            others = [i for i in range(B) if i != b]
            assert torch.allclose(got[others], ref0[others], rtol=1e-5, atol=1e-6)
    assert ops.device_status() == 0
