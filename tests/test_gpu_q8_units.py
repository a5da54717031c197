"""Warp-specialised Q8 kernel: unit, slot and table hand-over at the sizes where they change, bit-exact against the
CPU oracle.  (Tiny segments pass a stream slot from warp to warp within one decode; segments beyond 64 quads read x
from global memory; fewer units than warps and single-segment stripes leave warps idle; batches cross the 16-vector
lane groups and the 64-vector pass.)"""
import numpy as np
import pytest

from conftest import cuda_ok
import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]

if cuda_ok():
    import torch
    from matvans_b200 import ops


@pytest.mark.parametrize("rows,cols,seg_quads,local", [
    (33, 16, 0, True), (5000, 64, 4, True), (257, 1040, 4, False), (96, 2048, 68, True), (64, 8192, 128, False),
    (9600, 272, 0, True)])
def test_units_and_batches(rows, cols, seg_quads, local):
    rng = np.random.default_rng(rows + cols + seg_quads)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, local=local, seg_quads=seg_quads)
    s = rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)
    for B in (1, 2, 3, 17, 33, 64, 66):
        x = rng.integers(-128, 128, size=(B, cols)).astype(np.int8)
        y, ys = M.matvec(torch.from_numpy(x), scales=s)
        ref = oracle.matvec_i8(W, x)
        assert np.array_equal(y.cpu().numpy(), ref), B
        assert np.array_equal(ys.cpu().numpy(), (ref.astype(np.float32) * s[None, :]).astype(np.float32)), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 2, 5, 16])
def test_stack_of_uneven_items_runs_repeatedly(B):
    # more items than CTAs, items of 1 to 40 units, tables shared and not: the work queue, the table hand-over and
    # the accumulators over several launches of one plan
    rng = np.random.default_rng(B)
    shapes = [(4096, 64, 4), (640, 2560, 64), (3000, 160, 8), (64, 16, 0), (1504, 1024, 0)]
    Ws = [np.clip(np.round(rng.normal(0, 3.0, size=sh[:2])), -127, 127).astype(np.int8) for sh in shapes]
    Ms = [ops.Q8Matrix.encode(W, local=i % 2 == 0, seg_quads=sh[2]) for i, (W, sh) in enumerate(zip(Ws, shapes))]
    S = ops.Q8Stack(Ms, batch=B)
    for _ in range(3):
        for M, xd in zip(Ms, S.xs):
            xd.copy_(torch.from_numpy(rng.integers(-127, 128, size=(B, M.cols)).astype(np.int8)))
        S.y_flat.fill_(-1)
        S.run()
        for W, xd, y in zip(Ws, S.xs, S.ys):
            assert np.array_equal(y.cpu().numpy(), oracle.matvec_i8(W, xd.cpu().numpy())), W.shape
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads,local", [
    (33, 16, 0, True), (257, 1040, 4, False), (96, 2048, 68, True), (1500, 272, 12, True), (64, 8192, 128, False)])
def test_float_forward_units(rows, cols, seg_quads, local):
    # one vector (CUDA cores), the 16-vector lane groups and the 64-vector pass: fp32 sums against 64 bits, relative to
    # the sum of the magnitudes of a row's terms (a sum of n fp32 terms in any order is within n ulps of it; here a
    # warp's chain is at most cols / 16 accumulations and the warps' sums are added once), and bit for bit the same twice
    rng = np.random.default_rng(rows + cols + seg_quads)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, local=local, seg_quads=seg_quads)
    s = torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()
    W64 = torch.from_numpy(W).cuda().double()
    for B in (1, 2, 16, 17, 49, 64, 65):
        x = torch.from_numpy(rng.standard_normal((B, cols)).astype(np.float32)).cuda().to(torch.bfloat16)
        y = M.matvec_bf16(x, s)
        ref = (x.double() @ W64.T) * s.double()
        mag = (x.double().abs() @ W64.abs().T) * s.double()
        assert ((y.double() - ref).abs() / mag.clamp_min(1e-30)).max().item() < 2.0 ** -24 * (cols / 16 + 20), B
        assert torch.equal(y, M.matvec_bf16(x, s)), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads,local", [
    (33, 16, 0, True), (257, 1040, 4, False), (96, 2048, 68, True), (1500, 272, 12, True), (64, 8192, 128, False)])
def test_float_backward_units(rows, cols, seg_quads, local):
    # one vector (CUDA cores), the sums by vector (to 4) and by row (from 5), the 32-vector pass.  s . dy enters as two
    # bf16 terms (2^-17 of it, or exactly, at one vector); at most rows + 32 fp32 additions of 2^-23 each, tensor cores
    # truncating: relative to the sum of the magnitudes of a column's terms
    rng = np.random.default_rng(rows + cols + seg_quads)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, local=local, seg_quads=seg_quads)
    s = torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()
    W64 = torch.from_numpy(W).cuda().double()
    for B in (1, 2, 4, 5, 31, 32, 33):
        dy = torch.from_numpy(rng.standard_normal((B, rows)).astype(np.float32)).cuda().to(torch.bfloat16)
        dx = M.matvec_t_bf16(dy, s)
        ref = (dy.double() * s.double()) @ W64
        mag = (dy.double() * s.double()).abs() @ W64.abs()
        bound = (0.0 if B == 1 else 2.0 ** -17) + 2.0 ** -23 * (rows + 32)
        assert ((dx.double() - ref).abs() / mag.clamp_min(1e-30)).max().item() < bound, B
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads", [(2400, 11008, 0), (4736 + 40, 3104, 64), (7001, 5008, 0)])
def test_even_shares(rows, cols, seg_quads):
    # CTAs that share stripes at the borders of their units, whole ranges of stripes in between, the short last segment
    # and the ragged last stripe; exact sums, their scaled form, and the float form both ways (bounds as above; the
    # forward is the same bit for bit whatever the order its parts arrive in)
    rng = np.random.default_rng(rows)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, seg_quads=seg_quads)
    s = rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)
    sd, W64 = torch.from_numpy(s).cuda(), torch.from_numpy(W).cuda().double()
    for B in (1, 5, 16, 64):
        x = rng.integers(-128, 128, size=(B, cols)).astype(np.int8)
        y, ys = M.matvec(torch.from_numpy(x), scales=s)
        ref = torch.from_numpy(x).cuda().double() @ W64.T
        assert torch.equal(y.double(), ref), B
        assert torch.equal(ys, ref.float() * sd), B
        assert torch.equal(M.matvec(torch.from_numpy(x)), y), B
        xf = torch.from_numpy(rng.standard_normal((B, cols)).astype(np.float32)).cuda().to(torch.bfloat16)
        yf = M.matvec_bf16(xf, sd)
        mag = (xf.double().abs() @ W64.abs().T) * sd.double()
        err = (yf.double() - (xf.double() @ W64.T) * sd.double()).abs() / mag
        assert err.max().item() < 2.0 ** -24 * (cols / 16 + 20), B
        assert torch.equal(yf, M.matvec_bf16(xf, sd)), B
        dy = torch.from_numpy(rng.standard_normal((B, rows)).astype(np.float32)).cuda().to(torch.bfloat16)
        g = dy.double() * sd.double()
        err = (M.matvec_t_bf16(dy, sd).double() - g @ W64).abs() / (g.abs() @ W64.abs())
        assert err.max().item() < (0.0 if B == 1 else 2.0 ** -17) + 2.0 ** -23 * (rows + 32), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads,offset", [
    (33, 1, 0, 0), (100, 15, 0, 0), (257, 1037, 4, 0), (96, 2050, 68, 1), (5000, 275, 0, 0), (64, 8191, 130, 3),
    (2400, 6001, 0, 0), (64, 1040, 6, 0), (70, 1024, 64, 5)])
def test_ragged(rows, cols, seg_quads, offset):
    # rows of x that start anywhere, a last quad of 1 to 3 columns, segments of any number of quads, x off the grid;
    # dp4a, the small matrices' 8 vectors, the tensor cores' 16, their 64 and the pass after them
    rng = np.random.default_rng(rows + cols + seg_quads)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, local=rows != 100, seg_quads=seg_quads)
    s = rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)
    for B in (1, 2, 3, 5, 8, 9, 16, 19, 64, 70):
        xf = torch.randint(-128, 128, (offset + B * cols,), dtype=torch.int8, device="cuda")
        x = xf[offset:].view(B, cols)
        y, ys = M.matvec(x, scales=s)
        ref = oracle.matvec_i8(W, x.cpu().numpy())
        assert np.array_equal(y.cpu().numpy(), ref), B
        assert np.array_equal(ys.cpu().numpy(), (ref.astype(np.float32) * s[None, :]).astype(np.float32)), B
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads", [(96, 2048, 68), (64, 8192, 128), (500, 1040, 260)])
def test_x_from_global_memory_odd_batches(rows, cols, seg_quads):
    # segments of more than 64 quads read x from global memory; batches below the 4, 8 or 16 vectors that the consumer
    # holds (3 vectors, 5 to 7 of a small matrix, and with engine 1 up to 15) take no row past the batch's last.  x is the
    # head of a larger buffer; the rows behind it change and the outputs do not
    rng = np.random.default_rng(seg_quads)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, seg_quads=seg_quads)
    for B, engine in [(3, 0), (5, 0), (6, 0), (7, 0), (3, 1), (6, 1), (9, 1), (13, 1), (15, 1)]:
        buf = torch.randint(-128, 128, (16, cols), dtype=torch.int8, device="cuda")
        x = buf[:B]
        ref = oracle.matvec_i8(W, x.cpu().numpy())
        tuning = (4, 1, 1, 0, 0, engine)  # (a launch shape that these blocks fit)
        S = ops.Q8Stack([M], batch=B, xs=[x], tuning=tuning)
        for fill in (None, 127):
            if fill is not None:
                buf[B:] = fill
            for y in (M.matvec(x, tuning=tuning), S.run()[0]):
                assert np.array_equal(y.cpu().numpy(), ref), (B, engine)
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows", [2 ** 25 - 1, 2 ** 25 + 3])
def test_block_of_four_gigabytes_is_rejected(rows):
    # offsets that claim a block of 2^32 bytes and more, all of it readable: no 32-bit size may wrap round to a small one
    W = np.ones((32, 64), np.int8)
    M = ops.Q8Matrix.encode(W)
    M.blocks = torch.zeros(32 * (rows + 8), dtype=torch.int32, device="cuda")
    M.blk_off = torch.tensor([0, rows], dtype=torch.int32, device="cuda")
    M._view = M.view()
    x = torch.ones((1, 64), dtype=torch.int8, device="cuda")
    M.matvec(x)
    assert ops.device_status(raise_on_error=False) == 1  # MV_DEV_STREAM_OVERRUN: nothing was decoded
    G = ops.Q8Matrix.encode(W)
    assert np.array_equal(G.matvec(x).cpu().numpy(), oracle.matvec_i8(W, x.cpu().numpy()))
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,seg_quads", [(32, 4096, 64), (100, 1520, 36), (257, 8192, 0)])
def test_float_backward_reads_dy_alone(rows, cols, seg_quads):
    # many more columns than rows, dY off the 16-byte grid, a dX off it too, each in the middle of a larger buffer that is
    # all NaN or a sign value around it: dY is read within its rows, dX written within its columns (bounds as above; a dX off
    # the grid, and one vector, have no split of s . dy)
    rng = np.random.default_rng(rows + cols)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -127, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, seg_quads=seg_quads)
    s = torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()
    W64 = torch.from_numpy(W).cuda().double()
    for B in (1, 2, 5, 33):
        for dy_off, dx_off in [(0, 0), (1, 0), (5, 1), (8, 3)]:
            dyb = torch.full((B * rows + 4096,), float("nan"), dtype=torch.bfloat16, device="cuda")
            dy = dyb[dy_off:dy_off + B * rows].view(B, rows)
            dy.copy_(torch.from_numpy(rng.standard_normal((B, rows)).astype(np.float32)))
            dxb = torch.full((B * cols + 64,), -7.0, device="cuda")
            dx = dxb[dx_off:dx_off + B * cols].view(B, cols)
            M.matvec_t_bf16(dy, s, out=dx)
            g = dy.double() * s.double()
            err = (dx.double() - g @ W64).abs() / (g.abs() @ W64.abs()).clamp_min(1e-30)
            bound = (0.0 if B == 1 or dx_off % 4 else 2.0 ** -17) + 2.0 ** -23 * (rows + 32)
            assert err.max().item() < bound, (B, dy_off, dx_off)
            assert (dxb[:dx_off] == -7).all() and (dxb[dx_off + B * cols:] == -7).all(), (B, dy_off, dx_off)
    assert ops.device_status() == 0


def test_scaled_outputs_of_more_than_two_billion_elements():
    # 64 vectors of 2^25 + 32 rows in two parts a stripe: sums joined by atomics, then scaled, element numbers past 31 bits.
    # The matrix is one stripe's block over and over
    stripes, B = 2 ** 20 + 1, 64
    E = ops.Q8Matrix.encode(np.ones((32, 32), np.int8), local=False, seg_quads=4)
    off = E.blk_off.view(torch.int32)
    per = int(off[2])
    assert E.nseg == 2
    E.blocks = E.blocks.view(torch.int32)[:32 * per].repeat(stripes)
    E.blk_off = torch.cat([(torch.arange(stripes, dtype=torch.int32, device="cuda")[:, None] * per + off[None, :2]).reshape(-1),
                           torch.tensor([stripes * per], dtype=torch.int32, device="cuda")])
    E.rows = 32 * stripes
    E._view = E.view()
    x = torch.randint(-128, 128, (B, 32), dtype=torch.int8, device="cuda")
    s = torch.rand(E.rows, device="cuda")
    y, ys = E.matvec(x, scales=s, tuning=(8, 1, 1, 0, 2, 0))
    sums = x.sum(1, dtype=torch.int32)
    for b in range(B):
        assert bool((y[b] == sums[b]).all()) and torch.equal(ys[b], sums[b].float() * s), b
    assert ops.device_status() == 0


def wide(rng, rows, cols, seg_quads, local=True):
    W = rng.integers(-128, 128, size=(rows, cols)).astype(np.int8)  # 8 bits a weight, tables of 256 symbols
    return W, ops.Q8Matrix.encode(W, local=local, seg_quads=seg_quads)


@pytest.mark.parametrize("rows,seg_quads,local", [(40, 880, True), (96, 1132, True), (4768, 1132, True), (96, 1236, False)])
def test_blocks_that_fill_shared_memory(rows, seg_quads, local):
    # the largest blocks that a launch shape of one warp, one segment and one buffer lets through: more than the kernel's
    # tables and staging leave room for.  Single matrices in whole stripes, parts and even shares, stacks, with and without
    # scales, both engines
    rng = np.random.default_rng(rows + seg_quads)
    cols = 4 * (2 * seg_quads + 36)
    W, M = wide(rng, rows, cols, seg_quads, local)
    assert M.max_blk_rows >= seg_quads
    s = rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)
    for B in (1, 3, 16, 35) if rows < 1000 else (2,):
        x = rng.integers(-128, 128, size=(B, cols)).astype(np.int8)
        xd = torch.from_numpy(x).cuda()
        ref = oracle.matvec_i8(W, x)
        for parts, engine in ((0, 0), (2, 0), (0, 1)):
            y, ys = M.matvec(xd, scales=s, tuning=(1, 1, 1, 0, parts, engine))
            assert np.array_equal(y.cpu().numpy(), ref), (B, parts, engine)
            assert np.array_equal(ys.cpu().numpy(), (ref.astype(np.float32) * s[None, :]).astype(np.float32)), (B, parts, engine)
            if B <= 16:
                S = ops.Q8Stack([M, M], batch=B, xs=[xd, xd], tuning=(1, 1, 1, 0, parts, engine))
                for _ in range(2):
                    S.y_flat.fill_(-1)
                    assert all(np.array_equal(y.cpu().numpy(), ref) for y in S.run()), (B, parts, engine)
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 3, 16])
def test_chain_of_blocks_that_fill_shared_memory(B):
    rng = np.random.default_rng(B)
    W0, M0 = wide(rng, 4720, 128, 32)
    W1, M1 = wide(rng, 64, 4720, 1132)
    x = torch.from_numpy(rng.integers(-128, 128, size=(B, 128)).astype(np.int8)).cuda()
    C = ops.Q8Chain([M0, M1], [2e-4, 2e-5], batch=B, tuning=(1, 1, 1, 0), x0=x)
    for _ in range(2):
        C.run()
        xh = x.cpu().numpy()
        for W, scale, out, y in ((W0, 2e-4, C.xs[1], C.ys[0]), (W1, 2e-5, C.out8, C.ys[1])):
            yh = oracle.matvec_i8(W, xh)
            xh = np.clip(np.rint(yh.astype(np.float32) * np.float32(scale)), -128, 127).astype(np.int8)
            assert np.array_equal(y.cpu().numpy(), yh) and np.array_equal(out.cpu().numpy(), xh)
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,seg_quads", [(40, 1148), (96, 1400), (4768, 1160)])
def test_float_blocks_that_fill_shared_memory(rows, seg_quads):
    # bounds as above (these sums are fp32 throughout: a lane's chain of all columns forward, no split of s . dy backward)
    rng = np.random.default_rng(rows + seg_quads)
    cols = 4 * (2 * seg_quads + 36)
    W, M = wide(rng, rows, cols, seg_quads)
    s = torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()
    W64 = torch.from_numpy(W).cuda().double()
    for B in (1, 2, 9, 40) if rows < 1000 else (3,):
        for engine in (0, 1):
            t = (1, 1, 1, 0, 0, engine)
            x = torch.from_numpy(rng.standard_normal((B, cols)).astype(np.float32)).cuda().to(torch.bfloat16)
            dy = torch.from_numpy(rng.standard_normal((B, rows)).astype(np.float32)).cuda().to(torch.bfloat16)
            if seg_quads <= 1160:
                y = M.matvec_bf16(x, s, tuning=t)
                mag = (x.double().abs() @ W64.abs().T) * s.double()
                assert ((y.double() - (x.double() @ W64.T) * s.double()).abs() / mag).max().item() < 2.0 ** -24 * (cols + 20)
                assert torch.equal(y, M.matvec_bf16(x, s, tuning=t)), B
            dx = M.matvec_t_bf16(dy, s, tuning=t)
            g = dy.double() * s.double()
            assert ((dx.double() - g @ W64).abs() / (g.abs() @ W64.abs())).max().item() < 2.0 ** -24 * (12 + rows / 32 + 1)
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,cols,local", [(9600, 301, True), (16000, 401, True), (16001, 129, False), (33200, 65, True),
                                             (35000, 17, False), (34000, 303, True), (14000, 1021, True)])
def test_ragged_short_rows(rows, cols, local):
    # around the line between the two kernels for ragged products (grids that are resident at once, and of several rounds),
    # plain and scaled, on rows of x that start anywhere
    rng = np.random.default_rng(rows + cols)
    W = np.clip(np.round(rng.normal(0, 4.0, size=(rows, cols))), -128, 127).astype(np.int8)
    M = ops.Q8Matrix.encode(W, local=local)
    W64 = torch.from_numpy(W).cuda().double()
    s = torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda()
    for B in (1, 2, 4, 7, 8, 16, 17):
        x = torch.randint(-128, 128, (3 + B * cols,), dtype=torch.int8, device="cuda")[3:].view(B, cols)
        ref = x.double() @ W64.T
        y, ys = M.matvec(x, scales=s)
        assert torch.equal(y.double(), ref), B
        assert torch.equal(ys, ref.float() * s), B
        assert torch.equal(M.matvec(x), y), B
    assert ops.device_status() == 0


def test_many_items_share_one_table():
    # one table for all rows and items of a single short unit: records pass through their ring as fast as they can, most of
    # them with no table to stage, between them in a stack the few that have one
    rng = np.random.default_rng(5)
    shapes = [(60000, 16), (64, 512), (40000, 32), (30000, 16)]
    Ws = [np.clip(np.round(rng.normal(0, 3.0, size=sh)), -127, 127).astype(np.int8) for sh in shapes]
    Ms = [ops.Q8Matrix.encode(W, local=i == 1) for i, W in enumerate(Ws)]
    for B in (1, 3, 16):
        xs = [torch.from_numpy(rng.integers(-128, 128, size=(B, M.cols)).astype(np.int8)).cuda() for M in Ms]
        S = ops.Q8Stack(Ms, batch=B, xs=xs)
        for _ in range(10):
            S.y_flat.fill_(-1)
            S.run()
            for W, x, y in zip(Ws, xs, S.ys):
                assert np.array_equal(y.cpu().numpy(), oracle.matvec_i8(W, x.cpu().numpy())), (B, W.shape)
        for M, W, x in zip(Ms, Ws, xs):
            assert np.array_equal(M.matvec(x).cpu().numpy(), oracle.matvec_i8(W, x.cpu().numpy())), (B, W.shape)
    assert ops.device_status() == 0
