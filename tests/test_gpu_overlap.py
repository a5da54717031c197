"""Launches behind one another in a stream, eagerly and in a CUDA graph: a launch may begin while the one before it ends,
and stream order holds all the same.  What the launch before writes may be anything that the next one is given: x, the
matrix with its tables and offsets, the device's job table, a buffer that an earlier launch still reads.  Bit-exact against
the CPU oracle over many runs."""
import numpy as np
import pytest

from conftest import cuda_ok
import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]

if cuda_ok():
    import torch
    from matvans_b200 import codec, ops

RUNS = 40


def gauss(rng, shape, sigma=4.0, lim=60):
    return np.clip(np.round(rng.normal(0, sigma, size=shape)), -lim, lim).astype(np.int8)


def put(dst, src):
    """dst = src by an ordinary kernel (a contiguous copy_ would be a memory copy, which orders more than a kernel does)."""
    torch.add(src.view(torch.uint8), 0, out=dst.view(torch.uint8))


def eager_and_graph(body):
    """body() enqueues work and returns its outputs: eagerly, then captured and replayed twice."""
    yield body()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        out = body()
    for _ in range(2):
        g.replay()
        yield out


def two_q8(rng, rows, cols, local):
    """Two matrices whose encodings fill buffers of the same sizes, and the device arrays of both."""
    encs = [codec.q8_encode(gauss(rng, (rows, cols), s), local=local, seg_quads=64) for s in (2.0, 5.0)]
    Ws = [ops.Q8Matrix(e).decode().cpu().numpy() for e in encs]
    size = {k: max(e[k].size for e in encs) for k in ("blocks", "blk_off", "tbl", "tbl_off")}
    for e in encs:
        for k, n in size.items():
            e[k] = np.concatenate([e[k], np.full(n - e[k].size, e[k][-1], e[k].dtype)])
        for k in ("max_blk_rows", "tbl_stripe_max"):
            e[k] = max(x[k] for x in encs)
    M = ops.Q8Matrix(encs[0])
    src = [[ops.Q8Matrix(e).__dict__[k] for k in size] for e in encs]
    dst = [M.__dict__[k] for k in size]
    return M, Ws, src, dst


@pytest.mark.parametrize("rows,cols,local", [(320, 1024, True), (4800, 512, False), (9600, 256, True)])
@pytest.mark.parametrize("B", [1, 16, 33])
def test_q8_matrix_written_by_the_launch_before(rows, cols, local, B):
    rng = np.random.default_rng(rows + B)
    M, Ws, src, dst = two_q8(rng, rows, cols, local)
    x = torch.from_numpy(rng.integers(-128, 128, size=(B, cols)).astype(np.int8)).cuda()
    refs = [oracle.matvec_i8(W, x.cpu().numpy()) for W in Ws]

    def body():
        ys = []
        for i in range(RUNS):
            for d, s in zip(dst, src[i % 2]):  # the tables and offsets last
                put(d, s)
            ys.append(M.matvec(x))
        return ys
    for ys in eager_and_graph(body):
        for i, y in enumerate(ys):
            assert np.array_equal(y.cpu().numpy(), refs[i % 2]), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 8])
def test_job_table_written_by_the_launch_before(B):
    rng = np.random.default_rng(B)
    Ms = [ops.Q8Matrix.encode(gauss(rng, (640, 512))) for _ in range(4)]
    Ws = [M.decode().cpu().numpy() for M in Ms]
    x = torch.from_numpy(rng.integers(-128, 128, size=(B, 512)).astype(np.int8)).cuda()
    S = [ops.Q8Stack(Ms[i:i + 2], batch=B, xs=[x, x]) for i in (0, 2)]
    tables = [s.jobs_dev.clone() for s in S]
    refs = [[oracle.matvec_i8(W, x.cpu().numpy()) for W in Ws[i:i + 2]] for i in (0, 2)]

    def body():
        out = []
        for i in range(RUNS):
            put(S[0].jobs_dev, tables[i % 2])
            S[0].run()
            out.append([y.clone() for y in S[i % 2].ys])
        return out
    for out in eager_and_graph(body):
        for i, ys in enumerate(out):
            assert all(np.array_equal(y.cpu().numpy(), r) for y, r in zip(ys, refs[i % 2])), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("kind", ["awr", "aws", "wpr"])
def test_reference_layout_tables_written_by_the_launch_before(kind):
    rng = np.random.default_rng(len(kind))
    cls = {"awr": ops.AwrMatrix, "aws": ops.AwsMatrix, "wpr": ops.WprMatrix}[kind]
    Ws = [gauss(rng, (256, 1024), s) for s in (2.0, 6.0)]
    Ms = [cls.encode(W) for W in Ws]
    names = [k for k, v in Ms[0].__dict__.items() if isinstance(v, torch.Tensor)]
    if kind == "wpr":  # (the least symbol and the number of symbols go with a call, not with the arrays)
        Ws[1] = Ws[0][::-1].copy()
        Ms[1] = cls.encode(Ws[1])
    M = cls.encode(Ws[0])
    for k in names:
        n = max(getattr(m, k).numel() for m in Ms)
        for m in Ms + [M]:
            t = getattr(m, k)
            setattr(m, k, torch.cat([t, t.new_zeros(n - t.numel())]))
    for a in ("n_words", "payload_size"):
        if hasattr(M, a):
            setattr(M, a, max(getattr(m, a) for m in Ms))
    x = torch.from_numpy(rng.integers(-128, 128, size=(1, 1024)).astype(np.int8)).cuda()
    refs = [oracle.matvec_i8(W, x.cpu().numpy()) for W in Ws]

    def body():
        ys = []
        for i in range(RUNS):
            for k in names:
                put(getattr(M, k), getattr(Ms[i % 2], k))
            ys.append(M.matvec(x))
        return ys
    for ys in eager_and_graph(body):
        for i, y in enumerate(ys):
            assert np.array_equal(y.cpu().numpy(), refs[i % 2]), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("kinds", [("awr", "awr"), ("aws", "aws"), ("awr", "wpr"), ("aws", "q8"), ("wpr", "wpr")])
def test_outputs_as_the_next_launch_s_input(kinds):
    # two matrices in turn, each one's int8 output the next one's x, in two buffers that change roles
    rng = np.random.default_rng(sum(map(ord, "".join(kinds))))
    n = 512
    cls = {"awr": ops.AwrMatrix, "aws": ops.AwsMatrix, "wpr": ops.WprMatrix, "q8": ops.Q8Matrix}
    Ws = [gauss(rng, (n, n)) for _ in kinds]
    Ms = [cls[k].encode(W) for k, W in zip(kinds, Ws)]
    x0 = rng.integers(-128, 128, size=n).astype(np.int8)
    bufs = [torch.empty(n, dtype=torch.int8, device="cuda") for _ in range(2)]
    start = torch.from_numpy(x0).cuda()
    y = torch.empty((1, n), dtype=torch.int32, device="cuda")
    scale = np.float32(2e-3)

    def absmax(yh):
        d = np.float32(np.abs(yh.astype(np.int64)).max()) / np.float32(127.0)
        return np.rint(yh.astype(np.float32) / d).astype(np.int8)

    want, xh = [], x0
    for i in range(RUNS):
        yh = oracle.matvec_i8(Ws[i % 2], xh[None, :])[0]
        fused = kinds[i % 2] in ("awr", "aws")
        xh = np.clip(np.rint(yh.astype(np.float32) * scale), -128, 127).astype(np.int8) if fused else absmax(yh)
        want.append(xh)

    def body():
        out, cur = [], start
        for i in range(RUNS):
            M, dst = Ms[i % 2], bufs[i % 2]
            if kinds[i % 2] in ("awr", "aws"):
                M.matvec_requant(cur, float(scale), out=dst)
            else:
                M.matvec(cur, out=y)
                ops.requant_absmax(y, out8=dst)
            cur = dst
            if i % 7 == 6:
                out.append((i, cur.clone()))
        out.append((RUNS - 1, cur))
        return out
    for out in eager_and_graph(body):
        for i, v in out:
            assert np.array_equal(v.cpu().numpy(), want[i]), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 3, 16])
def test_plans_that_share_buffers(B):
    # a chain whose output is its own next input, and a stack that reads it and whose outputs every run overwrites
    rng = np.random.default_rng(B)
    dims = [512, 1024, 512]
    Ws = [gauss(rng, (dims[i + 1], dims[i])) for i in range(2)]
    Ms = [ops.Q8Matrix.encode(W) for W in Ws]
    x = torch.empty((B, 512), dtype=torch.int8, device="cuda")
    x0 = torch.from_numpy(rng.integers(-127, 128, size=(B, 512)).astype(np.int8)).cuda()
    scales = [2e-3, 2e-3]
    C = ops.Q8Chain(Ms, scales, batch=B, x0=x)
    S = ops.Q8Stack([Ms[0], Ms[0]], batch=B, xs=[C.out8, C.out8])
    want, xh = [], x0.cpu().numpy()
    for _ in range(RUNS):
        for W, s in zip(Ws, scales):
            xh = np.clip(np.rint(oracle.matvec_i8(W, xh).astype(np.float32) * np.float32(s)), -128, 127).astype(np.int8)
        want.append(xh)

    def body():
        put(x, x0)
        out = []
        for i in range(RUNS):
            C.run()
            S.run()
            S.run()
            if i % 5 == 4:
                out.append((i, C.out8.clone(), S.ys[1].clone()))
            put(x, C.out8)
        return out
    for out in eager_and_graph(body):
        for i, o8, y in out:
            assert np.array_equal(o8.cpu().numpy(), want[i]), i
            assert np.array_equal(y.cpu().numpy(), oracle.matvec_i8(Ws[0], want[i])), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("kind", ["q8", "awr", "aws", "wpr"])
def test_tables_written_late_by_a_launch_that_lets_the_next_begin_early(kind):
    # the launch before is one of the library's own products, which lets its successor begin long before it writes: an
    # identity matrix whose int8 output, byte for byte, is one of the next matrix's tables.  W and -W: tables of the same
    # sizes, in another order
    rng = np.random.default_rng(len(kind) + 11)
    rows, cols = 256, 1024
    W = gauss(rng, (rows, cols), 3.0, 6)  # (the extremes of both are there)
    Ws = [W, -W]
    enc = {"q8": lambda w: ops.Q8Matrix.encode(w, local=False, seg_quads=64), "awr": ops.AwrMatrix.encode,
           "aws": ops.AwsMatrix.encode, "wpr": ops.WprMatrix.encode}[kind]
    Ms = [enc(w) for w in Ws]
    table = {"q8": "tbl", "awr": "ppf", "aws": "ppf", "wpr": "ppf"}[kind]  # written by the product, the rest by kernels
    M = enc(W)
    if kind == "wpr":
        assert Ms[0].min_value == Ms[1].min_value and Ms[0].G == Ms[1].G
    names = [k for k, v in M.__dict__.items() if isinstance(v, torch.Tensor) and k != table]
    for k in names:
        n = max(getattr(m, k).numel() for m in Ms)
        for m in Ms + [M]:
            t = getattr(m, k)
            setattr(m, k, torch.cat([t, t.new_zeros(n - t.numel())]))
    for a in ("n_words", "payload_size", "max_blk_rows", "tbl_stripe_max"):
        if hasattr(M, a):
            setattr(M, a, max(getattr(m, a) for m in Ms))
    nbytes = getattr(M, table).numel() * getattr(M, table).element_size()
    assert nbytes == getattr(Ms[1], table).numel() * getattr(M, table).element_size()
    n = -(-nbytes // 128) * 128
    copier = ops.AwrMatrix.encode(np.eye(n, dtype=np.int8))
    dst = torch.zeros(n, dtype=torch.int8, device="cuda")
    dst[:nbytes] = getattr(M, table).view(torch.int8)
    setattr(M, table, dst[:nbytes].view(getattr(M, table).dtype))
    srcs = [torch.cat([getattr(m, table).view(torch.int8), dst.new_zeros(n - nbytes)]) for m in Ms]
    if kind == "q8":
        M._view = M.view()
    x = torch.from_numpy(rng.integers(-128, 128, size=(1, cols)).astype(np.int8)).cuda()
    refs = [oracle.matvec_i8(w, x.cpu().numpy()) for w in Ws]

    def body():
        ys = []
        for i in range(RUNS):
            for k in names:
                put(getattr(M, k), getattr(Ms[i % 2], k))
            copier.matvec_requant(srcs[i % 2], 1.0, out=dst)
            ys.append(M.matvec(x))
        return ys
    for ys in eager_and_graph(body):
        for i, y in enumerate(ys):
            assert np.array_equal(y.cpu().numpy(), refs[i % 2]), i
    assert ops.device_status() == 0


@pytest.mark.parametrize("B", [1, 2, 40, 70])
def test_float_form_and_scales_written_by_the_launch_before(B):
    # x, dY, row scales and the matrix by kernels right before each product, the float form both ways and the scaled integer
    # product: what an undisturbed call gives (dX to the order of its additions: two stripes' parts add up the same either way)
    rng = np.random.default_rng(B)
    rows, cols = 64, 2048
    M, Ws, src, dst = two_q8(rng, rows, cols, True)
    fs = [torch.from_numpy(rng.uniform(1e-3, 1e-2, size=rows).astype(np.float32)).cuda() for _ in range(2)]
    xf = [torch.randn((B, cols), device="cuda").bfloat16() for _ in range(2)]
    dy = [torch.randn((B, rows), device="cuda").bfloat16() for _ in range(2)]
    x8 = [torch.randint(-128, 128, (B, cols), dtype=torch.int8, device="cuda") for _ in range(2)]
    s, x, d, q = (torch.empty_like(v[0]) for v in (fs, xf, dy, x8))

    def calls():
        return [M.matvec_bf16(x, s), M.matvec_t_bf16(d, s), *M.matvec(q, scales=s)]
    want = []
    for i in range(2):
        for t, v in zip(dst + [s, x, d, q], src[i] + [fs[i], xf[i], dy[i], x8[i]]):
            put(t, v)
        torch.cuda.synchronize()
        want.append(calls())
        assert np.array_equal(want[i][2].cpu().numpy(), oracle.matvec_i8(Ws[i], x8[i].cpu().numpy()))
    torch.cuda.synchronize()

    def body():
        out = []
        for i in range(RUNS):
            for t, v in zip(dst + [s, x, d, q], src[i % 2] + [fs[i % 2], xf[i % 2], dy[i % 2], x8[i % 2]]):
                put(t, v)
            out.append(calls())
        return out
    for out in eager_and_graph(body):
        for i, got in enumerate(out):
            assert all(torch.equal(a, b) for a, b in zip(got, want[i % 2])), i
    assert ops.device_status() == 0
