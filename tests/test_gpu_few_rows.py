"""GPU parity at the edges of the few-row products (one to eight activation rows: exact integer or e4m3 MMAs, tiles of 128 rows,
stages of 256 elements, K ranges cut over clusters of up to sixteen), against the oracle's dequantised weights in double precision."""
import numpy as np
import pytest

from gpu_util import F, out_with_canary, read_and_check_canary
from oracle import binding as orc
from test_gpu_rows import make

pytestmark = pytest.mark.gpu

# (out_dim, in_dim): one tile and stage; a row and a stage more; rows cut eight- and sixteenfold; a tile for every SM and one more
SHAPES = ((128, 256), (129, 512), (640, 2816), (200, 16384), (19072, 512))
# rows that end inside a stage
RAGGED = {"mlx": ((1, 64), (130, 320), (640, 2112), (200, 12352)), "q8_0": ((1, 32), (129, 288), (640, 2080)), "fp8": ((1, 16), (129, 272), (640, 2064), (300, 8208))}


def _norm_err(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("fmt,tiled", [("mlx", True), ("mlx_wide", True), ("mlx", False), ("mlx_wide", False), ("q4_k", True), ("q5_k", True), ("q6_k", True),
                                       ("q8_0", True), ("fp8", True), ("fp8", False)])
def test_few_rows(gpu, pkg, fmt, tiled):
    """The 2-norm of the error over that of the result.  An element of x is held to 2^-27 of its group's (FP8: exactly, to 2^-32 of its chunk's) largest, dot products of
    a group are exact, and f32 sums of at most 512 terms (16384 elements, 32 a group) add 2^-24 of a partial sum each: 3e-7 for sums that
    grow like a walk, three times that where minima and biases cancel most of the products.  Without the lowest digit it were 1.6e-6."""
    kind = fmt.split("_w")[0]
    shapes = (() if not tiled and kind == "q8_0" else SHAPES) + (RAGGED.get(kind, ()) if not tiled or kind == "q8_0" else ())
    for out_dim, in_dim in shapes:
        h, run, W, bias = make(gpu, pkg, fmt, tiled, out_dim, in_dim)
        W = np.asarray(W, dtype=np.float64).reshape(out_dim, in_dim)
        ok = ~np.isnan(W).any(1)
        for rows in (1, 2, 3, 4, 5, 8):
            x = pkg.synth.activations(("few", rows, in_dim), rows * in_dim, bf16=False).reshape(rows, in_dim)
            x[rows // 2] *= F(2.0 ** 40)  # every row has its own scale
            if rows > 2:
                x[0] = 0
            xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
            run(out, xo, rows)
            gpu.Sync()
            got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim).astype(np.float64)
            want = x.astype(np.float64) @ W.T + (0 if bias is None else bias)
            assert np.isnan(got[:, ~ok]).all() and not np.isnan(got[:, ok]).any()
            bound = 3e-6 if kind in ("fp8", "mlx") and rows > 4 else 1e-6  # (the several-row kernel: f32 sums of 4096 elements in tensor memory, 1.5e-6 measured)
            for m in range(rows):
                # (a matrix of one row has a single output, which may cancel to nothing: against its terms)
                size = np.linalg.norm(want[m, ok]) if ok.sum() > 100 else np.linalg.norm(np.abs(x[m].astype(np.float64)) @ np.abs(W[ok]).T)
                assert np.linalg.norm(got[m, ok] - want[m, ok]) <= bound * size, (out_dim, in_dim, rows, m)
            xo.Free(); out.Free()
        h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,tiled", [("mlx", False), ("fp8", True), ("fp8", False)])
def test_a_row_that_is_not_finite_is_nan(gpu, pkg, fmt, tiled):
    """As the tiled integer products: the row is NaN throughout, and no other row knows of it.  (Row-major FP8 widths from 4096 on.)"""
    out_dim, in_dim = 200, 4352
    h, run, W, _ = make(gpu, pkg, fmt, tiled, out_dim, in_dim)
    ok = ~np.isnan(np.asarray(W).reshape(out_dim, in_dim)).any(1)
    x = pkg.synth.activations(("odd", fmt), 2 * in_dim, bf16=False).reshape(2, in_dim)
    got = []
    for k, bad in ((0, 1.0), (0, np.nan), (517, np.inf), (in_dim - 1, -np.inf)):
        y = x.copy()
        y[1, k] = bad
        xo, out = gpu.from_numpy(y.reshape(-1)), out_with_canary(gpu, 2 * out_dim)
        run(out, xo, 2)
        gpu.Sync()
        got.append(read_and_check_canary(out, 2 * out_dim).reshape(2, out_dim).copy())
        xo.Free(); out.Free()
    assert np.isfinite(got[0][:, ok]).all()
    for g in got[1:]:
        assert np.isnan(g[1]).all() and np.array_equal(g[0, ok].view(np.uint32), got[0][0, ok].view(np.uint32))
    h.Free()


@pytest.mark.parametrize("rows", [2, 4, 8])
def test_row_major_weights_of_one_call_share_a_launch(gpu, pkg, rows):
    """Up to four weights a launch, the bits of separate calls; tiles of several weights in one K cut (short, long and ragged rows)."""
    for in_dim in (512, 2112, 9216):
        hs = [make(gpu, pkg, fmt, False, o, in_dim)[0] for fmt, o in (("mlx", 300), ("mlx_wide", 1), ("mlx", 128), ("mlx", 129), ("mlx", 64))]
        x = gpu.from_numpy(pkg.synth.activations(("share", in_dim), rows * in_dim, bf16=False))
        one, both = ([out_with_canary(gpu, rows * h.OutDim) for h in hs] for _ in range(2))
        for h, o in zip(hs, one):
            gpu.GemmMLX(o, x, h, rows)
        before = gpu.LaunchCount()
        gpu.GemmMLXMulti(both, x, hs, rows)
        assert gpu.LaunchCount() - before == 2
        gpu.Sync()
        for h, a, b in zip(hs, one, both):
            # (how K is cut, and with it the order of the sums, follows the number of tiles of a launch)
            u, v = (read_and_check_canary(t, rows * h.OutDim).astype(np.float64) for t in (a, b))
            assert np.linalg.norm(u - v) <= 5e-7 * np.linalg.norm(u)
        for t in hs + [x] + one + both:
            t.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("qtype,gen,in_dim", [("Q4_K", "q4k_matrix", 2048), ("Q6_K", "q6k_matrix", 4096), ("Q8_0", "q8_0_matrix", 2080)])
def test_small_gguf_matrices_need_no_order(gpu, pkg, qtype, gen, in_dim):
    """Matrices that are tiled by their size alone: streams without an order between them, and graphs beside each other, give the
    bits of calls one after another.  Inputs of very different sizes: rows that two calls mix up are off by orders of magnitude."""
    import torch
    from oracle import binding as orc
    out_dim, n = 512, 10
    m = gpu.UploadGGUFMatrix(getattr(orc, qtype), getattr(pkg.synth, gen)("free", out_dim, in_dim), in_dim, out_dim)
    for rows in (1, 3, 8, 13):
        xs = [gpu.from_numpy(pkg.synth.activations(("free", i), rows * in_dim, bf16=False) * F(2.0 ** (7 * (i % 8) - 24))) for i in range(n)]
        want, outs = ([out_with_canary(gpu, rows * out_dim) for _ in range(n)] for _ in range(2))
        for x, o in zip(xs, want):
            m.ProjectBatchToBuffer(o, x, rows)
        gpu.Sync()
        want = [read_and_check_canary(o, rows * out_dim).astype(np.float64) for o in want]

        def check():
            gpu.Sync()
            torch.cuda.synchronize()
            for a, o in zip(want, outs):
                b = read_and_check_canary(o, rows * out_dim).astype(np.float64)
                # (13 rows: the several-row kernel where a stream has scratch, passes of eight where it has none)
                assert np.linalg.norm(a - b) <= (0 if rows <= 8 else 1e-6) * np.linalg.norm(a)

        streams = [torch.cuda.Stream() for _ in range(n)]
        for _ in range(5):
            for s, x, o in zip(streams, xs, outs):
                m.ProjectBatchToBuffer(o, x, rows, s)
        check()
        graphs, capture = [], torch.cuda.Stream()
        for x, o in zip(xs, outs):
            o.Zero()
            g = torch.cuda.CUDAGraph()
            gpu.Sync()
            with torch.cuda.graph(g, stream=capture):
                m.ProjectBatchToBuffer(o, x, rows, capture)
            graphs.append(g)
        gpu.Sync()
        for o in outs:
            o.Upload(np.full(rows * out_dim + 64, 123.0, dtype=F))
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        check()
        del graphs
        for t in xs + outs:
            t.Free()
    m.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("tiled", [True, False])
def test_tiny_fp8_activations(gpu, pkg, tiled):
    """Rows, and single chunks of 256 elements beside ordinary ones, down to the subnormal floats: the e4m3 pieces and their scales stay exact.  Every output
    is off by f32 sums (2^-24 of a partial sum each, as above), and by half a subnormal (2^-150) for every sum of a piece and 128 elements
    and where the weight's scale meets them: at most 400 for 33 chunks of six pieces."""
    out_dim, in_dim = 300, 4352 if tiled else 8208
    w, s, _ = pkg.synth.fp8_linear("tiny", out_dim, in_dim)
    gpu.SetOption("fp8_layout", 2 if tiled else 1)
    try:
        h = gpu.UploadFP8E4M3Linear(w, s, None, out_dim, in_dim)
    finally:
        gpu.SetOption("fp8_layout", 0)
    W = np.asarray(orc.fp8_dequant(w, s, out_dim, in_dim), dtype=np.float64).reshape(out_dim, in_dim)
    for rows in (1, 2, 3):
        for exponent in (-100, -104, -106, -109, -112, -119, -122, -127, -136, -146):
            for chunk in (False, True):
                x = pkg.synth.activations(("tiny", rows, exponent), rows * in_dim, bf16=False).reshape(rows, in_dim)
                part = x[-1, 256:512] if chunk else x[-1]
                part[...] = (part.astype(np.float64) * 2.0 ** exponent).astype(F)
                xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
                gpu.GemmFP8E4M3Buffer(out, xo, rows, h)
                gpu.Sync()
                got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim).astype(np.float64)
                want = x.astype(np.float64) @ W.T
                bound = 1e-6 * np.linalg.norm(want, axis=1) + np.sqrt(out_dim) * 2.0 ** -150 * (1 + 400 * np.abs(s).max())
                assert np.isfinite(got).all() and (np.linalg.norm(got - want, axis=1) <= bound).all(), (rows, exponent, chunk)
                xo.Free(); out.Free()
    h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,tiled", [("mlx", True), ("mlx", False), ("q4_k", True), ("q5_k", True), ("q6_k", True), ("q8_0", True)])
def test_tiny_activations(gpu, pkg, fmt, tiled):
    """The same for the integer formats: a digit's unit goes down to 2^-149.  Roundings to a subnormal: two (scale and minimum or bias) for every block of 16 elements
    or more in each of the two pairs of digits, 2^-150 each."""
    out_dim, in_dim = 300, 2048
    h, run, W, _ = make(gpu, pkg, fmt, tiled, out_dim, in_dim)
    W = np.asarray(W, dtype=np.float64).reshape(out_dim, in_dim)
    for rows in (1, 2, 4, 8):
        for exponent in (-96, -99, -104, -112, -121, -124, -127, -136, -146):
            for chunk in (False, True):
                x = pkg.synth.activations(("tiny", rows, exponent), rows * in_dim, bf16=False).reshape(rows, in_dim)
                part = x[-1, 256:512] if chunk else x[-1]
                part[...] = (part.astype(np.float64) * 2.0 ** exponent).astype(F)
                xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
                run(out, xo, rows)
                gpu.Sync()
                got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim).astype(np.float64)
                want = x.astype(np.float64) @ W.T
                bound = 1e-6 * np.linalg.norm(want, axis=1) + np.sqrt(out_dim) * 2.0 ** -150 * (4 * in_dim / 16)
                assert (np.linalg.norm(got - want, axis=1) <= bound).all(), (rows, exponent, chunk)
                xo.Free(); out.Free()
    h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,widths,rows", [("q8_0", (14624, 29216), (1, 3, 8, 12)), ("fp8", (15680, 31264), (1, 2)), ("mlx", (20800, 40992), (1, 2, 4))])
def test_rows_too_wide_for_one_cta(gpu, pkg, fmt, widths, rows):
    """Products without scratch whose K range is cut for no other reason than that its activations fill a CTA's shared memory: 75 tiles of rows too many for one
    piece, 74 for two.  Rows repeat every 96th one, which keeps the reference small; the bits of equal rows are equal."""
    for out_dim, in_dim in zip((9600, 9472), widths):
        part = 96
        n = -(-out_dim // part)
        if fmt == "mlx":
            in_dim = in_dim // 64 * 64
            w, s, b = (np.asarray(t) for t in pkg.synth.mlx_weight("wide", part, in_dim))
            W = orc.mlx_dequant(w, s, b, part, in_dim, 64)
            w, s, b = (np.tile(t.reshape(part, -1), (n, 1))[:out_dim].reshape(-1) for t in (w, s, b))
            hs = [gpu.UploadMLXWeight(w, s, b, in_dim, out_dim, 64, True)]
            half = out_dim // 2
            hs += [gpu.UploadMLXWeight(w[:half * in_dim // 8], s[:half * in_dim // 64], b[:half * in_dim // 64], in_dim, half, 64, True) for _ in range(2)]

            def run(o, x, m):
                gpu.GemmMLX(o, x, hs[0], m)
                outs = [out_with_canary(gpu, m * half) for _ in range(2)]
                gpu.GemmMLXMulti(outs, x, hs[1:], m)  # (their tiles count together)
                gpu.Sync()
                both = [read_and_check_canary(t, m * half).reshape(m, half) for t in outs]
                assert np.array_equal(both[0], both[1])
                assert np.linalg.norm(both[0] - o.Download()[:m * out_dim].reshape(m, out_dim)[:, :half]) <= 1e-6 * np.linalg.norm(both[0])
                for t in outs:
                    t.Free()
        elif fmt == "fp8":
            in_dim = in_dim // 16 * 16
            w, s, _ = pkg.synth.fp8_linear("wide", part, in_dim)
            W = orc.fp8_dequant(w, s, part, in_dim)
            w, s = np.tile(w.reshape(part, -1), (n, 1))[:out_dim].reshape(-1), np.tile(s, n)[:out_dim]
            gpu.SetOption("fp8_layout", 1)
            hs = [gpu.UploadFP8E4M3Linear(w, s, None, out_dim, in_dim)]
            gpu.SetOption("fp8_layout", 0)
            run = lambda o, x, m: gpu.GemmFP8E4M3Buffer(o, x, m, hs[0])
        else:
            raw = np.asarray(pkg.synth.q8_0_matrix("wide", part, in_dim))
            W = orc.gguf_dequant(raw, orc.Q8_0, in_dim, part)
            hs = [gpu.UploadGGUFMatrix(orc.Q8_0, np.tile(raw.reshape(part, -1), (n, 1))[:out_dim].reshape(-1), in_dim, out_dim)]
            run = lambda o, x, m: hs[0].ProjectBatchToBuffer(o, x, m)
        W = np.asarray(W, dtype=np.float64).reshape(part, in_dim)
        for m in rows:
            x = pkg.synth.activations(("wide", m, in_dim), m * in_dim, bf16=False).reshape(m, in_dim)
            xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, m * out_dim)
            run(out, xo, m)
            gpu.Sync()
            got = read_and_check_canary(out, m * out_dim).reshape(m, out_dim)
            assert np.array_equal(got, np.tile(got[:, :part], (1, n))[:, :out_dim])
            want = x.astype(np.float64) @ W.T
            assert np.linalg.norm(got[:, :part] - want) <= 1e-6 * np.linalg.norm(want)
            xo.Free(); out.Free()
        for h in hs:
            h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,n", [("q4_k", 2048), ("q5_k", 1024), ("q6_k", 2048), ("q8_0", 2048), ("q8_0", 2080), ("q8_0", 4128)])
@pytest.mark.parametrize("rows", [1, 2])
def test_outputs_of_small_gguf_matrices_that_overlap_x(gpu, pkg, fmt, n, rows):
    """An output in the place of x, or across its edge, of matrices that are tiled by their size alone and otherwise use no scratch: x is
    prepared in front, and the bits are those of buffers apart."""
    from test_gpu_rows import GGUF
    qtype, gen = GGUF[fmt]
    raw = getattr(pkg.synth, gen)("over", n, n)
    h, other_h = (gpu.UploadGGUFMatrix(qtype, raw, n, n) for _ in range(2))
    x = pkg.synth.activations(("over", rows), rows * n, bf16=False)
    xo, want = gpu.from_numpy(x), out_with_canary(gpu, rows * n)
    h.ProjectBatchToBuffer(want, xo, rows)
    gpu.Sync()
    want = read_and_check_canary(want, rows * n)
    buf, other = gpu.Malloc(2 * rows * n), gpu.Malloc(rows * n)
    for out_at, x_at in ((0, 0), (0, rows * n // 2), (rows * n - 4, 0)):
        for _ in range(20):
            out, xb = gpu.wrap(buf.Ptr + 4 * out_at, 4 * rows * n), gpu.wrap(buf.Ptr + 4 * x_at, 4 * rows * n)
            xb.Upload(x)
            h.ProjectBatchToBuffer(out, xb, rows)
            gpu.Sync()
            assert np.array_equal(out.Download().view(np.uint32), want.view(np.uint32))
            xb.Upload(x)
            gpu.ProjectQ4PairToBuffers(out, other, xb, rows, h, other_h)
            gpu.Sync()
            assert np.array_equal(out.Download().view(np.uint32), want.view(np.uint32))
            assert np.array_equal(other.Download().view(np.uint32), want.view(np.uint32))
    for t in (h, other_h, xo, buf, other):
        t.Free()
    assert gpu.KernelStatus() == 0


def test_ragged_gguf_rows_need_no_order_in_any_layout(gpu, pkg):
    """Q8_0 rows that end inside a stage, with the tensor-core layout asked for: launches on streams without an order between them give the bits of calls
    one after another (eight rows of values of very different sizes, so that activations of two calls do not mix unseen)."""
    import torch
    out_dim, in_dim, rows, n = 512, 4128, 8, 10
    gpu.SetOption("gguf_layout", 2)
    try:
        m = gpu.UploadGGUFMatrix(orc.Q8_0, pkg.synth.q8_0_matrix("free", out_dim, in_dim), in_dim, out_dim)
    finally:
        gpu.SetOption("gguf_layout", 0)
    xs = [gpu.from_numpy(pkg.synth.activations(("free", i), rows * in_dim, bf16=False) * F(2.0 ** (7 * (i % 8) - 24))) for i in range(n)]
    want, outs = ([out_with_canary(gpu, rows * out_dim) for _ in range(n)] for _ in range(2))
    before = gpu.LaunchCount()
    for x, o in zip(xs, want):
        m.ProjectBatchToBuffer(o, x, rows)
    assert gpu.LaunchCount() - before == n  # nothing is prepared in front, in scratch that they share
    gpu.Sync()
    streams = [torch.cuda.Stream() for _ in range(n)]
    for _ in range(5):
        for s, x, o in zip(streams, xs, outs):
            m.ProjectBatchToBuffer(o, x, rows, s)
    gpu.Sync()
    torch.cuda.synchronize()
    for a, b in zip(want, outs):
        a, b = (read_and_check_canary(t, rows * out_dim) for t in (a, b))
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for t in [m] + xs + want + outs:
        t.Free()
    assert gpu.KernelStatus() == 0


# The 2-norm of the error over that of the result, x normal.  Products and biases are each five times the sum that they cancel to; their f32 sums, a term for each
# of 64 groups, added by 16 chunks, are off by 2^-25 of at most 64 partial sums that grow like a walk: 4e-7 (1.6e-7 measured).  The several-row kernel's sums in
# tensor memory are off by 7.7e-7.
@pytest.mark.parametrize("rows", [5, 8])
def test_several_mlx_weights_of_a_call_keep_exact_sums(gpu, pkg, rows):
    in_dim, out_dim = 4096, 1024
    hs, Ws = [], []
    for k in range(4):
        w, sc, b = pkg.synth.mlx_weight(("lines", k), out_dim, in_dim)
        hs.append(gpu.UploadMLXWeight(w, sc, b, in_dim, out_dim, 64, True))
        Ws.append(np.asarray(orc.mlx_dequant(w, sc, b, out_dim, in_dim, 64), dtype=np.float64).reshape(out_dim, in_dim))
    x = pkg.synth.activations(("lines", rows), rows * in_dim, bf16=False)
    xo, outs = gpu.from_numpy(x), [out_with_canary(gpu, rows * out_dim) for _ in hs]
    gpu.GemmMLXMulti(outs, xo, hs, rows)
    gpu.Sync()
    for W, out in zip(Ws, outs):
        got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim).astype(np.float64)
        err = _norm_err(got, x.reshape(rows, in_dim).astype(np.float64) @ W.T)
        assert err <= 4e-7, err
    for t in hs + [xo] + outs:
        t.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,out_dim,in_dim,rows", [("q4_k", 10000, 256, 8), ("q5_k", 10000, 512, 5), ("q5_k", 640, 1024, 10), ("q6_k", 1024, 2048, 16), ("q6_k", 640, 2560, 24),
                                                     ("q6_k", 1536, 4096, 12)])
def test_small_gguf_matrices_keep_exact_sums(gpu, pkg, fmt, out_dim, in_dim, rows):
    """Sums of a block's products are exact here, f32 sums of at most 4096 / 16 of them off by 2^-25 of partial sums that grow like a walk: 1.2e-7 for the longest, by 16 chunks where
    minima cancel them (1.0e-7 measured).  The several-row kernel: 4.2e-7 to 5.1e-7 with minima, 1.2e-7 to 1.4e-7 for Q6_K.  Rows of further passes have the bits of calls by themselves."""
    from test_gpu_rows import GGUF
    qtype, gen = GGUF[fmt]
    raw = getattr(pkg.synth, gen)("exact", out_dim, in_dim)
    h = gpu.UploadGGUFMatrix(qtype, raw, in_dim, out_dim)
    W = np.asarray(orc.gguf_dequant(raw, qtype, in_dim, out_dim), dtype=np.float64).reshape(out_dim, in_dim)
    x = pkg.synth.activations(("exact", rows), rows * in_dim, bf16=False).reshape(rows, in_dim)
    xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
    h.ProjectBatchToBuffer(out, xo, rows)
    gpu.Sync()
    got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim)
    assert _norm_err(got.astype(np.float64), x.astype(np.float64) @ W.T) <= 1.2e-7
    last = (rows - 1) // 8 * 8
    xl, one = gpu.from_numpy(x[last:].reshape(-1)), out_with_canary(gpu, (rows - last) * out_dim)
    h.ProjectBatchToBuffer(one, xl, rows - last)
    gpu.Sync()
    assert np.array_equal(got[last:].view(np.uint32), read_and_check_canary(one, (rows - last) * out_dim).reshape(-1, out_dim).view(np.uint32))
    for t in (h, xo, out, xl, one):
        t.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,out_dim,in_dim", [("q8_0", 19072, 4096), ("q6_k", 19072, 4096), ("q8_0", 1000, 30720), ("q6_k", 1000, 30720)])
def test_sums_of_many_blocks(gpu, pkg, fmt, out_dim, in_dim):
    """Long K ranges, with a tile for every SM and with few tiles.  Sums of a chunk of 256 elements meet a sum of at most 16 chunks (120 of them cut into eight
    ranges and more): 2^-25 of 16 partial sums of a chunk and of 16 of chunks, that grow like walks, 1.2e-7 for both digits' sums (1.0e-7 measured; one sum of all
    blocks 1.5e-7 to 2.1e-7).  Rows repeat every 100th one."""
    from test_gpu_rows import GGUF
    qtype, gen = GGUF[fmt]
    part = 100
    raw = np.asarray(getattr(pkg.synth, gen)("many", part, in_dim))
    W = np.asarray(orc.gguf_dequant(raw, qtype, in_dim, part), dtype=np.float64).reshape(part, in_dim)
    h = gpu.UploadGGUFMatrix(qtype, np.tile(raw.reshape(part, -1), (-(-out_dim // part), 1))[:out_dim].reshape(-1), in_dim, out_dim)
    for rows in (1, 2, 4, 8):
        x = pkg.synth.activations(("many", rows), rows * in_dim, bf16=False).reshape(rows, in_dim)
        xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
        h.ProjectBatchToBuffer(out, xo, rows)
        gpu.Sync()
        got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim)
        err = _norm_err(got[:, :part].astype(np.float64), x.astype(np.float64) @ W.T)
        assert err <= 1.3e-7, (rows, err)
        assert np.array_equal(got, np.tile(got[:, :part], (1, -(-out_dim // part)))[:, :out_dim])
        xo.Free(); out.Free()
    h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("fmt,layout,out_dim,in_dim,rows", [
    ("fp8", 1, 300, 8208, (1, 2)), ("fp8", 1, 2560, 2560, (1, 2)), ("q6_k", 0, 1024, 2048, (1, 2, 4, 8, 10)), ("q6_k", 0, 300, 8192, (1, 2, 5)), ("q6_k", 2, 300, 2048, (5, 8)),
    ("q8_0", 0, 640, 2080, (1, 2, 4, 8)), ("q8_0", 2, 300, 2048, (5, 8)), ("q8_0", 2, 19000, 768, (5, 8))])
@pytest.mark.parametrize("cluster", [1, 0])
def test_an_infinity_in_few_rows(gpu, pkg, fmt, layout, out_dim, in_dim, rows, cluster):
    """Weights without a minimum whose other numbers of rows run on kernels of f32 or f16 products: +-inf by the weight's sign, NaN where two infinities meet, the weight
    is zero or a NaN code, as there; the other rows keep their bits.  Outputs of one CTA a tile, of clusters, and of sums that meet in scratch."""
    from test_gpu_rows import GGUF
    option = "fp8_layout" if fmt == "fp8" else "gguf_layout"
    gpu.SetOption(option, layout)
    try:
        if fmt == "fp8":
            w, s, b = pkg.synth.fp8_linear("inf", out_dim, in_dim, bias=True)
            w[(out_dim - 1) * in_dim + 7] = 0x7F
            h = gpu.UploadFP8E4M3Linear(w, s, b, out_dim, in_dim)
            W, run = orc.fp8_dequant(w, s, out_dim, in_dim), lambda o, x, n: gpu.GemmFP8E4M3Buffer(o, x, n, h)
        else:
            raw = getattr(pkg.synth, GGUF[fmt][1])("inf", out_dim, in_dim)
            h = gpu.UploadGGUFMatrix(GGUF[fmt][0], raw, in_dim, out_dim)
            W, run = orc.gguf_dequant(raw, GGUF[fmt][0], in_dim, out_dim), lambda o, x, n: h.ProjectBatchToBuffer(o, x, n)
    finally:
        gpu.SetOption(option, 0)
    W = np.asarray(W, dtype=np.float64).reshape(out_dim, in_dim)
    gpu.SetOption("mlx_cluster", cluster)
    try:
        for m in rows:
            x = pkg.synth.activations(("inf", m), m * in_dim, bf16=False).reshape(m, in_dim)
            got = []
            for bad in ({}, {100: np.inf}, {700: -np.inf, 701: F(1e30)}, {5: np.inf, in_dim - 3: np.inf}, {64: np.nan}):
                y = x.copy()
                for k, v in bad.items():
                    y[m // 2, k] = v
                xo, out = gpu.from_numpy(y.reshape(-1)), out_with_canary(gpu, m * out_dim)
                run(out, xo, m)
                gpu.Sync()
                got.append(read_and_check_canary(out, m * out_dim).reshape(m, out_dim))
                if bad:
                    with np.errstate(invalid="ignore"):
                        want = (y[m // 2].astype(np.float64) * W).sum(-1).astype(F)
                    assert np.array_equal(got[-1][m // 2], want, equal_nan=True), (m, bad)
                    others = [r for r in range(m) if r != m // 2]
                    assert np.array_equal(got[-1][others].view(np.uint32), got[0][others].view(np.uint32))
                xo.Free(); out.Free()
    finally:
        gpu.SetOption("mlx_cluster", 1)
    h.Free()
    assert gpu.KernelStatus() == 0


@pytest.mark.parametrize("option,value", [("mlx_unpack", 1), ("mlx_unpack", 2), ("mlx_ctas_per_sm", 1)])
@pytest.mark.parametrize("rows", [1, 3])
def test_options_of_the_cuda_core_kernels_reach_them(gpu, pkg, option, value, rows):
    """Row-major weights that go to the tensor cores by default: an option of the streaming kernel has it run, as "mlx_rows" does (rows of a warp change no sum)."""
    out_dim, in_dim = 1000, 8192
    h, run, _, _ = make(gpu, pkg, "mlx", False, out_dim, in_dim)
    x = gpu.from_numpy(pkg.synth.activations(("opt", rows), rows * in_dim, bf16=False))

    def product(**opts):
        for k, v in opts.items():
            gpu.SetOption(k, v)
        try:
            out = out_with_canary(gpu, rows * out_dim)
            run(out, x, rows)
            gpu.Sync()
            got = read_and_check_canary(out, rows * out_dim).view(np.uint32).copy()
            out.Free()
            return got
        finally:
            for k in opts:
                gpu.SetOption(k, 0)

    plain, asked = product(), product(**{option: value})
    assert np.array_equal(asked, product(**{option: value, "mlx_rows": 1}))
    assert not np.array_equal(asked, plain)
    for t in (h, x):
        t.Free()


def test_a_tile_more_than_sms_shares_the_last_round(gpu, pkg):
    """149 tiles of 8192 elements with eight rows, on the several-row kernel: the items behind the first round are shared by clusters, whose shorter sums in tensor memory
    keep the error at 5e-7 (a CTA with two tiles and the whole range: 8.4e-7).  Rows repeat every 100th one; bound halfway between."""
    part, out_dim, in_dim, rows = 100, 149 * 128, 8192, 8
    raw = np.asarray(pkg.synth.q4k_matrix("more", part, in_dim))
    W = np.asarray(orc.gguf_dequant(raw, orc.Q4_K, in_dim, part), dtype=np.float64).reshape(part, in_dim)
    h = gpu.UploadGGUFMatrix(orc.Q4_K, np.tile(raw.reshape(part, -1), (-(-out_dim // part), 1))[:out_dim].reshape(-1), in_dim, out_dim)
    x = pkg.synth.activations("more", rows * in_dim, bf16=False).reshape(rows, in_dim)
    xo, out = gpu.from_numpy(x.reshape(-1)), out_with_canary(gpu, rows * out_dim)
    h.ProjectBatchToBuffer(out, xo, rows)
    gpu.Sync()
    got = read_and_check_canary(out, rows * out_dim).reshape(rows, out_dim).astype(np.float64)
    err = np.linalg.norm(got - np.tile(x.astype(np.float64) @ W.T, (1, -(-out_dim // part)))[:, :out_dim]) / np.linalg.norm(got)
    assert err <= 6.7e-7, err
    for t in (h, xo, out):
        t.Free()
    assert gpu.KernelStatus() == 0
