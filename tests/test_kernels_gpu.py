"""Numerics of every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _status_clean():
    from piper_b200.ops import native

    yield
    native.check_status()


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


def _max_err(a, b):
    """Largest elementwise error, relative to the largest reference magnitude: one wrong element shows here even
    where the norm-wise error of a large tensor hides it."""
    a, b = a.float(), b.float()
    return ((a - b).abs().max() / (b.abs().max() + 1e-12)).item()


def _close(a, b, tol):
    """Norm-wise relative error below ``tol`` and every element within ``4 * tol`` of the reference's scale."""
    assert a.shape == b.shape, (a.shape, b.shape)
    assert torch.isfinite(a.float()).all()
    return _rel_err(a, b) < tol and _max_err(a, b) < 4 * tol


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 768, 192), (200, 328, 136), (4096, 1024, 512)])
def test_gemm_forward_layout(M, N, K):
    from piper_b200.ops import native

    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    c = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    native.lib().gemm(a, b, c, False, False, False, native.status_tensor())
    ref = a.float() @ b.float().t()
    assert _close(c, ref, 1e-2)


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 320), (200, 328, 136)])
def test_gemm_dgrad_and_wgrad_layouts(M, N, K):
    from piper_b200.ops import native

    torch.manual_seed(1)
    st = native.status_tensor()
    # dgrad: C[M,N] = A[M,K] * Bs[K,N]  (B stored [K, N])
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    bs = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    c = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    native.lib().gemm(a, bs, c, False, True, False, st)
    assert _close(c, a.float() @ bs.float(), 1e-2)
    # wgrad: C[M,N] = As[K,M]^T * Bs[K,N], fp32 accumulate into an existing buffer
    as_ = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    ref = acc + as_.float().t() @ bs.float()
    native.lib().gemm(as_, bs, acc, True, True, True, st)
    assert _close(acc, ref, 1e-2)
    # A MN-major with B K-major
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    c2 = torch.empty(M, N, device="cuda", dtype=torch.float32)
    native.lib().gemm(as_, b, c2, True, False, False, st)
    assert _close(c2, as_.float().t() @ b.float().t(), 1e-2)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 320), (200, 328, 136), (2304, 4608, 192)])
def test_gemm_256_tile_all_layouts(M, N, K):
    """The 256x256-tile kernel against fp32 references: every operand layout, both epilogues, ragged edges and
    (last shape) more tiles than SMs so that CTAs walk several tiles and reuse their accumulator halves."""
    from piper_b200.ops import native

    torch.manual_seed(3)
    st = native.status_tensor()
    lib = native.lib()
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    at, bt = a.t().contiguous(), b.t().contiguous()          # [K, M], [K, N]
    ref = a.float() @ b.float().t()
    for a_op, a_mn in ((a, False), (at, True)):
        for b_op, b_mn in ((b, False), (bt, True)):
            c = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
            lib.gemm_tiled(a_op, b_op, c, a_mn, b_mn, False, st, 256)
            assert _close(c, ref, 1e-2), (a_mn, b_mn)
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    want = acc + ref
    lib.gemm_tiled(at, bt, acc, True, True, True, st, 256)
    assert _close(acc, want, 1e-2)
    c128 = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    c256 = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    lib.gemm_tiled(a, b, c128, False, False, False, st, 128)
    lib.gemm_tiled(a, b, c256, False, False, False, st, 256)
    torch.cuda.synchronize()
    native.check_status()
    assert torch.equal(c128, c256)      # same k order and fp32 accumulation: identical bits


def test_linear_op_autograd():
    from piper_b200 import ops

    torch.manual_seed(2)
    x = torch.randn(2, 256, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(768, 512, device="cuda", dtype=torch.bfloat16) * 0.05).requires_grad_(True)
    y = ops.linear(x, w)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = torch.nn.functional.linear(xr, wr)
    yr.backward(g.float())
    assert _close(y, yr, 1e-2)
    assert _close(x.grad, xr.grad, 1e-2)
    assert _close(w.grad, wr.grad, 1e-2)


@pytest.mark.parametrize("M,N,K,bf16_tile,f32_tile", [(2048, 4096, 4096, 256, 128), (4096, 5120, 64, 128, 128),
                                                      (1000, 8192, 72, 128, 128), (8192, 1000, 4104, 256, 256),
                                                      (4096, 4352, 72, 256, 128), (257, 256, 64, 128, 128)])
def test_gemm_tile_choice_does_not_change_the_result(M, N, K, bf16_tile, f32_tile):
    """Shapes on both sides of the tile rule (one round of big tiles against two with long and short contractions, three
    against five, two against four, ragged, tall and wide fp32, tiny): the chosen kernel gives the bits of either tile, in both output types."""
    from piper_b200.ops import native

    torch.manual_seed(19)
    lib, st = native.lib(), native.status_tensor()
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    for dtype, tile in ((torch.bfloat16, bf16_tile), (torch.float32, f32_tile)):
        assert lib.gemm_tile_rows(M, N, K, dtype == torch.float32, 148) == tile
        auto, small, big = (torch.empty(M, N, device="cuda", dtype=dtype) for _ in range(3))
        lib.gemm(a, b, auto, False, False, False, st)
        lib.gemm_tiled(a, b, small, False, False, False, st, 128)
        lib.gemm_tiled(a, b, big, False, False, False, st, 256)
        assert torch.equal(auto, small) and torch.equal(auto, big)


@pytest.mark.parametrize("M,N,K", [(1, 40, 24), (129, 72, 8), (256, 256, 64), (513, 1000, 1000), (2304, 4608, 192)])
@pytest.mark.parametrize("tile", [128, 256])
def test_gemm_shapes_give_the_same_bits(M, N, K, tile):
    """Every tile width by one CTA and by a pair, in every operand layout and both output types (K = 192 and less: two
    staging blocks per fp32 epilogue warp, K = 1000: one): less than a tile, remainders of rows (a pair whose second CTA
    has none), columns and k-blocks, more tiles than SMs.  fp32 sums of K bf16 products: 2^-8 covers the rounding of the
    bf16 result, and all shapes add in one order."""
    from piper_b200.ops import native

    torch.manual_seed(21)
    lib, st = native.lib(), native.status_tensor()
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    layouts = [(x, xm, y, ym) for x, xm in ((a, False), (a.t().contiguous(), True))
               for y, ym in ((b, False), (b.t().contiguous(), True)) if not xm or M % 8 == 0]
    ref = a.float() @ b.float().t()
    held = torch.randn(M, N, device="cuda")
    first = None
    for x, xm, y, ym in layouts:
        for width in range(32, 257, 32):
            outs = (torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16), torch.full((M, N + 8), 7.0, device="cuda"),
                    torch.nn.functional.pad(held, (0, 8), value=7.0))
            for out, add in zip(outs, (False, False, True)):
                lib.gemm_shaped(x, y, out[:, :N], xm, ym, add, st, tile, width)
                assert (out[:, N:] == 7).all()                 # nothing beyond the last column
            if first is None:
                first = outs
                assert _close(outs[0][:, :N], ref, 2 ** -8) and _close(outs[1][:, :N], ref, 1e-5)
                assert _close(outs[2][:, :N], ref + held, 1e-5)
            assert all(torch.equal(o, f) for o, f in zip(outs, first)), (xm, ym, width)


@pytest.mark.parametrize("M,N,K,tile,width,splits", [(1, 8, 1024, 128, 32, 16), (100, 264, 5000, 128, 64, 7),
                                                     (129, 1000, 4096, 128, 256, 3), (300, 520, 6016, 256, 96, 5),
                                                     (513, 2056, 2112, 256, 256, 33), (1500, 256, 32000, 0, 0, 0),
                                                     (33, 72, 20000, 0, 0, 0)])
def test_gemm_split_contraction(M, N, K, tile, width, splits):
    """Parts of equal and of unequal length, a k-block each, ragged rows and columns, and the shapes that the rule splits by
    itself: against fp64, the same bits every time, and no further from it than the product in one part."""
    from piper_b200.ops import native

    lib, st = native.lib(), native.status_tensor()
    torch.manual_seed(33)
    for a_mn in (False, True):
        a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
        b = torch.randn(K, (N + 7) // 8 * 8, device="cuda").to(torch.bfloat16)[:, :N]
        if a_mn:
            at = torch.zeros(K, (M + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)
            at[:, :M] = a.t()
            x = at[:, :M]
        else:
            x = torch.zeros(M, (K + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :K]
            x.copy_(a)
        want = a.double() @ b.double()
        outs = [torch.full((M + 1, (N + 7) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
        for out in outs[:2]:
            if splits:
                lib.gemm_split(x, b, out[:M, :N], a_mn, True, st, tile, width, splits)
            else:
                assert lib.gemm_split_shape(M, N, K, True, False, 148)[2] > 1
                lib.gemm(x, b, out[:M, :N], a_mn, True, False, st)
        lib.gemm_shaped(x, b, outs[2][:M, :N], a_mn, True, False, st, 0, 0)
        assert torch.equal(outs[0], outs[1])
        assert (outs[0][M:] == 7).all() and (outs[0][:, N:] == 7).all()      # nothing beside the product
        err = [((o[:M, :N].double() - want).norm() / want.norm()).item() for o in outs]
        # one rounding to bf16 (rms 2^-9 / sqrt(3) at most); the sums in fp32 add far less
        assert err[0] < 2 ** -9 and err[0] <= err[2] * 1.01
        assert _close(outs[0][:M, :N], want, 2 ** -8)
    native.check_status()


def test_gemm_split_contraction_in_a_captured_graph_and_on_two_streams():
    """The sums' scratch belongs to the stream that runs the product: products of two streams at once, and a graph's, replayed on
    other inputs beside products that take scratch of their own."""
    from piper_b200.ops import native

    lib, status = native.lib(), native.status_tensor()
    torch.manual_seed(34)
    M, N, K = 100, 512, 20000
    assert lib.gemm_split_shape(M, N, K, True, False, 148)[2] > 1
    rn = lambda *shape: torch.randn(*shape, device="cuda").to(torch.bfloat16)
    xs, b = [rn(M, K) for _ in range(6)], rn(K, N)

    def product(x):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        lib.gemm(x, b, out, False, True, False, status)
        return out

    want = [product(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        got = [[], []]
        for x in xs:
            for stream, outs in zip(streams, got):
                with torch.cuda.stream(stream):
                    outs.append(product(x))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for outs in got for a, b in zip(outs, want))
    x = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        first, second = product(x), product(x)
    for i in (3, 1, 5):
        x.copy_(xs[i])
        graph.replay()
        other = product(xs[i - 1])
        assert torch.equal(first, want[i]) and torch.equal(second, want[i]) and torch.equal(other, want[i - 1])
    native.check_status()


@pytest.mark.parametrize("sizes,forked", [((4095,), []), ((4096,), [4096]), ((4096, 4095), [4096, 4095]),
                                          ((4095, 4096), [4096])])
def test_linear_gradients_around_the_fork_threshold(sizes, forked, monkeypatch):
    """2048 x 1024 weights: 4096 rows are the first size whose weight-gradient GEMM runs on the side stream.  Two uses of
    one weight in one scope add to its bucket in the order of their backward passes (a small one behind a forked one is
    forked too), so every repetition gives the same bits."""
    from piper_b200 import ops
    from piper_b200.ops import core

    assert core._GEMM_FORK == 2 and 4096 * 2048 * 1024 == core._FORK_MIN_MACS
    torch.manual_seed(20)
    w = (torch.randn(2048, 1024, device="cuda", dtype=torch.bfloat16) * 0.05).requires_grad_(True)
    xs = [torch.randn(T, 1024, device="cuda", dtype=torch.bfloat16, requires_grad=True) for T in sizes]
    gs = [torch.randn(T, 2048, device="cuda", dtype=torch.bfloat16) for T in sizes]
    seen, rows = [], []
    side_stream = core._side_stream
    monkeypatch.setattr(core, "_side_stream", lambda cur: (seen.append(rows[-1]), side_stream(cur))[1])

    def backward():
        seen.clear()
        for x, g in zip(xs, gs):
            x.grad = None
            rows.append(x.shape[0])
            ops.linear(x, w).backward(g)

    want = sum(g.float().t() @ x.detach().float() for x, g in zip(xs, gs))
    backward()                                                # no bucket: every fork is joined, no order to keep
    assert seen == [T for T in sizes if T == 4096]
    for x, g in zip(xs, gs):
        assert _close(x.grad, g.float() @ w.detach().float(), 1e-2)
    assert _close(w.grad, want, 1e-2)
    held = torch.randn(2048, 1024, device="cuda")            # what the bucket holds already: the order shows in the bits
    sink = torch.empty_like(held)
    core.grad_sinks.register(w, sink)
    try:
        results = []
        for _ in range(5):
            sink.copy_(held)
            with core.deferred_join():
                backward()
                assert seen == forked
            results.append(sink.clone())
        assert not core.deferred_join.buckets and not core.deferred_join.pending
    finally:
        core.grad_sinks.unregister(w)
    assert _close(results[0], want + held, 1e-4) and all(torch.equal(r, results[0]) for r in results)


@pytest.mark.parametrize("T,D", [(1, 2048), (591, 4096), (593, 2048), (593, 8192), (1777, 2048), (297, 8192)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_rows_per_cta(T, D, residual):
    """One CTA per row up to 592 rows (296 of 8192 elements), several rows per CTA behind: every row against fp32, rounded to bf16 once (2^-8), the
    residual sum exactly."""
    from piper_b200.ops import core

    torch.manual_seed(23)
    x, r = (torch.randn(T, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    w = torch.randn(D, device="cuda").to(torch.bfloat16)
    y, h, rstd = core.add_rmsnorm_fwd(x, r, w, 1e-6) if residual else (core.rmsnorm_fwd(x, w, 1e-6)[0], x,
                                                                       core.rmsnorm_fwd(x, w, 1e-6)[1])
    want_h = (x.float() + r.float()).to(torch.bfloat16) if residual else x
    assert torch.equal(h, want_h)
    want_r = torch.rsqrt(want_h.double().pow(2).mean(-1) + 1e-6)
    assert torch.allclose(rstd.double(), want_r, rtol=1e-5)
    want = want_h.double() * want_r.unsqueeze(-1) * w.double()
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("T,Hq,Hkv,hd,norm", [(128, 2, 2, 64, False), (1024, 17, 2, 128, False), (4096, 30, 5, 128, False),
                                              (256, 5, 1, 64, True), (1024, 16, 4, 128, True), (4096, 33, 4, 128, True)])
def test_qk_rope_heads_per_group(T, Hq, Hkv, hd, norm):
    """One, two, four and eight heads per lane group in both directions, with head counts that leave a shorter last group,
    against the fp32 reference; bf16 rounding of results, fp32 sums for the weights."""
    from piper_b200.ops import core

    torch.manual_seed(24)
    cos, sin = core.rope_tables(hd, T, 1e4, device="cuda")
    x = torch.randn(T, (Hq + 2 * Hkv) * hd, device="cuda").to(torch.bfloat16).requires_grad_(True)
    ws = [torch.randn(hd, device="cuda").to(torch.bfloat16).requires_grad_(True) for _ in range(2)] if norm else [None, None]
    out = core.qk_rope(x, cos, sin, *ws, T, Hq, Hkv, hd, False, 1e-6)
    g = torch.randn_like(out)
    out.backward(g)
    leaves = [t.detach().float().requires_grad_(True) for t in (x, *ws) if t is not None]
    ref = core._qk_rope_ref(leaves[0], cos, sin, *(leaves[1:] if norm else (None, None)), T, Hq, Hkv, hd, False, 1e-6)
    ref.backward(g.float())
    assert _close(out, ref, 2 ** -8) and _close(x.grad, leaves[0].grad, 2 ** -8)
    for w, l in zip(ws, leaves[1:]):
        assert _close(w.grad, l.grad, 2 ** -8)


@pytest.mark.parametrize("T,Hq,Hkv,hd,norms,inter", [(1, 1, 1, 64, "qk", True), (1, 1, 1, 128, "", False), (3, 7, 1, 64, "k", False),
                                                     (515, 9, 3, 64, "q", True), (2500, 21, 5, 128, "q", True),
                                                     (2500, 21, 5, 128, "k", False), (6001, 9, 3, 64, "qk", True),
                                                     (6001, 9, 3, 64, "", True)])
def test_qk_rope_tasks(T, Hq, Hkv, hd, norms, inter):
    """Fewer tasks than warps and several per warp, head counts that leave lane groups of a warp without a head, norms of
    one kind of heads only, positions that repeat; against the fp32 reference, bf16 rounding of results."""
    from piper_b200.ops import core

    torch.manual_seed(25)
    S = max(1, T // 2)
    cos, sin = core.rope_tables(hd, S, 1e4, device="cuda")
    x = torch.randn(T, (Hq + 2 * Hkv) * hd, device="cuda").to(torch.bfloat16).requires_grad_(True)
    ws = [torch.randn(hd, device="cuda").to(torch.bfloat16).requires_grad_(True) if c in norms else None for c in "qk"]
    out = core.qk_rope(x, cos, sin, *ws, S, Hq, Hkv, hd, inter, 1e-6)
    g = torch.randn_like(out)
    out.backward(g)
    xr, *wr = [None if t is None else t.detach().float().requires_grad_(True) for t in (x, *ws)]
    ref = core._qk_rope_ref(xr, cos, sin, *wr, S, Hq, Hkv, hd, inter, 1e-6)
    ref.backward(g.float())
    assert _close(out, ref, 2 ** -8) and _close(x.grad, xr.grad, 2 ** -8)
    assert torch.equal(out[:, (Hq + Hkv) * hd:], x[:, (Hq + Hkv) * hd:]) and torch.equal(x.grad[:, (Hq + Hkv) * hd:], g[:, (Hq + Hkv) * hd:])
    for w, l in zip(ws, wr):
        assert w is None or _close(w.grad, l.grad, 2 ** -8)


@pytest.mark.parametrize("T,D", [(300, 256), (300, 2048), (1000, 4096), (300, 8192), (7, 4096)])
def test_rmsnorm_and_residual(T, D):
    from piper_b200 import ops

    torch.manual_seed(3)
    x = torch.randn(T, D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(T, D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y, h = ops.add_rmsnorm(x, r, w, 1e-6)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    torch.autograd.backward([y, h], [gy, gh])
    xr, rr, wr = (t.detach().float().requires_grad_(True) for t in (x, r, w))
    hr = (xr + rr).to(torch.bfloat16).float() + 0 * (xr + rr)
    hr = xr + rr
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    torch.autograd.backward([yr, hr], [gy.float(), gh.float()])
    assert _close(y, yr, 1e-2) and _close(h, hr, 1e-2)
    assert _close(x.grad, xr.grad, 2e-2) and _close(r.grad, rr.grad, 2e-2)
    assert _close(w.grad, wr.grad, 2e-2)
    y2 = ops.rmsnorm(x.detach(), w.detach(), 1e-6)
    x0 = x.detach().float()
    assert _close(y2, x0 * torch.rsqrt(x0.pow(2).mean(-1, keepdim=True) + 1e-6) * w.detach().float(), 1e-2)


@pytest.mark.parametrize("T", [1, 5, 299, 1801])
@pytest.mark.parametrize("D", [8, 256, 512, 768, 1024, 1280, 1536, 1792, 2048, 2304, 2560, 3072, 3584, 4608, 5120, 6144, 7168, 8200])
def test_rmsnorm_widths(T, D):
    """Every number of threads and vectors per row, widths beside them for the general kernels, fewer rows than CTAs and
    several per CTA; against fp64 with the residual rounded as the op rounds it."""
    from piper_b200 import ops

    torch.manual_seed(35)
    x, r, gy, gh = (torch.randn(T, D, device="cuda").to(torch.bfloat16) for _ in range(4))
    w = torch.randn(D, device="cuda").to(torch.bfloat16).requires_grad_(True)
    x.requires_grad_(True)
    y, h = ops.add_rmsnorm(x, r, w, 1e-6)
    dx, dw = torch.autograd.grad([y, h], [x, w], [gy, gh])
    assert torch.equal(h, (x.float() + r.float()).to(torch.bfloat16))
    h64, w64 = h.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    y64 = h64 * torch.rsqrt(h64.pow(2).mean(-1, keepdim=True) + 1e-6) * w64
    dx64, dw64 = torch.autograd.grad(y64, [h64, w64], gy.double())
    dx64 = dx64 + gh.double()
    # one rounding to bf16 each; sums in fp32
    assert ((y.double() - y64).abs() <= 2 ** -8 * y64.abs() + 1e-6).all()
    assert ((dx.double() - dx64).abs() <= 2 ** -8 * dx64.abs() + 1e-4).all()
    assert ((dw.double() - dw64).abs() <= 2 ** -8 * dw64.abs() + 1e-5 * max(1, T) ** 0.5 * 4).all()
    plain = ops.rmsnorm(h.detach(), w.detach(), 1e-6)
    assert torch.equal(plain, y)


@pytest.mark.parametrize("hd,inter,qknorm,seqs", [(128, True, False, 2), (128, False, True, 2), (64, False, False, 2),
                                                  (64, True, True, 2), (128, False, True, 640), (64, True, True, 1200)])
def test_qk_rope(hd, inter, qknorm, seqs):
    """The large cases use 12 heads (two head chunks per token, the second one partial) and more tokens than one
    pass of the grid covers."""
    from piper_b200 import ops
    from piper_b200.ops.core import _qk_rope_ref

    torch.manual_seed(4)
    S, Hq, Hkv = (64, 4, 2) if seqs == 2 else (64, 8, 2)
    cos, sin = ops.rope_tables(hd, S, 10000.0, device="cuda")
    qkv = torch.randn(seqs * S, (Hq + 2 * Hkv) * hd, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    qw = torch.randn(hd, device="cuda", dtype=torch.bfloat16, requires_grad=True) if qknorm else None
    kw = torch.randn(hd, device="cuda", dtype=torch.bfloat16, requires_grad=True) if qknorm else None
    out = ops.qk_rope(qkv, cos, sin, qw, kw, S, Hq, Hkv, hd, inter, 1e-6)
    g = torch.randn_like(out)
    out.backward(g)
    q2 = qkv.detach().float().requires_grad_(True)
    qw2 = qw.detach().float().requires_grad_(True) if qknorm else None
    kw2 = kw.detach().float().requires_grad_(True) if qknorm else None
    ref = _qk_rope_ref(q2, cos, sin, qw2, kw2, S, Hq, Hkv, hd, inter, 1e-6)
    ref.backward(g.float())
    assert _close(out, ref, 1e-2)
    assert _close(qkv.grad, q2.grad, 2e-2)
    if qknorm:
        assert _close(qw.grad, qw2.grad, 3e-2) and _close(kw.grad, kw2.grad, 3e-2)


@pytest.mark.parametrize("B,S,Hq,Hkv,hd", [(1, 128, 2, 1, 128), (2, 256, 4, 2, 128), (1, 512, 4, 4, 64), (1, 1024, 8, 2, 128),
                                           (1, 4096, 32, 8, 128)])
def test_attention_fwd_bwd(B, S, Hq, Hkv, hd):
    from piper_b200 import ops
    from piper_b200.ops.core import _attention_ref

    torch.manual_seed(5)
    qkv = (torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda", dtype=torch.bfloat16)).requires_grad_(True)
    out = ops.attention(qkv, B, S, Hq, Hkv, hd)
    g = torch.randn_like(out)
    out.backward(g)
    q2 = qkv.detach().float().requires_grad_(True)
    ref, _ = _attention_ref(q2, B, S, Hq, Hkv, hd, 1.0 / math.sqrt(hd))
    ref.backward(g.float())
    assert _close(out, ref, 2e-2)
    W = (Hq + 2 * Hkv) * hd
    gq, gr = qkv.grad.view(-1, W), q2.grad.view(-1, W)
    assert _close(gq[:, : Hq * hd], gr[:, : Hq * hd], 3e-2)          # dQ
    assert _close(gq[:, Hq * hd: (Hq + Hkv) * hd], gr[:, Hq * hd: (Hq + Hkv) * hd], 3e-2)   # dK
    assert _close(gq[:, (Hq + Hkv) * hd:], gr[:, (Hq + Hkv) * hd:], 3e-2)   # dV


@pytest.mark.parametrize("B,S,Hq,Hkv,hd,growth,tiles", [(1, 640, 40, 40, 64, 0.0, 2), (2, 640, 24, 8, 128, 0.0, 2),
                                                        (1, 768, 40, 8, 128, 40.0, 2), (3, 256, 32, 4, 64, 40.0, 2),
                                                        (1, 640, 32, 32, 64, 0.0, 1), (1, 768, 32, 8, 128, 40.0, 1)])
def test_attention_paired_tiles(B, S, Hq, Hkv, hd, growth, tiles):
    """More query tiles than SMs, so a CTA takes two (one where the longest tile covers the rest): odd tile counts per
    head (a last CTA with one tile), pairs of heads and pairs of neighbouring query blocks.  ``growth`` makes later keys' scores larger, so the accumulated output
    is rescaled by small factors in most blocks."""
    from piper_b200 import ops
    from piper_b200.ops import native
    from piper_b200.ops.core import _attention_ref

    assert native.lib().attn_tiles_per_cta(B, S, Hq, 148) == tiles
    torch.manual_seed(15)
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda")
    ramp = 1.0 + growth * (torch.arange(B * S, device="cuda") % S) / S
    qkv[:, Hq * hd: (Hq + Hkv) * hd] *= ramp.unsqueeze(1)
    qkv = qkv.to(torch.bfloat16).requires_grad_(True)
    out = ops.attention(qkv, B, S, Hq, Hkv, hd)
    g = torch.randn_like(out)
    out.backward(g)
    q2 = qkv.detach().float().requires_grad_(True)
    ref, _ = _attention_ref(q2, B, S, Hq, Hkv, hd, 1.0 / math.sqrt(hd))
    ref.backward(g.float())
    assert _close(out, ref, 2e-2)
    nq, nk = Hq * hd, Hkv * hd
    for lo, hi in ((0, nq), (nq, nq + nk), (nq + nk, nq + 2 * nk)):
        assert _close(qkv.grad[:, lo:hi], q2.grad[:, lo:hi], 3e-2), (lo, hi)


@pytest.mark.parametrize("B,S,Hq,Hkv,hd,parts", [(1, 640, 8, 2, 64, 4), (1, 1024, 8, 4, 128, 2), (1, 512, 16, 2, 128, 4),
                                                 (1, 1024, 16, 2, 64, 8), (2, 1280, 8, 1, 128, 8), (1, 384, 12, 2, 128, 2)])
def test_attention_backward_splits_a_group(B, S, Hq, Hkv, hd, parts):
    """dK and dV of a key block by several CTAs: against an fp32 reference and, up to the order of the fp32 sums and one
    bf16 rounding, against the launch without scratch, where one CTA adds all heads; the same bits every time."""
    from piper_b200.ops import native
    from piper_b200.ops.core import _attention_ref, attention_fwd

    lib, st = native.lib(), native.status_tensor()
    assert lib.attn_bwd_parts(B, S, Hq, Hkv, 148) == parts
    torch.manual_seed(22)
    scale = 1.0 / math.sqrt(hd)
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda").to(torch.bfloat16)
    g = torch.randn(B * S, Hq * hd, device="cuda").to(torch.bfloat16)
    out, lse = attention_fwd(qkv, B, S, Hq, Hkv, hd, scale)
    grads = []
    for floats in (lib.attn_bwd_floats(B, S, Hq, Hkv, hd), lib.attn_bwd_floats(B, S, Hq, Hkv, hd), B * Hq * S):
        delta = torch.full((floats,), float("nan"), device="cuda")
        grads.append(torch.empty_like(qkv))
        lib.attn_bwd(qkv, out, g, lse, delta, grads[-1], B, S, Hq, Hkv, hd, scale, st)
    assert torch.equal(grads[0], grads[1])
    assert _close(grads[0], grads[2], 2 ** -8) and torch.equal(grads[0][:, : Hq * hd], grads[2][:, : Hq * hd])
    q2 = qkv.float().requires_grad_(True)
    ref, _ = _attention_ref(q2, B, S, Hq, Hkv, hd, scale)
    ref.backward(g.float())
    nq, nk = Hq * hd, Hkv * hd
    for lo, hi in ((0, nq), (nq, nq + nk), (nq + nk, nq + 2 * nk)):
        assert _close(grads[0][:, lo:hi], q2.grad[:, lo:hi], 3e-2), (lo, hi)


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_largest_probability_is_exact(hd):
    """One key of the second block beats every earlier one by 2^0.1 to 2^7.9 and alone has a value, so a row is v / l.
    With the row's own maximum its probability is 1 and only l's fp32 sums (1e-6) and the output's rounding to bf16 are
    left: one element in 2,000 at most falls on the other side.  A probability that is itself rounded to bf16 moves
    the result by up to 2^-9, half of its last place."""
    from piper_b200.ops import core

    S, Hq = 256, 4
    torch.manual_seed(16)
    g = torch.linspace(0.1, 7.9, 128 * Hq)[torch.randperm(128 * Hq)].view(128, Hq) * math.log(2.0) * math.sqrt(hd)
    q, k, v = torch.zeros(S, Hq, hd), torch.zeros(S, hd), torch.zeros(S, hd)
    q[128:, :, 0] = g
    k[128, 0] = 1.0
    v[128] = torch.randn(hd)
    qkv = torch.cat([q.reshape(S, Hq * hd), k, v], dim=1).to(torch.bfloat16).cuda()
    out, lse = core.attention_fwd(qkv, 1, S, Hq, 1, hd, 1.0 / math.sqrt(hd))
    s = qkv[128:, : Hq * hd].view(128, Hq, hd)[:, :, 0].double() / math.sqrt(hd)
    others = torch.arange(128, 256, device="cuda", dtype=torch.float64).view(128, 1)     # earlier keys have score 0
    l = 1.0 + others * torch.exp(-s)
    want = (qkv[128, (Hq + 1) * hd:].double() / l.unsqueeze(-1)).to(torch.bfloat16)
    assert (out[128:].view(128, Hq, hd) != want).float().mean() < 0.01
    assert torch.allclose(lse[0, :, 128:].t().double(), s + torch.log(l), rtol=1e-5)


@pytest.mark.parametrize("T,V,D,launches", [(64, 1000, 264, 1), (300, 301, 256, 1), (0, 16, 64, 1), (77, 40, 256, 1),
                                            (96, 16480, 512, 3), (97, 16480, 512, 1), (3001, 35003, 264, 3),
                                            (0, 131072, 64, 3)])
def test_embedding_gradient(T, V, D, launches):
    """Compact accumulation into a bf16 table and the fp32 table (small tables, T >= V), on both sides of the line between
    them; many repeated tokens, some outside the table."""
    from piper_b200 import ops
    from piper_b200.ops import native

    torch.manual_seed(17)
    table = torch.randn(V, D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    tok = torch.randint(0, max(1, V // 4), (T,), device="cuda")
    tok[1::3] = tok[0] if T else 0
    out = ops.embedding(tok, table)
    g = torch.randn_like(out)
    before = native.lib().kernel_launch_count()
    out.backward(g)
    assert native.lib().kernel_launch_count() - before == launches
    ref = torch.zeros(V, D, device="cuda").index_add_(0, tok, g.float())
    assert table.grad.dtype == torch.bfloat16
    # one rounding of an fp32 sum of up to a third of the tokens in another order
    assert torch.allclose(table.grad.float(), ref, rtol=2 ** -8, atol=1e-5 * max(1, T / 100))
    if launches == 3 and T:
        bad = tok.clone()
        bad[2], bad[3] = -1, V                    # rejected by the forward pass; the backward pass leaves them out
        scratch = torch.full(((V + 3) // 4 * 4 + T * D,), 7, dtype=torch.int32, device="cuda")
        d_table = torch.full_like(table, 7.0)
        native.lib().embedding_bwd_bf16(bad, g, scratch, d_table)
        keep = torch.ones(T, dtype=torch.bool, device="cuda")
        keep[2:4] = False
        ref = torch.zeros(V, D, device="cuda").index_add_(0, tok[keep], g[keep].float())
        assert torch.allclose(d_table.float(), ref, rtol=2 ** -8, atol=1e-5 * max(1, T / 100))


@pytest.mark.parametrize("T,F", [(9000, 776), (5000, 14336)])
def test_swiglu_grid_stride_walk(T, F):
    """More vectors than the grid has threads, with a row length that the grid stride does not divide."""
    from piper_b200 import ops

    torch.manual_seed(16)
    h = torch.randn(T, 2 * F, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    a = ops.swiglu(h)
    g = torch.randn_like(a)
    a.backward(g)
    hr = h.detach().float().requires_grad_(True)
    ar = torch.nn.functional.silu(hr[:, :F]) * hr[:, F:]
    ar.backward(g.float())
    assert _close(a, ar, 1e-2) and _close(h.grad, hr.grad, 1e-2)


def test_swiglu_large_gates():
    """Gates of every magnitude: exp(-g) underflows on one side and overflows on the other."""
    from piper_b200 import ops

    g = torch.cat([torch.linspace(-120, 120, 4088, device="cuda"),
                   torch.tensor([0.0, -0.0, 1e4, -1e4, 1e38, -1e38, float("inf"), float("nan")], device="cuda")])
    u = torch.where(torch.arange(4096, device="cuda") % 2 == 0, 1.5, -0.75)
    h = torch.cat([g, u])[None].bfloat16().requires_grad_(True)
    a = ops.swiglu(h)
    a.backward(torch.ones_like(a))
    h64 = h.detach().double().requires_grad_(True)
    a64 = torch.nn.functional.silu(h64[:, :4096]) * h64[:, 4096:]
    a64.backward(torch.ones_like(a64))
    # one rounding to bf16; exp of an argument of magnitude 88 is good to 2^-17; where exp(-g) overflows the result is zero
    # for at most 1.5 x 90 x 2^-128.  The gate's gradient is u s (1 + g (1 - s)), whose two terms cancel to their fp32
    # rounding near g = -1.28.
    fin = slice(0, 4094)
    assert torch.allclose(a.double()[:, fin], a64[:, fin], rtol=2 ** -8, atol=4e-37)
    assert torch.allclose(h.grad.double()[:, fin], h64.grad[:, fin], rtol=2 ** -8, atol=1e-6)
    assert torch.allclose(h.grad.double()[:, 4096:][:, fin], h64.grad[:, 4096:][:, fin], rtol=2 ** -8, atol=4e-37)
    assert a[0, 4094] == float("inf") or a[0, 4094] == float("-inf")
    assert a[0, 4095].isnan() and h.grad[0, 4095].isnan() and h.grad[0, 8191].isnan()


_SWIGLU_BY_DIVISION = """
extern "C" __global__ void swiglu_by_division(const float* g, const float* u, const float* d, float* a, float* dg, float* du,
                                              long long n) {
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= n) return;
  a[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
  const float s = 1.f / (1.f + __expf(-g[i]));
  du[i] = d[i] * (g[i] * s);
  dg[i] = d[i] * u[i] * s * (1.f + g[i] * (1.f - s));
}
"""


@pytest.mark.parametrize("backward", [False, True])
def test_swiglu_has_the_bits_of_a_division(backward):
    """Every bf16 gate with every up value (forward) or every upstream gradient (backward): the kernels, which do not divide,
    against one that does, with the same exponential.  A sigmoid one unit in the last place of fp32 off shows in about one of
    2^15 products, so nothing less than all of them pins it."""
    from piper_b200 import ops

    divided = torch.cuda._compile_kernel(_SWIGLU_BY_DIVISION, "swiglu_by_division")
    torch.manual_seed(43)
    every = torch.arange(-32768, 32768, device="cuda").to(torch.int16).view(torch.bfloat16)
    rows, F = 64, every.numel()
    g = every.expand(rows, F)
    gf = g.float().contiguous()
    bad = torch.zeros(3, dtype=torch.int64, device="cuda")
    for values in every.split(rows):
        u, up = values[:, None], torch.randn(rows, 1, device="cuda").bfloat16()
        if backward:
            u, up = up, u
        u, up = u.expand(rows, F).contiguous(), up.expand(rows, F).contiguous()
        h = torch.cat([g, u], 1).requires_grad_(backward)
        act = ops.swiglu(h)
        got = [act.detach()]
        if backward:
            (dh,) = torch.autograd.grad(act, h, up)
            got += [dh[:, :F].contiguous(), dh[:, F:].contiguous()]
        want = [torch.empty(rows, F, device="cuda") for _ in range(3)]
        divided(grid=(rows * F // 256, 1, 1), block=(256, 1, 1), args=[gf, u.float(), up.float(), *want, rows * F])
        for i, (x, y) in enumerate(zip(got, want)):
            y = y.bfloat16()
            bad[i] += ((x.view(torch.int16) != y.view(torch.int16)) & ~(x.isnan() & y.isnan())).sum()
    assert bad.tolist() == [0, 0, 0]


@pytest.mark.parametrize("T,D,F", [(128, 256, 512), (384, 512, 1536), (2048, 1024, 2048)])
def test_overlapped_launches_keep_their_order(T, D, F):
    """A kernel may start while the one before it runs, but reads what that one leaves: every op behind one that has just
    written its input, weights that the optimizer kernel and a tensor op have just changed, a buffer that the allocator
    hands on at once, the same with the device idle between any two ops, and in a captured graph."""
    from piper_b200 import ops
    from piper_b200.ops import moe, native

    torch.manual_seed(37)
    rn = lambda *shape: torch.randn(*shape, device="cuda").to(torch.bfloat16)
    x, r, w13, w2, wn = rn(T, D), rn(T, D), rn(2 * F, D) * D ** -0.5, rn(D, F) * F ** -0.5, rn(D)
    wqkv, labels = rn(3 * D, D) * D ** -0.5, torch.randint(0, D, (T,), device="cuda")
    we, logits = rn(8, D, D) * D ** -0.5, rn(T, 8)
    cos, sin = ops.rope_tables(64, 128, 1e4, device="cuda")
    up = rn(T, D)
    state = [torch.randn(w2.numel(), device="cuda") for _ in range(4)]

    def chain(idle):
        step = torch.cuda.synchronize if idle else lambda: None
        w = w2.clone()
        master, m, v, g = (t.clone() for t in state)
        v.abs_()
        step(); native.lib().adam_flat(master, m, v, g, w.view(-1), 1e-3, 0.9, 0.95, 1e-8, 0.0, 1, 1.0, True)
        leaves = [t.clone().requires_grad_(True) for t in (x, w13, w, wn, wqkv, we, logits)]
        xl, a13, a2, an, aq, ae, lg = leaves
        with torch.no_grad():
            step(); an.mul_(1.5)
        step(); y, h = ops.add_rmsnorm(xl, r, an, 1e-6)
        step(); qkv = ops.linear(y, aq)
        step(); qkv = ops.qk_rope(qkv, cos, sin, None, None, 128, D // 64, D // 64, 64, True, 1e-6)
        step(); o = ops.attention(qkv, T // 128, 128, D // 64, D // 64, 64)
        step(); f = ops.linear(o, a13)
        step(); f = ops.linear(ops.swiglu(f), a2)
        step(); y, h = ops.add_rmsnorm(f, h, an, 1e-6)
        step(); wts, idx, counts = moe.moe_route(lg, 1, True)
        step(); rows, pos, gs, gl, ec = moe.moe_dispatch(y, idx, counts)
        step(); e = moe.grouped_linear(rows, ae, *moe.moe_group_table(ec, ae))
        step(); out = moe.moe_combine(e, pos, wts, gs, gl, counts) + h
        step(); loss = ops.cross_entropy(out, labels)
        step(); grads = torch.autograd.grad(loss, leaves)
        return [loss.detach(), *grads]

    want = chain(True)
    for _ in range(20):
        # rows of one expert come in the order of their arrival, and so do the sums of its weight's gradient
        for i, (a, b) in enumerate(zip(chain(False), want)):
            assert torch.equal(a, b) if i != 6 else _close(a, b, 2 ** -8), i
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = chain(False)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for i, (a, b) in enumerate(zip(captured, want)):
        assert torch.equal(a, b) if i != 6 else _close(a, b, 2 ** -8), i
    native.check_status()


def test_overlapped_launches_behind_another_stream():
    """A kernel launched to overlap the one before it in its stream also waits for what the stream waits for: products and passes
    handed from one stream to another and back through buffers that hold the step before, with the device idle between any two,
    without, and in a captured graph."""
    from piper_b200.ops import native

    lib, status = native.lib(), native.status_tensor()
    torch.manual_seed(44)
    T, D, F, steps = 2048, 2048, 4096, 8
    rn = lambda *shape: torch.randn(*shape, device="cuda").to(torch.bfloat16)
    x, w13, w2 = rn(steps, T, D), rn(2 * F, D) * D ** -0.5, rn(D, F) * F ** -0.5
    h, act, y, g, z = rn(T, 2 * F), rn(T, F), rn(T, D), rn(T, D), rn(T, D)
    side = torch.cuda.Stream()

    def run(idle):
        step = torch.cuda.synchronize if idle else lambda: None
        cur, out = torch.cuda.current_stream(), torch.zeros_like(x)
        for i in range(steps):
            step(); lib.gemm(x[i], w13, h, False, False, False, status)
            step(); lib.swiglu_fwd(h, act)
            side.wait_stream(cur)
            with torch.cuda.stream(side):
                step(); lib.gemm(act, w2, y, False, False, False, status)
                step(); lib.add_bf16(y, x[i], g)
            step(); lib.add_bf16(x[i], x[i - 1], z)
            cur.wait_stream(side)
            step(); lib.add_bf16(g, z, out[i])
        return out

    want = run(True)
    torch.cuda.synchronize()
    for _ in range(20):
        assert torch.equal(run(False), want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run(False)
    for _ in range(3):
        captured.zero_()
        graph.replay()
        assert torch.equal(captured, want)
    native.check_status()


@pytest.mark.parametrize("sinks", [False, True])
def test_overlapped_launches_of_forked_gradients(sinks, monkeypatch):
    """Layers whose weight gradients run on a second stream, joined layer by layer or, for buckets, at the end of the scope: the
    gradients of the same layers on one stream."""
    from piper_b200 import ops
    from piper_b200.ops import core, native

    torch.manual_seed(45)
    T, D, F = 2048, 2048, 4096
    rn = lambda *shape: torch.randn(*shape, device="cuda").to(torch.bfloat16)
    x, up = rn(T, D), rn(T, D)
    ws = [rn(2 * F, D) * D ** -0.5, rn(D, F) * F ** -0.5, rn(2 * F, D) * D ** -0.5, rn(D, F) * F ** -0.5]
    assert all(T * w.numel() >= core._FORK_MIN_MACS for w in ws)
    for t in (x, *ws):
        t.requires_grad_(True)
    buckets = [torch.zeros(w.shape, device="cuda") for w in ws]

    def run():
        for b in buckets:
            b.zero_()
        with core.deferred_join():
            f = x
            for a, b in ((ws[0], ws[1]), (ws[2], ws[3])):
                f = ops.linear(ops.swiglu(ops.linear(f, a)), b)
            grads = torch.autograd.grad(f, [x, *ws], up, allow_unused=sinks)
        return [grads[0], *([b.clone() for b in buckets] if sinks else grads[1:])]

    if sinks:
        for w, b in zip(ws, buckets):
            ops.grad_sinks.register(w, b)
    try:
        with monkeypatch.context() as m:
            m.setattr(core, "_GEMM_FORK", 0)
            want = run()
        for _ in range(10):
            assert all(torch.equal(a, b) for a, b in zip(run(), want))
    finally:
        for w in ws:
            ops.grad_sinks.unregister(w)
    native.check_status()


@pytest.mark.parametrize("B,S,Hq,Hkv,hd", [(1, 128, 2, 1, 64), (2, 256, 2, 2, 128), (1, 384, 3, 1, 64), (1, 640, 2, 2, 128),
                                           (1, 1408, 4, 1, 64), (1, 2048, 8, 2, 128), (1, 2048, 16, 4, 64)])
def test_attention_halves_of_key_blocks(B, S, Hq, Hkv, hd):
    """One query tile per CTA, with no, one and several key blocks in its second half, an odd number of blocks, and more tiles
    than SMs: output, log-sum-exp and gradients against fp64.  Large scores in single key blocks make the halves' maxima
    differ by more than exp2 can hold in 16 bits."""
    from piper_b200.ops import core, native

    assert native.lib().attn_tiles_per_cta(B, S, Hq, 148) == 1
    torch.manual_seed(39)
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda")
    qkv.view(B, S, -1)[:, 128:256, Hq * hd:(Hq + Hkv) * hd] *= 12          # keys of the second block
    qkv = qkv.to(torch.bfloat16).requires_grad_(True)
    out, lse = core.attention_fwd(qkv, B, S, Hq, Hkv, hd, hd ** -0.5)
    g = torch.randn_like(out)
    (dqkv,) = torch.autograd.grad(out, qkv, g)
    x = qkv.detach().double().requires_grad_(True)
    q, k, v = (t.transpose(1, 2) for t in x.view(B, S, Hq + 2 * Hkv, hd).split([Hq, Hkv, Hkv], 2))
    k, v = (t.repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    scores = (q @ k.transpose(2, 3) * hd ** -0.5).masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = (torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(B * S, Hq * hd)
    (dref,) = torch.autograd.grad(ref, x, g.double())
    # probabilities are rounded to bf16 (2^-9 of a weighted mean of v), results once more; scores are fp32 sums
    assert _close(out, ref, 2 ** -7) and _close(dqkv, dref, 2 ** -6)
    assert ((out.double() - ref).norm() / ref.norm()) < 4e-3
    want = torch.logsumexp(scores, -1)
    assert ((lse.double() - want).abs() <= 1e-5 * want.abs().clamp(min=1)).all()


@pytest.mark.parametrize("S,Hq,Hkv,hd,B", [(2048, 16, 4, 128, 2), (2048, 16, 16, 64, 3), (1024, 28, 4, 128, 2), (512, 44, 11, 64, 2)])
def test_attention_of_a_sequence_alone_and_in_a_batch(S, Hq, Hkv, hd, B):
    """Alone its tiles have a CTA each, in the batch they share one, and a row's sums are added in another order: the outputs
    differ by roundings to bf16 only.  In batches of one kind they have the same bits."""
    from piper_b200.ops import core, native

    tiles = lambda n: native.lib().attn_tiles_per_cta(n, S, Hq, 148)
    assert (tiles(1), tiles(B), tiles(B + 1)) == (1, 2, 2)
    torch.manual_seed(41)
    x = torch.randn(B + 1, S, (Hq + 2 * Hkv) * hd, device="cuda").to(torch.bfloat16)
    run = lambda t: core.attention_fwd(t.reshape(-1, t.shape[-1]), t.shape[0], S, Hq, Hkv, hd, hd ** -0.5)
    alone, lse = run(x[:1])
    both, lse2 = run(x[:B])
    more, lse3 = run(x)
    assert torch.equal(both, more[:B * S]) and torch.equal(lse2, lse3[:B])
    q, k, v = (t.double().transpose(0, 1) for t in x[0].view(S, Hq + 2 * Hkv, hd).split([Hq, Hkv, Hkv], 1))
    k, v = (t.repeat_interleave(Hq // Hkv, 0) for t in (k, v))
    scores = (q @ k.transpose(1, 2) * hd ** -0.5).masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    # every probability is rounded to bf16 once on either side (2^-9 of it each), and so is the output
    spread = (torch.softmax(scores, -1) @ v.abs()).transpose(0, 1).reshape(S, Hq * hd)
    a, b = alone.double(), both[:S].double()
    assert not torch.equal(alone, both[:S])
    assert ((a - b).abs() <= 2 ** -8 * spread + 2 ** -9 * (a.abs() + b.abs()) + 1e-5).all()
    assert ((lse[0].double() - lse2[0].double()).abs() <= 1e-5 * lse[0].double().abs().clamp(min=1)).all()


@pytest.mark.parametrize("N,K", [(4096, 14336), (512, 256), (2048, 2048)])
def test_forward_products_of_a_row_do_not_depend_on_the_others(N, K):
    """Tiles and their shapes follow the number of rows; the sum of a row is the same products in the same order."""
    from piper_b200 import ops

    torch.manual_seed(42)
    x = torch.randn(2500, K, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    y = ops.linear(x, w)
    for rows in (1, 100, 129, 700, 2048):
        assert torch.equal(ops.linear(x[:rows], w), y[:rows]), rows


@pytest.mark.parametrize("T,ignored", [(0, 0.0), (1, 0.0), (33, 0.3), (1023, 1.0), (1024, 0.0), (5000, 0.3), (65536, 0.1), (65537, 0.1)])
def test_cross_entropy_mean(T, ignored):
    """One CTA's sum over any number of rows, and the sum by tensor ops above its limit: value, gradient, and the gradient of
    the gradient by the upstream one, from the C++ formula and the Python one."""
    from piper_b200.ops import core, native

    torch.manual_seed(31)
    logits = torch.randn(T, 16, device="cuda").to(torch.bfloat16).requires_grad_(True)
    labels = torch.randint(0, 16, (T,), device="cuda")
    labels[torch.rand(T, device="cuda") < ignored] = -100
    if ignored == 1.0:
        labels.fill_(-100)
    n = max(1, int((labels != -100).sum()))
    up = torch.tensor(0.7, device="cuda", requires_grad=True)
    results = []
    for installed in (True, False):
        if not installed:
            native.lib().native_op_remove("cross_entropy_mean")
        try:
            rows, _ = core.cross_entropy_fwd(logits, labels, -100)
            mean = core.cross_entropy(logits, labels)
            per_row = rows.detach().requires_grad_(True)
            by_op, count = core.cross_entropy_mean(per_row, labels, -100)
            assert not count.requires_grad and int(count) == n
            (g,) = torch.autograd.grad(by_op, per_row, up, create_graph=True)
            results.append([mean.detach(), g.detach(), *torch.autograd.grad(g.sum(), up)])
        finally:
            native.lib().native_op_install("cross_entropy_mean")
        want = rows.detach().double().sum() / n
        # one rounding of a sum in 64 bits; above the limit fp32 partial sums of positive terms
        assert abs(mean.double() - want) <= (2 ** -23 if T <= core.CE_MEAN_ROWS else 1e-6) * abs(want)
        assert torch.equal(g.detach(), torch.full((T,), 0.7, device="cuda") / n)
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_swiglu_embedding_ce_adam():
    from piper_b200 import ops
    from piper_b200.ops import native

    torch.manual_seed(6)
    h = torch.randn(333, 2 * 1024, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    a = ops.swiglu(h)
    g = torch.randn_like(a)
    a.backward(g)
    hr = h.detach().float().requires_grad_(True)
    ar = torch.nn.functional.silu(hr[:, :1024]) * hr[:, 1024:]
    ar.backward(g.float())
    assert _close(a, ar, 1e-2) and _close(h.grad, hr.grad, 1e-2)

    table = torch.randn(1000, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    tok = torch.randint(0, 1000, (4, 77), device="cuda")
    e = ops.embedding(tok, table)
    ge = torch.randn_like(e)
    e.backward(ge)
    tr = table.detach().float().requires_grad_(True)
    torch.nn.functional.embedding(tok, tr).backward(ge.float())
    assert torch.equal(e, table.detach()[tok])
    assert _close(table.grad, tr.grad, 1e-2)

    V = 5000
    logits = (torch.randn(257, V, device="cuda", dtype=torch.bfloat16) * 3).requires_grad_(True)
    labels = torch.randint(0, V, (257,), device="cuda")
    labels[5] = -100
    loss = ops.cross_entropy(logits, labels)
    loss.backward()
    lr = logits.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lr, labels)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-3 * max(1.0, abs(ref.item()))
    assert _close(logits.grad, lr.grad, 2e-2)

    n = 100_003
    master = torch.randn(n, device="cuda")
    m = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    grad = torch.randn(n, device="cuda")
    p16 = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    pr = master.clone().requires_grad_(True)
    opt = torch.optim.Adam([pr], lr=1e-2, betas=(0.9, 0.95), eps=1e-8)
    for step in (1, 2):
        native.lib().adam_flat(master, m, v, grad, p16, 1e-2, 0.9, 0.95, 1e-8, 0.0, step, 1.0, True)
        pr.grad = grad.clone()
        opt.step()
    assert _close(master, pr.detach(), 1e-5)
    assert _close(p16, pr.detach(), 1e-2)
