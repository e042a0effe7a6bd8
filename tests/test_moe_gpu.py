"""MoE kernels on the GPU against the PyTorch fp32 reference bodies of the same ops."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


@pytest.mark.parametrize("T,E,k", [(300, 8, 2), (1024, 128, 8)])
def test_router_forward_backward(T, E, k):
    from piper_b200.ops import moe as M, native

    torch.manual_seed(0)
    logits = (torch.randn(T, E, device="cuda") * 2).to(torch.bfloat16).requires_grad_(True)
    w, idx, counts = M.moe_route(logits, k, True)
    lr = logits.detach().cpu().float().requires_grad_(True)
    p = torch.softmax(lr, dim=-1)
    # bf16 logits tie often and tie-breaking is implementation-defined: check the selection by value
    kth = torch.topk(p, k, dim=-1).values[:, -1:]
    sel = torch.gather(p, 1, idx.cpu().long())
    assert (sel >= kth - 1e-6).all()
    assert all(len(set(r)) == k for r in idx.cpu().tolist())
    assert torch.equal(counts.cpu(), torch.bincount(idx.cpu().reshape(-1).long(), minlength=E).to(torch.int32))
    wr = sel / sel.sum(-1, keepdim=True)
    assert _rel(w, wr) < 1e-3
    g = torch.randn(T, k, device="cuda")
    (w * g).sum().backward()
    (wr * g.cpu()).sum().backward()
    assert _rel(logits.grad, lr.grad) < 2e-2
    native.check_status()


@pytest.mark.parametrize("T,D,E,k,F", [(256, 256, 8, 2, 128), (512, 512, 16, 4, 256), (1000, 2048, 128, 8, 768)])
def test_dispatch_grouped_mlp_combine(T, D, E, k, F):
    from piper_b200 import ops
    from piper_b200.ops import moe as M, native

    torch.manual_seed(1)
    x = (torch.randn(T, D, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
    logits = torch.randn(T, E, device="cuda").to(torch.bfloat16)
    w13 = (torch.randn(E, 2 * F, D, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_(True)
    w2 = (torch.randn(E, D, F, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_(True)
    weights, idx, counts = M.moe_route(logits, k, True)
    weights = weights.detach().requires_grad_(True)
    rows, pos, g_start, g_len, epc = M.moe_dispatch(x, idx, counts)
    gs, gl = M.moe_group_table(epc, w13)
    h = M.grouped_linear(rows, w13, gs, gl)
    o = M.grouped_linear(ops.swiglu(h), w2, gs, gl)
    out = M.moe_combine(o, pos, weights, g_start, g_len, counts)
    g = torch.randn_like(out)
    out.backward(g)
    native.check_status()

    # the same pipeline with the reference bodies on the CPU in fp32, reusing the GPU's routing decisions
    xr = x.detach().cpu().float().requires_grad_(True)
    w13r = w13.detach().cpu().float().requires_grad_(True)
    w2r = w2.detach().cpu().float().requires_grad_(True)
    wr = weights.detach().cpu().requires_grad_(True)
    rows_r, pos_r, gs_r, gl_r, _ = M.moe_dispatch(xr, idx.cpu(), counts.cpu())
    h_r = M.grouped_linear(rows_r, w13r, gs_r, gl_r)
    o_r = M.grouped_linear(ops.swiglu(h_r), w2r, gs_r, gl_r)
    out_r = M.moe_combine(o_r, pos_r, wr, gs_r, gl_r, counts.cpu())
    out_r.backward(g.cpu().float())
    assert torch.equal(gs.cpu(), gs_r) and torch.equal(gl.cpu(), gl_r)
    assert sorted(pos.tolist()) == sorted(pos_r.tolist())
    assert _rel(out, out_r) < 2e-2
    assert _rel(x.grad, xr.grad) < 3e-2
    assert _rel(weights.grad, wr.grad) < 3e-2
    assert _rel(w13.grad, w13r.grad) < 3e-2
    assert _rel(w2.grad, w2r.grad) < 3e-2


@pytest.mark.parametrize("E,k", [(8, 8), (33, 3), (64, 1), (256, 8)])
def test_router_expert_counts(E, k):
    """One to eight probability slots per lane, the last one partly filled, and the smallest and largest k."""
    from piper_b200.ops import moe as M

    torch.manual_seed(2)
    rank = torch.rand(130, E, device="cuda").argsort(1)
    logits = (torch.linspace(-4, 4, E, device="cuda")[rank]).to(torch.bfloat16)
    w, idx, counts = M.moe_route(logits, k, True)
    p = torch.softmax(logits.float(), dim=-1)
    wr, _ = torch.topk(p, k, dim=-1)
    assert torch.allclose(torch.gather(p, 1, idx.long()), wr, rtol=1e-6)
    assert all(len(set(r)) == k for r in idx.cpu().tolist())
    assert _rel(w, wr / wr.sum(-1, keepdim=True)) < 1e-5       # fp32 softmax with __expf
    assert torch.equal(counts, torch.bincount(idx.reshape(-1).long(), minlength=E).to(torch.int32))


@pytest.mark.parametrize("T,D,E,k", [(5, 72, 4, 1), (130, 264, 8, 3), (33, 1032, 48, 12), (64, 256, 40, 33)])
def test_permute_and_combine_entry_counts(T, D, E, k):
    """Entry counts with a gather of their own, between them, above eight and above a warp; rows that are no multiple
    of 32 vectors; experts without rows."""
    from piper_b200.ops import moe as M, native

    torch.manual_seed(3)
    x = torch.randn(T, D, device="cuda").to(torch.bfloat16).requires_grad_(True)
    idx = torch.rand(T, E, device="cuda").argsort(1)[:, :k].to(torch.int32).contiguous()
    counts = torch.bincount(idx.reshape(-1).long(), minlength=E).to(torch.int32)
    weights = torch.rand(T, k, device="cuda", requires_grad=True)
    rows, pos, g_start, g_len, _ = M.moe_dispatch(x, idx, counts)
    end = g_start + g_len
    assert torch.equal(g_start[1:], end[:-1]) and torch.equal(g_len, (counts + 127) // 128 * 128)
    assert torch.equal(rows.detach()[pos.long()], x.detach().repeat_interleave(k, dim=0))
    used = torch.zeros(rows.shape[0], dtype=torch.bool, device="cuda")
    used[pos.long()] = True
    assert not rows.detach()[: int(end[-1])][~used[: int(end[-1])]].any()          # padding rows are zero
    out = M.moe_combine(rows * 1.0, pos, weights, g_start, g_len, counts)
    g = torch.randn_like(out)
    out.backward(g)
    xr, wr = x.detach().double(), weights.detach().double()
    gd = g.double()
    assert _rel(out, xr * wr.sum(1, keepdim=True)) < 1e-2
    assert _rel(x.grad, gd * wr.sum(1, keepdim=True)) < 1e-2
    assert _rel(weights.grad, (xr * gd).sum(1, keepdim=True).expand(T, k)) < 1e-2
    native.check_status()


@pytest.mark.parametrize("N,K,sources", [(128, 256, 1), (136, 72, 2), (200, 328, 1), (512, 264, 2)])
def test_grouped_weight_gradient(N, K, sources):
    """bf16 result and fp32 bucket (stored, then accumulated), ragged edges of both dimensions, more than one row
    segment per expert and experts without rows."""
    from piper_b200.ops import native

    torch.manual_seed(4)
    E = 6
    lens = torch.tensor([[128, 0, 256, 384, 0, 128], [256, 0, 0, 128, 128, 0]][:sources], dtype=torch.int32)
    g_len = lens.reshape(-1).cuda()
    g_start = (torch.cumsum(g_len, 0) - g_len).to(torch.int32)
    R = int(g_len.sum())
    x = torch.randn(R, K, device="cuda").to(torch.bfloat16)
    dy = torch.randn(R, N, device="cuda").to(torch.bfloat16)
    want = torch.zeros(E, N, K, dtype=torch.float64, device="cuda")
    for gi, (s, n) in enumerate(zip(g_start.tolist(), g_len.tolist())):
        want[gi % E] += dy[s:s + n].double().t() @ x[s:s + n].double()
    lib, st = native.lib(), native.status_tensor()
    b16 = torch.full((E, N, K), 7.0, device="cuda", dtype=torch.bfloat16)
    lib.grouped_gemm(2, x, dy, None, b16, g_start, g_len, E, N, K, False, st)
    f32 = torch.full((E, N, K), 7.0, device="cuda")
    lib.grouped_gemm(2, x, dy, None, f32, g_start, g_len, E, N, K, False, st)
    scale = want.abs().max()
    assert ((f32.double() - want).abs().max() / scale) < 1e-5          # fp32 sums of up to 512 products
    assert torch.equal(b16, f32.to(torch.bfloat16))                     # the same accumulators, rounded once
    lib.grouped_gemm(2, x, dy, None, f32, g_start, g_len, E, N, K, True, st)
    assert ((f32.double() - 2 * want).abs().max() / scale) < 2e-5
    native.check_status()


@pytest.mark.parametrize("E,N,K,sources", [(40, 520, 72, 1), (40, 264, 712, 2), (3, 128, 64, 2), (5, 72, 520, 1)])
def test_grouped_products_by_pairs_and_single_ctas(E, N, K, sources):
    """Forty experts take CTA pairs, a few single CTAs.  Ragged features on both sides, segments of no rows, one half
    token tile, whole ones and both; rows outside every segment are left alone.  fp32 sums rounded once to bf16."""
    from piper_b200.ops import native

    torch.manual_seed(5)
    units = torch.tensor([0, 1, 2, 3, 5, 4])[torch.arange(E * sources) % 6]
    g_len = (units * 128).to(torch.int32).cuda()
    g_start = (torch.cumsum(g_len, 0) - g_len).to(torch.int32)
    used, R = int(g_len.sum()), int(g_len.sum()) + 128
    x = torch.randn(R, K, device="cuda").to(torch.bfloat16)
    dy = torch.randn(R, N, device="cuda").to(torch.bfloat16)
    w = torch.randn(E, N, K, device="cuda").to(torch.bfloat16)
    y = torch.full((R, N), 7.0, device="cuda", dtype=torch.bfloat16)
    dx = torch.full((R, K), 7.0, device="cuda", dtype=torch.bfloat16)
    lib, st = native.lib(), native.status_tensor()
    lib.grouped_gemm(0, x, None, w, y, g_start, g_len, E, N, K, False, st)
    lib.grouped_gemm(1, None, dy, w, dx, g_start, g_len, E, N, K, False, st)
    native.check_status()
    assert (y[used:] == 7).all() and (dx[used:] == 7).all()
    for gi, (s, n) in enumerate(zip(g_start.tolist(), g_len.tolist())):
        if n:
            for got, want in ((y[s:s + n], x[s:s + n].double() @ w[gi % E].double().t()),
                              (dx[s:s + n], dy[s:s + n].double() @ w[gi % E].double())):
                assert ((got.double() - want).abs().max() / want.abs().max()) < 2 ** -8


def _weight_gradient_with_few_live_experts(E, N, K, sources, live):
    """dW of E experts of which a few have rows: bf16 and fp32 stored over a filled buffer, fp32 accumulated.  fp32 sums of
    up to 640 bf16 products (1e-5 of the largest); experts without rows are zero, or what the buffer held."""
    from piper_b200.ops import native

    torch.manual_seed(8)
    has_rows = {"first": lambda e: e < 3, "last": lambda e: e >= E - 3, "alternating": lambda e: e % 2 == 1,
                "all": lambda e: True, "none": lambda e: False}[live]
    lens = [[128 * (1 + (e + s) % 3) if has_rows(e) and (s == 0 or e % 4 != 1) else 0 for e in range(E)]
            for s in range(sources)]
    g_len = torch.tensor(lens, dtype=torch.int32).reshape(-1).cuda()
    g_start = (torch.cumsum(g_len, 0) - g_len).to(torch.int32)
    R = int(g_len.sum()) + 128                                # rows behind the last segment belong to nobody
    x = torch.randn(R, K, device="cuda").to(torch.bfloat16)
    dy = torch.randn(R, N, device="cuda").to(torch.bfloat16)
    lib, st = native.lib(), native.status_tensor()
    b16 = torch.full((E, N, K), 7.0, device="cuda", dtype=torch.bfloat16)
    f32, added = torch.full((E, N, K), 7.0, device="cuda"), torch.full((E, N, K), 3.0, device="cuda")
    for out, accumulate in ((b16, False), (f32, False), (added, True)):
        lib.grouped_gemm(2, x, dy, None, out, g_start, g_len, E, N, K, accumulate, st)
    native.check_status()
    spans = list(zip(g_start.tolist(), g_len.tolist()))
    for e in range(E):
        want = sum((dy[s:s + n].double().t() @ x[s:s + n].double() for s, n in spans[e::E] if n),
                   torch.zeros(N, K, dtype=torch.float64, device="cuda"))
        bound = 1e-5 * max(1.0, float(want.abs().max()))
        assert (f32[e].double() - want).abs().max() <= (bound if has_rows(e) else 0), e
        assert torch.equal(b16[e], f32[e].to(torch.bfloat16)), e
        assert (added[e].double() - 3 - want).abs().max() <= (bound if has_rows(e) else 0), e


# 128 experts of 5 x 5 pair tiles: some forty tiles per pair, most of them of experts without rows; the smaller ones take
# single CTAs.
_FEW_LIVE = [(128, 1032, 1096, 1, "first"), (128, 1032, 1096, 1, "last"), (128, 1032, 1096, 2, "alternating"),
             (128, 1032, 1096, 1, "none"), (40, 520, 328, 2, "all"), (8, 520, 72, 1, "first"), (12, 136, 264, 2, "last")]


@pytest.mark.parametrize("E,N,K,sources,live", _FEW_LIVE)
def test_grouped_weight_gradient_with_few_live_experts(E, N, K, sources, live):
    _weight_gradient_with_few_live_experts(E, N, K, sources, live)


def test_grouped_weight_gradient_with_few_live_experts_in_static_order():
    """In a process of its own: the order of the tiles is read from the environment once."""
    root = Path(__file__).resolve().parent.parent
    code = ("from tests.test_moe_gpu import _FEW_LIVE, _weight_gradient_with_few_live_experts as check\n"
            "for case in _FEW_LIVE: check(*case)")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=root,
                   env={**os.environ, "PIPER_GEMM_STATIC_TILES": "1"})


def test_qwen3_moe_model_trains_on_one_gpu():
    from piper_b200 import piper_exec_dag, piper_setup
    from piper_b200.models.qwen3 import PiperQwen3Model, Qwen3Config
    from piper_b200.nn import cross_entropy_loss
    from piper_b200.ops import native

    cfg = Qwen3Config(dim=512, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=128, vocab_size=2048, num_experts=16,
                      top_k=4, moe_hidden=256, max_seq_len=256)
    seq = 256
    g = torch.Generator().manual_seed(3)
    tok = torch.randint(0, cfg.vocab_size, (4, seq + 1), generator=g)
    x, y = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    sched = [{"op": "place", "filter": {"PP": 0}, "devices": [0]},
             {"op": "split", "filter": {}, "dim_name": "MB", "num_microbatches": 2}]
    piper_setup(PiperQwen3Model, (cfg, 1, seq), optim_fn=torch.optim.Adam, optim_kwargs={"lr": 1e-3},
                example_inputs=[x], example_outputs=y, model_dtype=torch.bfloat16,
                const_attrs=PiperQwen3Model.const_attrs(cfg, seq), schedule_directives=sched, device="cuda")
    first = [float(v) for v in piper_exec_dag(cross_entropy_loss)]
    for _ in range(8):
        last = [float(v) for v in piper_exec_dag(cross_entropy_loss)]
    native.check_status()
    assert all(v == v for v in first + last)
    assert sum(last) < sum(first) - 0.5, (first, last)


def test_grouped_gemm_with_no_rows():
    """A rank that receives no rows in an expert exchange: forward/input-gradient products are empty and the
    weight gradient is zero (or left untouched when accumulating)."""
    from piper_b200.ops import native

    dev = torch.device("cuda")
    E, N, K = 4, 256, 128
    lib, st = native.lib(), native.status_tensor(dev)
    w = torch.randn(E, N, K, device=dev, dtype=torch.bfloat16)
    rows = torch.empty(0, K, device=dev, dtype=torch.bfloat16)
    dy = torch.empty(0, N, device=dev, dtype=torch.bfloat16)
    g_start = torch.zeros(2 * E, dtype=torch.int32, device=dev)
    g_len = torch.zeros(2 * E, dtype=torch.int32, device=dev)
    out = torch.empty(0, N, device=dev, dtype=torch.bfloat16)
    lib.grouped_gemm(0, rows, None, w, out, g_start, g_len, E, N, K, False, st)
    dx = torch.empty(0, K, device=dev, dtype=torch.bfloat16)
    lib.grouped_gemm(1, None, dy, w, dx, g_start, g_len, E, N, K, False, st)
    dw = torch.full((E, N, K), 3.0, device=dev)
    lib.grouped_gemm(2, rows, dy, None, dw, g_start, g_len, E, N, K, True, st)
    assert torch.all(dw == 3.0)
    lib.grouped_gemm(2, rows, dy, None, dw, g_start, g_len, E, N, K, False, st)
    torch.cuda.synchronize()
    native.check_status()
    assert torch.all(dw == 0.0)


@pytest.mark.parametrize("sources,E,N,K", [(3, 4, 512, 192), (2, 8, 320, 256)])
def test_grouped_gemm_with_groups_from_several_sources(sources, E, N, K):
    """Rows grouped by (source, local expert) with gaps between the sources' regions, empty groups and ragged
    output widths: forward, input gradient and weight gradient against per-segment fp32 products."""
    from piper_b200.ops import native

    torch.manual_seed(3)
    dev = torch.device("cuda")
    lib, st = native.lib(), native.status_tensor(dev)
    blocks = torch.randint(0, 4, (sources * E,)).tolist()          # 128-row blocks per group, some empty
    blocks[1] = 0
    region = (sum(blocks) // sources + 3) * 128                     # every source's region, with slack
    g_start, g_len, at = [], [], 0
    for s in range(sources):
        at = max(at, s * region)
        for e in range(E):
            n = blocks[s * E + e] * 128
            g_start.append(at)
            g_len.append(n)
            at += n
    R = at + 128
    gs = torch.tensor(g_start, dtype=torch.int32, device=dev)
    gl = torch.tensor(g_len, dtype=torch.int32, device=dev)
    w = (torch.randn(E, N, K, device=dev) * 0.1).to(torch.bfloat16)
    rows = torch.randn(R, K, device=dev).to(torch.bfloat16)
    dy = torch.randn(R, N, device=dev).to(torch.bfloat16)
    out = torch.zeros(R, N, device=dev, dtype=torch.bfloat16)
    dx = torch.zeros(R, K, device=dev, dtype=torch.bfloat16)
    dw = torch.zeros(E, N, K, device=dev)
    lib.grouped_gemm(0, rows, None, w, out, gs, gl, E, N, K, False, st)
    lib.grouped_gemm(1, None, dy, w, dx, gs, gl, E, N, K, False, st)
    lib.grouped_gemm(2, rows, dy, None, dw, gs, gl, E, N, K, False, st)
    torch.cuda.synchronize()
    native.check_status()
    want_dw = torch.zeros_like(dw)
    for g, (a, n) in enumerate(zip(g_start, g_len)):
        if n == 0:
            continue
        e = g % E
        ref = rows[a:a + n].float() @ w[e].float().t()
        assert (out[a:a + n].float() - ref).abs().max() <= 2e-2 * ref.abs().max(), g
        ref = dy[a:a + n].float() @ w[e].float()
        assert (dx[a:a + n].float() - ref).abs().max() <= 2e-2 * ref.abs().max(), g
        want_dw[e] += dy[a:a + n].float().t() @ rows[a:a + n].float()
    assert (dw - want_dw).abs().max() <= 2e-2 * want_dw.abs().max()
    assert torch.count_nonzero(out[R - 128:]) == 0                  # rows outside every group are not written
