"""The op registration against what programs rely on: dispatch modes, fake tensors, saved-tensor hooks, keyword calls,
gradients of single outputs."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch
import torch.utils.checkpoint

from piper_b200 import ops
from piper_b200.ops import core, moe


def test_ops_are_single_dispatcher_calls_and_hooks_see_their_saved_tensors():
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    x, w = torch.randn(4, 16, requires_grad=True), torch.randn(8, 16, requires_grad=True)
    packed = []
    with Mode(), torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t)[1], lambda t: t):
        y = ops.linear(x=x, w=w)
    assert seen.count("piper.linear.default") == 1 and packed == [x.shape, w.shape]
    y.sum().backward()
    assert torch.allclose(w.grad, x.detach().sum(0).expand(8, 16)) and x.grad is not None
    with torch.no_grad():
        assert not ops.linear(x, w).requires_grad
    # weights without gradients: a weight-gradient formula looks its bucket up by address, which tracers do not have
    torch.library.opcheck(torch.ops.piper.linear.default, (x, w.detach()))
    torch.library.opcheck(torch.ops.piper.swiglu.default, (x,))


def test_full_graph_capture_records_the_op():
    x, w = torch.randn(4, 16, requires_grad=True), torch.randn(8, 16)
    for backend in ("eager", "aot_eager"):
        f = torch.compile(lambda a: ops.linear(a, w).sum(), backend=backend, fullgraph=True)
        assert torch.allclose(f(x), ops.linear(x, w).sum())


@pytest.mark.parametrize("pick", [0, 1, 2])
def test_gradients_of_one_output_alone(pick):
    """Outputs that a program did not use send no gradient: the formula sees zeros in their place."""
    x, r, w = torch.randn(4, 16, requires_grad=True), torch.randn(4, 16), torch.randn(16)
    out = core.add_rmsnorm_fwd(x, r, w, 1e-5)[pick]
    (g,) = torch.autograd.grad(out.sum(), x)
    h = (x.detach() + r).requires_grad_(True)
    rstd = torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5)
    want = torch.autograd.grad([h * rstd * w, h][pick].sum(), h)[0] if pick < 2 else torch.zeros_like(x)
    assert torch.allclose(g, want, atol=1e-5)
    qkv = torch.randn(128, 3 * 64, requires_grad=True)
    o, lse = core.attention_fwd(qkv, 1, 128, 1, 1, 64, 0.125)
    assert torch.isfinite(torch.autograd.grad((o if pick else lse).sum(), qkv)[0]).all()


def test_integer_outputs_carry_no_gradient():
    counts = torch.tensor([3, 5], dtype=torch.int32)
    start, length = moe.moe_group_table(counts, torch.randn(2, 4, 4, requires_grad=True))
    assert not start.requires_grad and length.tolist() == [128, 128]


class _Drop(torch.autograd.Function):
    """A consumer that sends no gradient back."""

    @staticmethod
    def forward(ctx, y):
        return y.sum() * 0.0

    @staticmethod
    def backward(ctx, g):
        return None


def _one_output_calls():
    T, E, k, D = 6, 4, 2, 16
    idx = torch.rand(T, E).argsort(1)[:, :k].to(torch.int32).contiguous()
    counts = torch.bincount(idx.reshape(-1).long(), minlength=E).to(torch.int32)
    rows, pos, g_start, g_len, _ = moe.moe_dispatch(torch.randn(T, D), idx, counts)
    cos, sin = torch.randn(T, 32), torch.randn(T, 32)
    return {
        "linear": (core.linear, [(T, D), (8, D)]),
        "rmsnorm": (lambda x, w: core.rmsnorm_fwd(x, w, 1e-5)[0], [(T, D), (D,)]),
        "add_rmsnorm": (lambda x, r, w: core.add_rmsnorm_fwd(x, r, w, 1e-5)[0], [(T, D), (T, D), (D,)]),
        "residual_add": (core.residual_add, [(T, D), (T, D)]),
        "qk_rope": (lambda x, q, k_: core.qk_rope(x, cos, sin, q, k_, T, 1, 1, 64, False, 1e-5),
                    [(T, 192), (64,), (64,)]),
        "attention": (lambda x: core.attention_fwd(x, 1, 128, 1, 1, 64, 0.1)[0], [(128, 192)]),
        "swiglu": (core.swiglu, [(T, D)]),
        "embedding": (lambda t: core.embedding(torch.arange(T), t), [(9, D)]),
        "cross_entropy": (lambda x: core.cross_entropy_fwd(x, torch.zeros(T, dtype=torch.long), -100)[0], [(T, D)]),
        "moe_route": (lambda x: moe.moe_route(x, k, True)[0], [(T, E)]),
        "moe_dispatch": (lambda x: moe.moe_dispatch(x, idx, counts)[0], [(T, D)]),
        "grouped_linear": (lambda r, w: moe.grouped_linear(r, w, g_start, g_len), [tuple(rows.shape), (E, 8, D)]),
        "moe_combine": (lambda r, w: moe.moe_combine(r, pos, w, g_start, g_len, counts), [tuple(rows.shape), (T, k)]),
    }


@pytest.mark.parametrize("name", sorted(_one_output_calls()))
def test_a_gradient_that_does_not_arrive_counts_as_zeros(name):
    fn, shapes = _one_output_calls()[name]
    args = [torch.randn(s, requires_grad=True) for s in shapes]
    _Drop.apply(fn(*args)).backward()
    for a in args:
        assert a.grad is not None and a.grad.shape == a.shape and a.grad.dtype == a.dtype and not a.grad.any()


def test_reentrant_checkpoint_over_a_block_that_only_detaches_its_input():
    x, w = torch.randn(4, 16, requires_grad=True), torch.randn(8, 16, requires_grad=True)
    q = torch.randn(3, requires_grad=True)
    out = torch.utils.checkpoint.checkpoint(lambda y, z: z * 2 + y.detach().sum(), core.linear(x, w), q, use_reentrant=True)
    out.sum().backward()
    assert not x.grad.any() and not w.grad.any() and torch.equal(q.grad, torch.full((3,), 2.0))


_MODULE_CHANGES = """
import importlib, torch
from piper_b200 import ops
from piper_b200.ops import core, moe, registry
torch.manual_seed(0)
x, w = torch.randn(4, 16, requires_grad=True), torch.randn(8, 16, requires_grad=True)
want = (x @ w.t()).detach()
before = ops.linear
for module in (registry, core, moe):
    importlib.reload(module)
for f in (before, core.linear, torch.ops.piper.linear):
    x.grad = None
    y = f(x, w)
    y.sum().backward()
    # sums of 8 fp32 numbers below 5 in two orders: 2 x 7 x 2^-24 x 40, which a sum near zero exceeds relatively
    assert torch.allclose(y, want) and torch.allclose(x.grad, w.detach().sum(0).expand(4, 16), atol=4e-5)
start, length = moe.moe_group_table(torch.tensor([3, 5], dtype=torch.int32), torch.randn(2, 4, 4))
assert length.tolist() == [128, 128]

op = core.linear
op.register_kernel("cpu", lambda a, b: a @ b.t() + 1)
assert torch.allclose(op(x, w), want + 1)
with op.set_kernel_enabled("cpu", False):
    assert torch.allclose(op(x, w), want)
op.register_kernel(None)(lambda a, b: a @ b.t() + 2)
assert torch.allclose(op(x, w), want + 2)
op.register_autocast("cpu", torch.bfloat16)
with torch.autocast("cpu", dtype=torch.bfloat16):
    assert op(x, w).dtype == torch.bfloat16
op.register_vmap(lambda info, dims, a, b: (a * 3, dims[0]))
assert torch.equal(torch.func.vmap(op, in_dims=(0, None))(x.detach()[None], w.detach()), x.detach()[None] * 3)
op.register_fake(lambda a, b: a.new_empty(7))
with torch._subclasses.FakeTensorMode():
    assert op(torch.empty(4, 16), torch.empty(8, 16)).shape == (7,)
op.register_autograd(lambda ctx, g: (torch.full((4, 16), 5.0), None))
x.grad = None
op(x, w).sum().backward()
assert (x.grad == 5).all()
"""


def test_op_modules_reload_and_ops_take_further_registrations():
    """In a process of its own: both change the ops for everything after them."""
    root = Path(__file__).resolve().parent.parent
    subprocess.run([sys.executable, "-c", _MODULE_CHANGES], check=True, timeout=300, cwd=root)


_EARLIER_KERNEL = """
import torch
from piper_b200.ops import core, native
torch.library.register_kernel("piper::swiglu", "cuda", lambda h: h[..., : h.shape[-1] // 2] * 0 + 2)
lib = native.lib()                 # loaded by the first CUDA call of a program
assert not lib.native_op_install("swiglu") and lib.native_op_install("linear")
table = torch._C._dispatch_dump_table("piper::swiglu").splitlines()
assert [line for line in table if line.startswith("CUDA:")] and not [line for line in table if "bindings_ops" in line]
lib.native_op_remove("linear")
assert lib.native_op_install("linear")
if torch.cuda.is_available():
    h = torch.ones(2, 8, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    assert (core.swiglu(h) == 2).all()
"""


@pytest.mark.parametrize("where", ["cpu", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_kernels_registered_before_the_library_is_loaded_stay(where):
    """A program's own CUDA kernel, registered with the dispatcher, is not hidden by the library's."""
    from piper_b200.ops import native

    if not native.lib_path().exists():
        pytest.skip("the native library has not been built")
    root = Path(__file__).resolve().parent.parent
    subprocess.run([sys.executable, "-c", _EARLIER_KERNEL], check=True, timeout=300, cwd=root)


def test_the_library_has_the_state_before_it_counts_as_loaded(monkeypatch, tmp_path):
    """A stand-in library that records its calls: flags and buckets are handed over before an op is installed, nobody sees
    the library as loaded before that, and a bucket that another thread registers meanwhile is not lost."""
    import threading
    import types

    from piper_b200.ops import native

    calls, handing, registered = [], threading.Event(), threading.Event()

    class Call:
        def __init__(self, name):
            self.name = name

        def __call__(self, *args):
            calls.append((self.name, native.loaded(), args))
            if self.name == "sink_clear":
                handing.set()
                registered.wait(0.2)              # the other thread waits for the lock, so this runs out

        default = property(lambda self: self)

    fake = types.SimpleNamespace(**{n: Call(n) for n in (
        "set_op_flag", "set_fork_macs", "sink_clear", "sink_set", "sink_unset", "native_op_install", "native_op_remove")})
    (tmp_path / "lib.so").touch()
    monkeypatch.setattr(native, "_LIB_PATH", tmp_path / "lib.so")
    monkeypatch.setattr(native, "_loaded", False)
    monkeypatch.setattr(native, "torch", types.SimpleNamespace(ops=types.SimpleNamespace(
        piper_c=fake, load_library=lambda path: None)))
    early, late = torch.randn(4), torch.randn(5)
    core.grad_sinks.register(early, torch.zeros(4))

    def register():
        handing.wait(10)
        core.grad_sinks.register(late, torch.zeros(5))
        registered.set()

    thread = threading.Thread(target=register)
    thread.start()
    try:
        assert native.lib() is fake and native.loaded()
        thread.join(10)
        assert registered.is_set()
        loading = [c for c in calls if not c[1]]
        kinds = [name for name, _, _ in loading]
        assert kinds == sorted(kinds, key=["set_op_flag", "set_fork_macs", "sink_clear", "sink_set", "native_op_install"].index)
        assert {a[0] for n, _, a in loading if n == "native_op_install"} >= {"linear", "moe_dispatch"}
        sinks = [a[0] for n, _, a in calls if n == "sink_set"]
        assert early.data_ptr() in sinks and late.data_ptr() in sinks
    finally:
        core.grad_sinks.unregister(early)
        core.grad_sinks.unregister(late)


def _cuda_calls():
    """Calls on CUDA tensors, with the arguments that take gradients."""
    def rn(*shape):
        return torch.randn(*shape, device="cuda").to(torch.bfloat16)

    E, k, T = 8, 2, 4
    idx = torch.arange(T * k, device="cuda", dtype=torch.int32).view(T, k)          # one row per expert: a fixed order
    counts = torch.ones(E, device="cuda", dtype=torch.int32)
    cos, sin = torch.randn(128, 32, device="cuda"), torch.randn(128, 32, device="cuda")
    with torch.no_grad():
        rows, pos, g_start, g_len, _ = moe.moe_dispatch(rn(T, 64), idx, counts)
    rows = rows[: int((g_start + g_len)[-1])].clone()
    labels, tokens = torch.randint(0, 64, (6,), device="cuda"), torch.tensor([7, 0, 3, 1, 8, 5], device="cuda")
    return {
        "linear": (core.linear, [rn(3, 2, 64), rn(8, 64)]),
        "rmsnorm_fwd": (lambda x, w: core.rmsnorm_fwd(x, w, 1e-5), [rn(3, 2, 256), rn(256)]),
        "add_rmsnorm_fwd": (lambda x, r, w: core.add_rmsnorm_fwd(x, r, w, 1e-5), [rn(6, 256), rn(6, 256), rn(256)]),
        "residual_add": (core.residual_add, [rn(6, 64), rn(6, 64)]),
        "qk_rope": (lambda x: core.qk_rope(x, cos, sin, None, None, 128, 2, 1, 64, True, 1e-5), [rn(128, 256)]),
        "qk_rope normed": (lambda x, q, w: core.qk_rope(x, cos, sin, q, w, 128, 2, 1, 64, False, 1e-5),
                           [rn(128, 256), rn(64), rn(64)]),
        "attention_fwd": (lambda x: core.attention_fwd(x, 1, 128, 2, 1, 64, 0.125), [rn(128, 256)]),
        "swiglu": (core.swiglu, [rn(2, 3, 64)]),
        "embedding": (lambda t: core.embedding(tokens, t), [rn(9, 64)]),
        "cross_entropy_fwd": (lambda x: core.cross_entropy_fwd(x, labels, -100), [rn(6, 64)]),
        "moe_route": (lambda x: moe.moe_route(x, k, True), [rn(T, E)]),
        "moe_group_table": (lambda w: moe.moe_group_table(counts, w), [rn(E, 8, 8)]),
        "moe_dispatch": (lambda x: moe.moe_dispatch(x, idx, counts), [rn(T, 64)]),
        "grouped_linear": (lambda r, w: moe.grouped_linear(r, w, g_start, g_len), [rows, rn(E, 72, 64)]),
        "moe_combine": (lambda r, w: moe.moe_combine(r, pos, w, g_start, g_len, counts),
                        [rows, torch.rand(T, k, device="cuda")]),
    }


def _one_pass(fn, args, form):
    """Outputs, gradients, buckets of one pass in some form of the call."""
    torch.manual_seed(7)
    if form == "strided":
        args = [torch.stack((args[0], args[0]), -1)[..., 0], *args[1:]]
    leaves = [a.detach().requires_grad_(form != "first only" or i == 0) for i, a in enumerate(args)]
    sinks = {}
    if form in ("sinks", "deferred"):
        sinks = {i: torch.randn(a.shape, device="cuda") for i, a in enumerate(leaves) if i > 0}
    for i, sink in sinks.items():
        core.grad_sinks.register(leaves[i], sink)
    queue = core.wgrad_store.begin() if form == "deferred" else []
    try:
        with torch.set_grad_enabled(form != "no grad"):
            out = fn(*leaves)
        outs = list(out) if isinstance(out, tuple) else [out]
        heads = [o for o in outs if o.requires_grad][:1 if form == "first output" else None]
        if heads and form == "dropped":
            _Drop.apply(heads[0]).backward()
        elif heads:
            torch.autograd.backward(heads, [torch.full((), 0.5, device="cuda", dtype=o.dtype).expand_as(o)
                                            if form == "broadcast" else torch.randn_like(o) for o in heads])
        core.wgrad_store.end()
        assert not core.wgrad_store.drain(queue)             # every weight that defers has a bucket here
    finally:
        core.wgrad_store.end()
        for i in sinks:
            core.grad_sinks.unregister(leaves[i])
    return [o.detach() for o in outs], [a.grad for a in leaves], list(sinks.values()), [o.requires_grad for o in outs]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "no grad", "first only", "first output", "strided", "broadcast", "dropped", "sinks",
                                  "deferred"])
def test_native_formulas_do_what_the_python_ones_do(form):
    """Every op on CUDA tensors by its C++ kernels and by the Python ones, in the forms in which programs call them: the
    same bits, the same absent gradients, the same sums in the buckets (of norm weights of rotary heads, which atomics add
    up in any order, to fp32 rounding of 128 x 2 summands)."""
    from piper_b200.ops import native

    torch.manual_seed(6)
    lib = native.lib()
    for name, (fn, args) in _cuda_calls().items():
        op = name.split()[0]
        if form == "strided" and op in ("grouped_linear", "moe_combine"):
            continue                                         # rows come from dispatch, whole
        got = _one_pass(fn, args, form)
        lib.native_op_remove(op)
        try:
            want = _one_pass(fn, args, form)
        finally:
            lib.native_op_install(op)
        assert got[3] == want[3], name
        for part, (a, b) in enumerate(zip(got[:3], want[:3])):
            assert len(a) == len(b)
            for i, (x, y) in enumerate(zip(a, b)):
                assert (x is None) == (y is None), (name, part, i)
                if x is None:
                    continue
                assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride(), (name, part, i)
                if name == "qk_rope normed" and (part == 2 or part == 1 and i > 0):
                    assert torch.allclose(x.float(), y.float(), rtol=1e-2, atol=1e-3), (name, part, i)
                elif not (op == "moe_dispatch" and part == 0 and i == 0):       # rows behind the last segment are undefined
                    assert torch.equal(x, y), (name, part, i)
    native.check_status()


@pytest.mark.gpu
def test_native_formulas_under_a_recomputing_checkpoint():
    """A non-reentrant checkpoint recomputes the saved tensors in their unpack hooks, inside the backward pass of the formula
    that asks for them: the same outputs and gradients as without it (weights of rotary heads, which atomics add up in any order,
    to the rounding of their bf16 results)."""
    from piper_b200.ops import native

    torch.manual_seed(9)
    for name, (fn, args) in _cuda_calls().items():
        def block(*leaves):
            return fn(*(a * 1.0 for a in leaves))            # what is saved is made inside the block
        plain = _one_pass(block, args, "plain")
        again = _one_pass(lambda *leaves: torch.utils.checkpoint.checkpoint(block, *leaves, use_reentrant=False), args, "plain")
        assert plain[3] == again[3], name
        for x, y in zip(plain[0] + plain[1], again[0] + again[1]):
            assert (x is None) == (y is None), name
            if x is not None and name.startswith("qk_rope normed"):
                assert torch.allclose(x.float(), y.float(), rtol=1e-2, atol=1e-3), name
            elif x is not None and name != "moe_dispatch":
                assert torch.equal(x, y), name
            elif x is not None and x.shape == args[0].shape:       # rows behind the last segment are undefined
                assert torch.equal(x, y), name
    native.check_status()


@pytest.mark.gpu
def test_native_bodies_refuse_the_shapes_that_the_python_ones_refuse():
    """The bodies unpack their arguments' shapes, and so does the fake body: [tokens, experts], [tokens, features], [experts, N,
    K], [tokens, k], at least one dimension for the activation."""
    def b16(*shape):
        return torch.zeros(shape, device="cuda", dtype=torch.bfloat16)

    i1, i2 = torch.zeros(4, device="cuda", dtype=torch.int32), torch.zeros(4, 2, device="cuda", dtype=torch.int32)
    calls = [lambda: moe.moe_route(b16(4, 3, 8), 2, True), lambda: moe.moe_route(b16(8), 2, True), lambda: core.swiglu(b16()),
             lambda: moe.moe_dispatch(b16(4, 3, 8), i2, i1), lambda: moe.moe_dispatch(b16(4, 8), i1, i1),
             lambda: moe.grouped_linear(b16(128, 8), b16(8, 8), i1, i1),
             lambda: moe.moe_combine(b16(128, 8), i1, torch.zeros(4, device="cuda"), i1, i1, i1)]
    for call in calls:
        with pytest.raises((RuntimeError, ValueError, IndexError)):
            call()


@pytest.mark.gpu
def test_native_bodies_refuse_empty_rows():
    """A last dimension of zero (or half of one) raises, as it did in Python, and does not divide by zero."""
    def b16(*shape):
        return torch.zeros(shape, device="cuda", dtype=torch.bfloat16)

    cos = torch.zeros(4, 0, device="cuda")
    for call in (lambda: core.rmsnorm_fwd(b16(4, 0), b16(0), 1e-5), lambda: core.add_rmsnorm_fwd(b16(4, 0), b16(4, 0), b16(0), 1e-5),
                 lambda: core.swiglu(b16(4, 0)), lambda: core.swiglu(b16(4, 1)),
                 lambda: core.qk_rope(b16(4, 0), cos, cos, None, None, 4, 2, 1, 0, False, 1e-5)):
        with pytest.raises((RuntimeError, ZeroDivisionError)):
            call()


@pytest.mark.gpu
def test_linear_and_cross_entropy_refuse_empty_rows_of_a_wider_matrix():
    """Columns [0, 0) of a matrix are contiguous and keep its row stride: what the kernels check lets them by."""
    x, w = (torch.zeros(4, 8, device="cuda", dtype=torch.bfloat16)[:, :0] for _ in range(2))
    for call in (lambda: core.linear(x, w), lambda: core.linear(x.clone(), w.clone()), lambda: core.linear(x[None], w),
                 lambda: core.cross_entropy(x, torch.zeros(4, device="cuda", dtype=torch.long))):
        with pytest.raises(RuntimeError):
            call()


@pytest.mark.gpu
def test_cross_entropy_refuses_labels_that_the_device_cannot_read():
    """Labels in host memory raise before a kernel gets their address, in the loss and in its mean; pinned ones are read."""
    logits = torch.randn(4, 16, device="cuda").to(torch.bfloat16)
    labels = torch.tensor([1, -100, 15, 3])
    loss, _ = core.cross_entropy_fwd(logits, labels.cuda(), -100)
    for call in (lambda: core.cross_entropy(logits, labels), lambda: core.cross_entropy_mean(loss, labels, -100)):
        with pytest.raises(RuntimeError):
            call()
    assert torch.equal(core.cross_entropy(logits, labels.pin_memory()), core.cross_entropy(logits, labels.cuda()))


@pytest.mark.gpu
def test_a_traced_mean_loss_has_no_guard_on_its_rows():
    """A program exported or compiled with any number of rows runs with one token and with more than one CTA adds up."""
    class Loss(torch.nn.Module):
        def forward(self, logits, labels):
            return core.cross_entropy(logits, labels)

    def args(rows):
        return torch.randn(rows, 64, device="cuda").to(torch.bfloat16), torch.randint(0, 64, (rows,), device="cuda")

    torch.manual_seed(11)
    rows, graphs = torch.export.Dim("rows"), []
    exported = torch.export.export(Loss(), args(40), dynamic_shapes=({0: rows}, {0: rows})).module()
    compiled = torch.compile(Loss(), backend=lambda gm, _: graphs.append(gm) or gm.forward, dynamic=True, fullgraph=True)
    for n in (40, 50, core.CE_MEAN_ROWS + 1):
        a, b = args(n)
        want = core.cross_entropy(a, b)
        assert torch.equal(exported(a, b), want) and torch.equal(compiled(a, b), want)
    assert len(graphs) == 1
    # more labels than rows, all of which count, as they do in tensor operations
    losses, more = core.cross_entropy_fwd(a[:3], b[:3], -100)[0], b[:7]
    assert torch.equal(core.cross_entropy(a[:3], more), losses.sum() / (more != -100).sum())     # not the reciprocal of a number


@pytest.mark.gpu
def test_per_token_cross_entropy_gradient_keeps_its_graph():
    """With a gradient per token the formula is tensor arithmetic: under create_graph its result can be differentiated by the
    upstream gradient, by the C++ formula as by the Python one."""
    from piper_b200.ops import native

    torch.manual_seed(10)
    logits = torch.randn(6, 64, device="cuda").to(torch.bfloat16).requires_grad_(True)
    labels = torch.tensor([3, -100, 0, 63, 7, 7], device="cuda")
    up, v = torch.randn(6, device="cuda", requires_grad=True), torch.randn(6, 64, device="cuda")
    results = []
    for installed in (True, False):
        if not installed:
            native.lib().native_op_remove("cross_entropy_fwd")
        try:
            loss, _ = core.cross_entropy_fwd(logits, labels, -100)
            (g,) = torch.autograd.grad(loss, logits, up, create_graph=True)
            assert g.requires_grad
            results.append([g, *torch.autograd.grad((g.float() * v).sum(), up)])
        finally:
            native.lib().native_op_install("cross_entropy_fwd")
    assert all(torch.equal(a, b) for a, b in zip(*results))
    p = torch.softmax(logits.detach().double(), -1) - torch.nn.functional.one_hot(labels.clamp(min=0), 64)
    want = (p * v).sum(-1) * (labels != -100)
    bound = 2 ** -8 * (p * v).abs().sum(-1)                  # every summand is rounded to bf16 (2^-9), in fp32 sums
    assert ((results[0][1] - want).abs() <= bound).all()


@pytest.mark.gpu
def test_profilers_and_dispatch_modes_see_native_formulas_as_python_ones():
    """The kernels that a pass launches are ops of their own, which a profiler lists; a dispatch mode sees the op itself and what a
    backward pass allocates.  (The C++ formulas run below autograd, so there it sees their kernels as well.)"""
    from torch.utils._python_dispatch import TorchDispatchMode

    from piper_b200.ops import native

    def listed(fn, args):
        seen = []

        class Mode(TorchDispatchMode):
            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                seen.append(str(func))
                return func(*args, **(kwargs or {}))

        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
            _one_pass(fn, args, "plain")
        with Mode():
            _one_pass(fn, args, "plain")
        asks = ("rmsnorm_bwd_num_partials", "attn_bwd_floats")       # sizes: no kernels
        return (sorted(e.name for e in prof.events() if e.name.startswith("piper_c::") and not e.name.endswith(asks)),
                [n for n in seen if n.startswith("piper.")], any(n.startswith("aten.empty") for n in seen))

    torch.manual_seed(11)
    for name, (fn, args) in _cuda_calls().items():
        op = name.split()[0]
        got = listed(fn, args)
        native.lib().native_op_remove(op)
        try:
            want = listed(fn, args)
        finally:
            native.lib().native_op_install(op)
        assert got == want and got[0], (name, got, want)


_CUDA_CHANGES = """
import importlib, torch
from piper_b200 import ops
from piper_b200.ops import core, moe, native, registry
def rn(*s): return torch.randn(*s, device="cuda").to(torch.bfloat16)
x, w = rn(8, 64).requires_grad_(True), rn(16, 64)
want = ops.linear(x, w).detach()
sink = torch.zeros(16, 64, device="cuda")
core.grad_sinks.register(w, sink)
for module in (registry, core, moe):
    importlib.reload(module)
for f in (ops.linear, core.linear, torch.ops.piper.linear):
    assert torch.equal(f(x, w), want)
w.requires_grad_(True)
core.linear(x, w).sum().backward()
assert w.grad is not None and not sink.any()           # the buckets of the module before are forgotten
for bad in (x.detach().float(), x.detach().half()):
    try:
        core.linear(bad, w)
        raise SystemExit("accepted " + str(bad.dtype))
    except TypeError as e:
        assert str(bad.dtype) in str(e)
core.gather_gemms[w.data_ptr()] = lambda x2, y: y.fill_(3)
assert (core.linear(x, w) == 3).all() and torch.equal(core.linear(x, w), want)     # used once
moe.set_ep_context(None, (torch.tensor([1, 2], device="cuda", dtype=torch.int32),) * 2)
counts = torch.tensor([3, 5], device="cuda", dtype=torch.int32)
assert moe.moe_group_table(counts, rn(2, 8, 8))[0].tolist() == [1, 2]
moe.set_ep_context(None, None)
assert moe.moe_group_table(counts, rn(2, 8, 8))[0].tolist() == [0, 128]
seen = []
with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t)[1], lambda t: t):
    core.linear(x, w)
assert seen == [x.shape, w.shape]
op = core.linear
op.register_autograd(lambda ctx, g: (torch.full((8, 64), 5.0, device="cuda", dtype=torch.bfloat16), None))
x.grad = None
op(x, w).sum().backward()
assert (x.grad == 5).all()
op = core.swiglu
op.register_kernel("cuda", lambda h: h[..., :1] * 0 + 2)
assert (op(x) == 2).all()
with op.set_kernel_enabled("cuda", False):
    assert not (op(x) == 2).all()
with torch._subclasses.FakeTensorMode():
    h = torch.empty(4, 32, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    assert core.rmsnorm_fwd(h, torch.empty(32, device="cuda", dtype=torch.bfloat16), 1e-5)[0].shape == (4, 32)
try:
    torch.func.grad(lambda a: core.residual_add(a, a).sum())(x.detach())
    raise SystemExit("functorch transforms were refused before")
except RuntimeError:
    pass
native.check_status()
"""


@pytest.mark.gpu
def test_native_formulas_give_way_to_python_state_and_registrations():
    root = Path(__file__).resolve().parent.parent
    subprocess.run([sys.executable, "-c", _CUDA_CHANGES], check=True, timeout=300, cwd=root)
