"""Registration of the ``torch.ops.piper.*`` ops with the dispatcher.

An op is a schema, one body for all devices, a fake (meta) body and an autograd formula.  The autograd kernel is a
plain ``torch.autograd.Function`` around a call of the same op below autograd, so dispatch modes, fake tensors and
saved-tensor hooks see the op and its saved tensors as with ``torch.library.custom_op``; what is left out is that
wrapper's own work per call, which is host time in front of every launch.  Measured with the kernels of a B200 behind
them, forward and backward: a residual norm 150 us a pass through the wrapper and 120 us through this one (its kernels
take 63 us); the attention layer on 4 x 128 tokens, whose small GEMMs are no longer forked either, 604 and 350 us.

On CUDA tensors both kernels of an op are replaced by those of ``csrc/bindings_ops.inc`` once the native library is
loaded: the same bodies and formulas without Python in front of every launch.  A program that registers a formula or a
CUDA kernel of its own gets the Python ones back for that op.

Gradients that did not arrive (a consumer's backward returned None, or a reentrant checkpoint did not use its input):
the formula of an op with one output is handed zeros in their place.  Where an op has several outputs, most of them
without a gradient in every pass, filling them all would cost launches, so its formula gets None and treats it as zeros.
"""
from __future__ import annotations

import contextlib
from typing import Callable, Optional

import torch

from . import native

_below_autograd = torch._C._AutoDispatchBelowAutograd
# One library per op, kept over a reload of this module: defining an op again replaces it.
_libs: dict = globals().get("_libs", {})
_ops: dict = globals().get("_ops", {})


def _library(name: str) -> torch.library.Library:
    stale = _libs.pop(name, None)
    if stale is not None:
        stale._destroy()
    _libs[name] = torch.library.Library("piper", "FRAGMENT")
    return _libs[name]


def host_op(name: str, body: Callable) -> None:
    """Makes a Python function callable from the library as ``piper::<name>``."""
    library = _library(name)
    library.define(name + torch.library.infer_schema(body, mutates_args=()))
    library.impl(name, body, "CompositeExplicitAutograd")


def _install_native(lib) -> None:
    for op in list(_ops.values()):
        if op._use_native:
            lib.native_op_install(op.name)


native.install["registry"] = _install_native


class Op:
    """What ``custom_op`` returns.  The registration methods of ``torch.library.custom_op`` objects are also attributes of
    ``overload``, the callable that the op modules export."""

    def __init__(self, name: str, body: Callable) -> None:
        self.name, self.qualname = name, "piper::" + name
        self._kernels: dict = {}
        self._formula: Optional[Callable] = None
        self._use_native = True
        self._lib = _library(name)
        self._body = body
        self._lib.define(name + torch.library.infer_schema(body, mutates_args=()),
                         tags=(torch.Tag.pt2_compliant_tag,))
        self._lib.impl(name, body, "CompositeExplicitAutograd")
        self.overload = getattr(torch.ops.piper, name).default
        for method in ("register_autocast", "register_autograd", "register_effect", "register_fake", "register_kernel",
                       "register_torch_dispatch", "register_vmap", "set_kernel_enabled"):
            setattr(self.overload, method, getattr(self, method))
        with native.lock:
            _ops[name] = self
            if native.loaded():
                native.lib().native_op_install(name)

    def _drop_native(self) -> None:
        with native.lock:
            self._use_native = False
            if native.loaded():
                native.lib().native_op_remove(self.name)

    def register_fake(self, fn: Callable) -> Callable:
        torch.library.register_fake(self.qualname, fn, lib=self._lib, allow_override=True)
        return fn

    def register_autograd(self, backward: Callable, *, setup_context: Optional[Callable] = None) -> None:
        """``backward(ctx, *grads)`` returns a gradient per input; see above for gradients that did not arrive."""
        overload = self.overload
        one_output = len(overload._schema.returns) == 1

        class Formula(torch.autograd.Function):
            @staticmethod
            def forward(ctx, *args):
                with _below_autograd():
                    out = overload(*args)
                if not one_output:
                    ctx.set_materialize_grads(False)
                if setup_context is not None:
                    setup_context(ctx, args, out)
                return out

        Formula.backward = staticmethod(backward)
        Formula.__name__ = Formula.__qualname__ = f"piper_{self.name}"
        registered, self._formula = self._formula is not None, Formula.apply
        if registered:
            self._drop_native()
            return

        def autograd(*args):
            if torch.is_grad_enabled() and any(isinstance(a, torch.Tensor) and a.requires_grad for a in args):
                return self._formula(*args)
            with _below_autograd():
                return overload(*args)

        self._lib.impl(self.name, autograd, "Autograd")

    def register_kernel(self, device_types, func: Optional[Callable] = None) -> Callable:
        """A body for one device type, several, or (None) all, in place of the general one."""
        if func is None:
            return lambda f: self.register_kernel(device_types, f)
        if device_types is None or isinstance(device_types, str):
            device_types = ("cpu", "cuda") if device_types is None else (device_types,)
        if any(torch.device(device).type == "cuda" for device in device_types):
            self._drop_native()
        for device in device_types:
            known = device in self._kernels
            self._kernels[device] = func
            if not known:
                torch.library.register_kernel(
                    self.overload, device, lambda *args, _d=device: (self._kernels[_d] or self._body)(*args),
                    lib=self._lib)
        return func

    @contextlib.contextmanager
    def set_kernel_enabled(self, device_type: str, enabled: bool = True):
        """Scope in which a device's registered kernel is used or the general body in its place."""
        before = self._kernels.get(device_type)
        if before is not None and not enabled:
            self._kernels[device_type] = None
        try:
            yield
        finally:
            if before is not None:
                self._kernels[device_type] = before

    def register_vmap(self, func: Optional[Callable] = None):
        return torch.library.register_vmap(self.overload, func, lib=self._lib)

    def register_torch_dispatch(self, torch_dispatch_class, fn: Optional[Callable] = None):
        return torch.library.register_torch_dispatch(self.qualname, torch_dispatch_class, fn, lib=self._lib)

    def register_autocast(self, device_type: str, cast_inputs: torch.dtype):
        return torch.library.register_autocast(self.overload, device_type, cast_inputs, lib=self._lib)

    def register_effect(self, effect) -> None:
        torch.library._register_effectful_op(self.qualname, effect)


def custom_op(qualname: str) -> Callable[[Callable], Op]:
    namespace, name = qualname.split("::")
    assert namespace == "piper"
    return lambda body: Op(name, body)
