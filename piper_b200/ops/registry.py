"""Registration of the ``torch.ops.piper.*`` ops with the dispatcher.

An op is a schema, one body for all devices, a fake (meta) body and an autograd formula.  The autograd kernel is a
plain ``torch.autograd.Function`` around a call of the same op below autograd, so dispatch modes, fake tensors and
saved-tensor hooks see the op and its saved tensors as with ``torch.library.custom_op``; what is left out is that
wrapper's own work per call, which is host time in front of every launch.  Measured with the kernels of a B200 behind
them, forward and backward: a residual norm 145 us a pass through the wrapper and 118 us through this one (its kernels
take 63 us); the attention layer on 4 x 128 tokens, with its small GEMMs no longer forked, 671 and 332 us.

Gradients that did not arrive (a consumer's backward returned None, or a reentrant checkpoint did not use its input):
the formula of an op with one output is handed zeros in their place.  Where an op has several outputs, most of them
without a gradient in every pass, filling them all would cost launches, so its formula gets None and treats it as zeros.
"""
from __future__ import annotations

from typing import Callable, Optional

import torch

_lib = torch.library.Library("piper", "FRAGMENT")
_below_autograd = torch._C._AutoDispatchBelowAutograd


class Op:
    """What ``custom_op`` returns: callable like the op, with the registration decorators."""

    def __init__(self, name: str, body: Callable) -> None:
        self.name = name
        schema = torch.library.infer_schema(body, mutates_args=())
        _lib.define(name + schema, tags=(torch.Tag.pt2_compliant_tag,))
        self.overload = getattr(torch.ops.piper, name).default
        _lib.impl(name, body, "CompositeExplicitAutograd")

    def register_fake(self, fn: Callable) -> Callable:
        torch.library.register_fake("piper::" + self.name, fn, lib=_lib)
        return fn

    def register_autograd(self, backward: Callable, setup_context: Optional[Callable] = None) -> None:
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
        apply = Formula.apply

        def autograd(*args):
            if torch.is_grad_enabled() and any(isinstance(a, torch.Tensor) and a.requires_grad for a in args):
                return apply(*args)
            with _below_autograd():
                return overload(*args)

        _lib.impl(self.name, autograd, "Autograd")


def custom_op(qualname: str) -> Callable[[Callable], Op]:
    namespace, name = qualname.split("::")
    assert namespace == "piper"
    return lambda body: Op(name, body)
