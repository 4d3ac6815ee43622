"""Several linear layers that read the same input as one matrix product.

The weights are stacked along their output rows; every part starts at a multiple of eight columns of the result, so
that kernels may read it in 16-byte pieces.  `router_logits` is the one product whose result is wanted in fp32.
"""
import torch
import torch.nn as nn
import torch.nn.functional as F
from torch._C import _get_tracing_state, _len_torch_dispatch_stack, _len_torch_function_stack
from torch._C._functorch import peek_interpreter_stack
from torch.autograd import forward_ad
from torch.compiler import is_compiling

from .. import _cabi
from .activation import silu_and_mul

FEW_ROWS = 16
_PLAIN = (torch.Tensor, nn.Parameter)


def _few_rows_pay(n, k, gated):
    """Whether the kernel is the faster one for up to 16 rows and a weight (n, k).  us, kernel and library, 16 rows unless said:
    4,096 x 12,288 21.4 and 22.3, 4,096 x 4,096 9.3 and 9.8, 2,048 x 18,944 21.3 and 25.7; deeper ones the library's from 2,432
    features on (2,560 x 14,336 20.9 and 18.9).  Over 4,736 features CTAs take a second turn: 4,608 x 1,536 5.2 and 5.6, 6,144 x 1,024
    5.3 and 5.4, but 5,120 x 1,536 7.0 and 6.3, 6,144 x 512 4.4 and 4.3, 32,768 x 256 11.0 and 5.6.  Gated, with the activation's
    launch saved: 12,288 x 512 6.5 and 7.5, 16,384 x 512 8.0 and 7.6."""
    if n <= 4096:
        return k <= (18944 if n <= 2048 else 12288)
    if n * k > 8 << 20:
        return False
    return n <= 12288 if gated else n <= 4736 or (n <= 6144 and 768 <= k <= 1024)


def _eager(x, weight):
    """Plain tensors, and nobody about who means to see the product: subclasses, modes, tracing, autocast, forward mode and function
    transforms are served by the library's."""
    return type(x) in _PLAIN and type(weight) in _PLAIN and not (
        is_compiling() or _get_tracing_state() is not None or _len_torch_dispatch_stack() or _len_torch_function_stack() or
        torch.is_autocast_enabled() or forward_ad._current_level >= 0 or peek_interpreter_stack() is not None)


def _few_rows(x, weight, gated):
    """The product of a decode step's rows, or None where it is the library's: more rows, other types, sizes or layouts, a device
    that is not the current one, a weight with which the library's is faster (csrc/few_rows.cu), or one that others must see."""
    if type(x) is not torch.Tensor and not _eager(x, weight):       # before anything is asked of its sizes
        return None
    n, k = weight.shape
    rows = x.shape[0]
    if not (x.is_cuda and x.dim() == 2 and 0 < rows <= FEW_ROWS and x.dtype == weight.dtype and x.shape[1] == k and
            x.dtype in (torch.bfloat16, torch.float16)) or k % 64 or n % (16 if gated else 8) or not _few_rows_pay(n, k, gated) or \
            x.device != weight.device or x.get_device() != torch.cuda.current_device() or not _eager(x, weight) or \
            (torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad)):
        return None
    if x.stride(1) != 1 or not weight.is_contiguous() or x.data_ptr() % 16 or weight.data_ptr() % 16 or \
            (rows > 1 and (x.stride(0) % 8 or x.stride(0) < k)):
        return None
    n = n // 2 if gated else n
    out = torch.empty((rows, n), dtype=x.dtype, device=x.device)
    _cabi.check(_cabi.lib().mv_few_rows(out.data_ptr(), x.data_ptr(), x.stride(0) if rows > 1 else k, weight.data_ptr(), rows, n, k,
                                        int(gated), _cabi.dtype_code(x.dtype), _cabi.stream_ptr()))
    return out


def linear(x, weight):
    """x (rows, in) times weight (out, in)^T."""
    y = _few_rows(x, weight, False)
    return F.linear(x, weight) if y is None else y


def swiglu_linear(x, weight):
    """silu_and_mul(linear(x, weight)), weight (2 * out, in) = [gate; up]."""
    y = _few_rows(x, weight, True)
    return silu_and_mul(F.linear(x, weight)) if y is None else y


class StackedLinear(nn.Module):
    """parts: {name: (out, in) weight}, biases: {name: (out,)} for some of them.  Calling it with (rows, in) returns
    {name: (rows, out) view}."""

    def __init__(self, parts, biases=None):
        super().__init__()
        rows, self.spans, at = [], {}, 0
        for name, w in parts.items():
            n = w.shape[0]
            self.spans[name] = (at, at + n)
            pad = -n % 8
            rows.append(w)
            if pad:
                rows.append(w.new_zeros(pad, w.shape[1]))
            at += n + pad
        self.weight = nn.Parameter(torch.cat(rows) if len(rows) > 1 else rows[0], requires_grad=False)
        self.bias = None
        if biases:
            b = self.weight.new_zeros(at)
            for name, t in biases.items():
                b[self.spans[name][0]:self.spans[name][1]] = t
            self.bias = nn.Parameter(b, requires_grad=False)

    def forward(self, h):
        y = F.linear(h, self.weight, self.bias)
        return {name: y[:, a:b] for name, (a, b) in self.spans.items()}


def router_logits(h, weight):
    """(rows, in) x (experts, in) -> fp32 (rows, experts), products accumulated and kept in fp32."""
    if h.dtype == torch.float32:
        return F.linear(h, weight)
    return torch.mm(h, weight.t(), out_dtype=torch.float32)
