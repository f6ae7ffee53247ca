"""Which calls may take a native short cut: plain CUDA tensors with nothing around them that wants to see the call."""
import torch
from torch import Tensor
from torch.autograd import forward_ad
from torch.nn import Parameter


def plain_context() -> bool:
    """No tracing or compiling, no functorch transform, no torch-function or dispatch mode, no forward-mode level: outside these a
    call means what its tensors say.  A microsecond in all."""
    return not (torch.compiler.is_compiling() or torch._C._get_tracing_state() is not None
                or torch._C._are_functorch_transforms_active() or torch._C._len_torch_function_stack()
                or torch._C._len_torch_dispatch_stack() or getattr(forward_ad, "_current_level", 0) >= 0)


def plain_tensors(*tensors) -> bool:
    """Whether a call on these may go to a native function instead of the tensor expressions that give the same: tensors (or
    None in place of one that is optional) of no subclass, on a GPU, in a plain context.  Everything else -- and every
    refusal -- is theirs."""
    for t in tensors:
        if t is not None and not ((type(t) is Tensor or type(t) is Parameter) and t.is_cuda):
            return False
    return plain_context()
