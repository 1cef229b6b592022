"""torch.autograd binding of the hand-written adjoint.

``FlareEnergy.apply(positions, gp, structure, precision)`` returns the energy
of a mapped SparseGP model for device positions (float64, n x 3).  Its
backward is the library's adjoint (forces are -dE/dx), so
``torch.autograd.grad(E, positions)`` gives -forces without any stored
descriptor derivatives.  The virial stress of the same evaluation is left on
the structure as ``structure.last_stress`` (flare order xx, xy, xz, yy, yz,
zz).
"""
import torch

from . import _lib
from ._lib import check, lib
from .api import PRECISIONS


def _evaluate(positions, gp, structure, precision):
    """Energy (0-d), forces (n, 3) and stress (6) of the mapped model on the current
    stream; every element is written by the library."""
    if positions.dtype != torch.float64 or not positions.is_cuda:
        raise TypeError("positions must be a CUDA float64 tensor")
    pos = positions.detach().contiguous()
    stream = torch.cuda.current_stream(pos.device).cuda_stream
    check(lib().fpp_structure_set_positions(structure.handle, pos.data_ptr(), 1, stream))
    gp._ensure_mapped(stream)
    n = structure.noa
    e = torch.empty((), dtype=torch.float64, device=pos.device)
    f = torch.empty((n, 3), dtype=torch.float64, device=pos.device)
    s = torch.empty(6, dtype=torch.float64, device=pos.device)
    check(lib().fpp_predict_mapped(gp._model.handle, structure.handle,
                                   PRECISIONS[precision], e.data_ptr(), f.data_ptr(),
                                   s.data_ptr(), None, 1, stream))
    structure.last_stress = s
    return e, f, s


class FlareEnergy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, positions, gp, structure, precision="mixed"):
        e, f, _ = _evaluate(positions, gp, structure, precision)
        ctx.save_for_backward(f)
        return e

    @staticmethod
    def backward(ctx, grad_e):
        (f,) = ctx.saved_tensors
        return -grad_e * f, None, None, None


def _plain(positions, n):
    """Whether the graph would accept these positions of n atoms and nothing watches it:
    an ordinary n x 3 FP64 CUDA tensor, gradients on, no anomaly detection (which raises
    for NaN forces in the backward pass), no tracing or compilation, no functorch
    transform, no saved-tensor hooks."""
    if (type(positions) is not torch.Tensor or positions.dtype != torch.float64
            or not positions.is_cuda or positions.shape != (n, 3)
            or positions.layout != torch.strided or positions.is_inference()):
        return False
    if (not torch.is_grad_enabled() or torch.is_anomaly_enabled() or torch.jit.is_tracing()
            or torch.compiler.is_compiling()):
        return False
    try:
        return not (torch._C._are_functorch_transforms_active()
                    or torch._C._autograd._top_saved_tensors_default_hooks(False) is not None)
    except (AttributeError, TypeError):  # another PyTorch: take the graph
        return False


def energy_forces_stress(gp, structure, positions, precision="mixed"):
    """Energy, forces and stress for device positions (detached; for an
    autograd-connected energy use FlareEnergy.apply).

    The forces are minus the gradient of FlareEnergy, which is what its forward
    computes: they are returned from there unless something watches the graph
    (a backward pass through the engine costs as much host time as the whole
    evaluation of a hundred atoms)."""
    if _plain(positions, structure.noa):
        return _evaluate(positions, gp, structure, precision)
    pos = positions.detach().requires_grad_(True)
    e = FlareEnergy.apply(pos, gp, structure, precision)
    (g,) = torch.autograd.grad(e, pos)
    return e.detach(), -g, structure.last_stress
