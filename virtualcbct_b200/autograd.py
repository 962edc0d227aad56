"""Differentiable polychromatic projection for material decomposition.

``project(volumes, projector)`` maps six float element volumes (densities x
1000, layout [Z][nmat][N][N], CUDA float32) to the spectral projections
[V][H][W] through the CUDA forward kernel; its backward is the hand-written
adjoint kernel, which recomputes each ray's spectral state (the per-energy
attenuation and its derivative) instead of storing it.  The six per-ray
element path integrals it is recomputed from are either kept from the
forward launch (``vcbct_projector_forward_state`` / ``_adjoint_state``, 24 B
per ray) or re-marched (``vcbct_projector_adjoint``) when keeping them would
exceed ``keep_limit`` bytes.  No reference counterpart: the reference's
nearest analogue is the unused sensitivity backprojection of
Release_CBCT_Projection_CM/lengthproj.cpp:10-131.
"""
from __future__ import annotations

import torch

from .projector import Projector, _volume_key


# Bytes of per-ray path integrals kept between the passes; None: keep them
# when they take at most a quarter of the device's free memory (11 GB for 720
# views of 800 x 800 is kept on a 180 GB GPU).
KEEP_LIMIT = None
# Asking the driver for the free memory takes 69 us to several ms on a shared
# node, a fifth of a small step or more (56x56x9, 36 views of 30 x 46: 347 us,
# 240 without).  It is not asked for path integrals below this share of the
# device's memory (22 MB of 180 GB, about the unit of 20 MB in which torch takes
# device memory), nor where torch already holds the memory of the whole step
# free, as from the second step of a loop on (looking that up takes 11 us, 3 to
# 7 % of steps of 0.4 ms: hence the share).
SMALL_SHARE = 1 << 13


def _held_free() -> int:
    """Bytes that torch's allocator holds free on the current device."""
    s = torch.cuda.memory_stats_as_nested_dict()
    now = [s.get(k, {}).get("all", {}).get("current", 0) for k in ("reserved_bytes", "allocated_bytes")]
    return now[0] - now[1]


def _keep(nbytes: int, keep_limit, rest: int = 0) -> bool:
    """Whether to keep ``nbytes`` of path integrals; ``rest``: bytes that the
    step allocates after them."""
    if keep_limit is None:
        if nbytes <= torch.cuda.get_device_properties(torch.cuda.current_device()).total_memory // SMALL_SHARE:
            return True
        if nbytes + rest <= _held_free():
            return True
        free, _ = torch.cuda.mem_get_info()
        return nbytes <= free // 4
    return nbytes <= keep_limit


class _MbfpaProject(torch.autograd.Function):
    @staticmethod
    def forward(ctx, volumes: torch.Tensor, projector: Projector, keep_limit):
        if not volumes.is_cuda or volumes.dtype != torch.float32:
            raise TypeError("volumes must be a CUDA float32 tensor [Z][nmat][N][N]")
        vol = volumes.detach().contiguous()
        projector.load_volume_f32(vol)
        g = projector.geom
        out = torch.empty((g.V, g.H, g.W), dtype=torch.float32, device="cuda")
        L = None
        # after them: the gradient, and a residual and its square of the projections' size
        if _keep(g.V * g.H * g.W * g.nmat * 4, keep_limit, 4 * vol.numel() + 2 * 4 * out.numel()):
            try:
                L = torch.empty((g.V, g.H, g.W, g.nmat), dtype=torch.float32, device="cuda")
            except torch.OutOfMemoryError:
                pass
        if L is not None:
            projector.forward_state(out, L)
            ctx.save_for_backward(vol, L)
        else:
            projector.forward(out)
            ctx.save_for_backward(vol)
        ctx.projector = projector
        return out

    @staticmethod
    def backward(ctx, grad_out: torch.Tensor):
        saved = ctx.saved_tensors
        vol = saved[0]
        p: Projector = ctx.projector
        # the adjoint reads the float volume the forward used: reload it only
        # if the projector has been given another volume since
        if p.loaded != _volume_key("f32", vol):
            p.load_volume_f32(vol)
        grad = torch.zeros_like(vol)
        go = grad_out.contiguous().float()
        if len(saved) > 1:
            p.adjoint_state(saved[1], go, grad)
        else:
            p.adjoint(go, grad)
        return grad, None, None


def project(volumes: torch.Tensor, projector: Projector, keep_limit=KEEP_LIMIT) -> torch.Tensor:
    """Differentiable spectral forward projection of float element volumes.
    The per-ray path integrals are kept for the backward pass when they fit
    in ``keep_limit`` bytes (0: always re-march; None: in a quarter of the free
    device memory, or together with the rest of the step in memory that torch
    already holds)."""
    return _MbfpaProject.apply(volumes, projector, keep_limit)


def decomposition_step(volumes: torch.Tensor, target: torch.Tensor, projector: Projector,
                       lr: float = 0.0, keep_limit=KEEP_LIMIT):
    """One gradient step of least-squares material decomposition:
    loss = 0.5 * sum (project(volumes) - target)^2.  Returns (loss, grad) and,
    when lr > 0, updates ``volumes`` in place (clamped at zero)."""
    v = volumes.detach().requires_grad_(True)
    pred = project(v, projector, keep_limit)
    loss = 0.5 * torch.sum((pred - target) ** 2)
    (grad,) = torch.autograd.grad(loss, v)
    if lr > 0.0:
        with torch.no_grad():
            volumes.sub_(lr * grad).clamp_(min=0.0)
    return loss.detach(), grad
