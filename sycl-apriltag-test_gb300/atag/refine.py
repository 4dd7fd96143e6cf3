"""Subpixel corner refinement with a hand-written adjoint (CUDA), exposed as a
torch.autograd.Function.  The forward model is documented in
include/atag.h (atag_refine_forward) and csrc/k_refine.cu."""
import ctypes

import torch

from . import lib

_P = ctypes.c_void_p
SAMPLES_PER_EDGE = 64


def _ptr(t):
    return _P(t.data_ptr()) if t is not None else None


def _stream():
    return _P(lib.current_stream())


def _forward(image, corners, want_samples):
    L = lib.init()
    image = image.contiguous()
    corners = corners.contiguous()
    q = corners.shape[0]
    refined = torch.empty_like(corners)
    residual = torch.empty((q, 4), dtype=torch.float32, device=corners.device)
    samples = torch.empty((q, 4, SAMPLES_PER_EDGE), dtype=torch.float32, device=corners.device) if want_samples else None
    lib.check(L.atag_refine_forward(_ptr(image), image.shape[1], image.shape[0], _ptr(corners), q, _ptr(refined),
                                    _ptr(residual), _ptr(samples), _stream()), "atag_refine_forward")
    return refined, residual, samples


def refine_forward(image: torch.Tensor, corners: torch.Tensor):
    """image: H x W float32 (CUDA); corners: Q x 4 x 2 float32.  Returns
    (refined Q x 4 x 2, residual Q x 4, samples Q x 4 x 64)."""
    return _forward(image, corners, True)


def _backward(image, corners, grad_refined, grad_residual, want_image_grad, want_samples_grad):
    L = lib.init()
    image = image.contiguous()
    corners = corners.contiguous()
    q = corners.shape[0]
    g_c = torch.empty_like(corners)
    g_s = torch.empty((q, 4, SAMPLES_PER_EDGE), dtype=torch.float32, device=corners.device) if want_samples_grad else None
    g_i = torch.zeros_like(image) if want_image_grad else None
    gr = grad_refined.contiguous() if grad_refined is not None else None
    gres = grad_residual.contiguous() if grad_residual is not None else None
    lib.check(L.atag_refine_backward(_ptr(image), image.shape[1], image.shape[0], _ptr(corners), q, _ptr(gr),
                                     _ptr(gres), _ptr(g_c), _ptr(g_s), _ptr(g_i), _stream()), "atag_refine_backward")
    return g_c, g_s, g_i


def refine_backward(image, corners, grad_refined=None, grad_residual=None, want_image_grad=False):
    """Returns (dL/dcorners Q x 4 x 2, dL/dsamples Q x 4 x 64, dL/dimage or None)."""
    return _backward(image, corners, grad_refined, grad_residual, want_image_grad, True)


class RefineCorners(torch.autograd.Function):
    """refined, residual = RefineCorners.apply(image, corners)"""

    @staticmethod
    def forward(ctx, image, corners):
        # the samples and their gradient (1 KB each per quad) are not asked for
        refined, residual, _ = _forward(image.detach(), corners.detach(), False)
        ctx.save_for_backward(image, corners)
        return refined, residual

    @staticmethod
    def backward(ctx, grad_refined, grad_residual):
        image, corners = ctx.saved_tensors
        g_c, _, g_i = _backward(image.detach(), corners.detach(), grad_refined, grad_residual,
                                ctx.needs_input_grad[0], False)
        return (g_i if ctx.needs_input_grad[0] else None), (g_c if ctx.needs_input_grad[1] else None)


def refine(image, corners):
    return RefineCorners.apply(image, corners)
