"""Differentiable float32 SGM: the CUDA forward/backward kernels (csrc/float_sgm.cu) behind a
torch.autograd.Function, plus a plain-PyTorch restatement used by the tests as the autograd and
finite-difference reference.

    disp = float_sgm(cost, p1, p2, temperature=1.0)   # cost [B,H,W,D] float32 CUDA, p1/p2 [B,H,W]
"""
from __future__ import annotations

import ctypes as C
import functools

import torch

from . import load_library

_PATHS = ((1, False), (2, False), (1, True), (2, True))  # (scan dim, reversed): T->B, L->R, B->T, R->L


def _lib():
    lib = load_library()
    if not hasattr(lib, "_float_sgm_bound"):
        vp, i32, f32 = C.c_void_p, C.c_int32, C.c_float
        lib.sgm_float_checkpoint_elems.argtypes = [i32, i32, i32, i32]
        lib.sgm_float_checkpoint_elems.restype = C.c_size_t
        lib.sgm_float_workspace_elems.argtypes = [i32, i32, i32, i32]
        lib.sgm_float_workspace_elems.restype = C.c_size_t
        lib.sgm_float_forward.argtypes = [vp, vp, vp, i32, i32, i32, i32, f32, vp, vp, vp, vp, vp]
        lib.sgm_float_forward.restype = i32
        lib.sgm_float_disparity.argtypes = [vp, vp, vp, i32, i32, i32, i32, f32, vp, vp, vp, vp]
        lib.sgm_float_disparity.restype = i32
        lib.sgm_float_backward.argtypes = [vp, vp, vp, i32, i32, i32, i32, f32, vp, vp, vp, vp, vp, vp, vp, vp, vp]
        lib.sgm_float_backward.restype = i32
        lib._float_sgm_bound = True
    return lib


def _aligned(t):
    """the kernels read the cost volume with 16-byte vector loads"""
    return t if t.data_ptr() % 16 == 0 else t.clone()


@functools.lru_cache(maxsize=64)
def _elems(B, H, W, D):
    """(volume, records, workspace) sizes in floats, each a multiple of 16 bytes"""
    lib = _lib()
    return B * H * W * D, lib.sgm_float_checkpoint_elems(B, H, W, D), lib.sgm_float_workspace_elems(B, H, W, D)


def _check(lib, status, what):
    if status != 0:
        raise RuntimeError(f"float SGM {what} failed: {lib.sgm_last_error(None).decode()}")


class FloatSGM(torch.autograd.Function):
    # A 64x48 crop's forward and backward are ~40 us of kernels: the host's share is kept small with
    # one allocation for what the backward pass needs and one for each pass's scratch.
    @staticmethod
    def forward(ctx, cost, p1, p2, temperature=1.0, grad_enabled=True):
        if not (cost.is_cuda and cost.dtype == torch.float32 and cost.dim() == 4):
            raise ValueError("cost must be a float32 CUDA tensor [B,H,W,D]")
        B, H, W, D = cost.shape
        dev, n = cost.device, B * H * W
        # the kernels read, and write the gradients of, one penalty a pixel
        if not (p1.numel() == n == p2.numel() and p1.device == dev == p2.device):
            raise ValueError(f"p1 and p2 must be [{B}, {H}, {W}] on {dev} (got {list(p1.shape)} on {p1.device}, "
                             f"{list(p2.shape)} on {p2.device})")
        cost, p1, p2 = _aligned(cost.contiguous()), p1.contiguous().float(), p2.contiguous().float()
        lib = _lib()
        vol, rec, scratch = _elems(B, H, W, D)
        temperature = float(temperature)
        keep = grad_enabled and any(ctx.needs_input_grad)  # else no backward pass: nothing is kept for it
        kept = cost.new_empty(vol + rec if keep else vol)  # S, then the records
        work, disp = cost.new_empty(scratch), cost.new_empty(B, H, W)
        sum_, stream = kept.data_ptr(), torch.cuda.current_stream(dev).cuda_stream
        if not keep:
            _check(lib, lib.sgm_float_disparity(cost.data_ptr(), p1.data_ptr(), p2.data_ptr(), B, H, W, D, temperature,
                                                sum_, work.data_ptr(), disp.data_ptr(), stream), "forward")
            return disp
        _check(lib, lib.sgm_float_forward(cost.data_ptr(), p1.data_ptr(), p2.data_ptr(), B, H, W, D, temperature,
                                          sum_, sum_ + 4 * vol, work.data_ptr(), disp.data_ptr(), stream), "forward")
        ctx.save_for_backward(kept)
        ctx.sizes, ctx.maps, ctx.temperature = (B, H, W, D), (p1.shape, p2.shape), temperature
        return disp

    @staticmethod
    def backward(ctx, grad_disp):
        (kept,) = ctx.saved_tensors  # S and the records: the inputs are not needed again
        B, H, W, D = ctx.sizes
        lib = _lib()
        vol, _, scratch = _elems(B, H, W, D)
        g = grad_disp.contiguous().float()
        work = kept.new_empty(vol + scratch)  # gradient of S, workspace
        gcost, gp1, gp2 = kept.new_empty(B, H, W, D), torch.empty_like(g), torch.empty_like(g)
        sum_, gsum = kept.data_ptr(), work.data_ptr()
        # S in the place of the inputs, which the call asks for and does not read
        _check(lib, lib.sgm_float_backward(sum_, sum_, sum_, B, H, W, D, ctx.temperature, sum_, sum_ + 4 * vol,
                                           g.data_ptr(), gsum, gsum + 4 * vol, gcost.data_ptr(), gp1.data_ptr(),
                                           gp2.data_ptr(), torch.cuda.current_stream(kept.device).cuda_stream),
               "backward")
        if ctx.maps != (g.shape, g.shape):  # maps of another shape with as many values
            gp1, gp2 = gp1.view(ctx.maps[0]), gp2.view(ctx.maps[1])
        return gcost, gp1, gp2, None, None


def float_sgm(cost, p1, p2, temperature: float = 1.0):
    return FloatSGM.apply(cost, p1, p2, temperature, torch.is_grad_enabled())


def reference_sgm(cost, p1, p2, temperature: float = 1.0, return_sum: bool = False):
    """The same function in plain PyTorch ops (any device / dtype; differentiable by autograd)."""
    B, H, W, D = cost.shape
    inf = torch.full(cost.shape[:-1] + (1,), float("inf"), dtype=cost.dtype, device=cost.device)
    total = 0
    for dim, rev in _PATHS:
        n = cost.shape[dim]
        idx = range(n - 1, -1, -1) if rev else range(n)
        outs = [None] * n
        L = None
        for s, k in enumerate(idx):
            c = cost.select(dim, k)
            if s == 0:
                L = c
            else:
                P1 = p1.select(dim, k).unsqueeze(-1)
                P2 = p2.select(dim, k).unsqueeze(-1)
                m = L.min(-1, keepdim=True).values
                ninf = inf.select(dim, 0)
                lm = torch.cat([ninf, L[..., :-1]], -1) + P1
                lp = torch.cat([L[..., 1:], ninf], -1) + P1
                t = torch.minimum(torch.minimum(torch.minimum(L, lm), lp), m + P2)
                L = c + t - m
            outs[k] = L
        total = total + torch.stack(outs, dim)
    w = torch.softmax(-total / temperature, dim=-1)
    d = torch.arange(D, dtype=cost.dtype, device=cost.device)
    disp = (w * d).sum(-1)
    return (disp, total) if return_sum else disp
