"""A whole OPT decoder block as one native call (``csrc/block_forward.cu``): the host cost of a block is one call instead of
seven.  The same kernels run in the same order on the same operands as in ``OPTModel._layer_forward``."""
from __future__ import annotations

import ctypes

import torch

from . import _lib

WEIGHTS = ("ln1_w", "ln1_b", "qkv_w", "qkv_b", "out_w", "out_b", "ln2_w", "ln2_b", "fc1_w", "fc1_b", "fc2_w", "fc2_b")


class _Block(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_int) for n in ("B", "L", "d", "F", "H", "pre_norm", "act", "pad_")] +
                [("eps", ctypes.c_float), ("scale", ctypes.c_float)] +
                [(n, ctypes.c_void_p) for n in WEIGHTS] +
                [(n, ctypes.c_void_p) for n in ("h_in", "h_out", "h_mid", "xn", "qkv", "ctx", "f", "pad_left", "err")])


class BlockRunner:
    """Workspaces and constant arguments of the blocks of one forward (B sequences of L tokens, bf16 CUDA)."""

    def __init__(self, B: int, L: int, d: int, F: int, H: int, pre_norm: bool, act: int, eps: float,
                 pad_left: torch.Tensor | None, device):
        M = B * L
        self.shape = (B, L, d)
        sizes = (("h_mid", d), ("xn", d), ("qkv", 3 * d), ("ctx", d), ("f", F))
        # 256-element steps keep every workspace as aligned as an allocation of its own
        offs, total = {}, 0
        for n, w in sizes:
            offs[n] = total
            total += (M * w + 255) // 256 * 256
        self._ws = torch.empty(total, dtype=torch.bfloat16, device=device)
        self._pad = pad_left
        self._err = _lib.err_word(device)
        if pad_left is not None:
            assert pad_left.dtype == torch.int32 and pad_left.is_cuda and pad_left.is_contiguous()
        base = _lib.ptr(self._ws).value
        self.args = _Block(B=B, L=L, d=d, F=F, H=H, pre_norm=int(pre_norm), act=act, eps=eps, scale=(d // H) ** -0.5,
                           pad_left=_lib.ptr(pad_left).value, err=_lib.ptr(self._err).value,
                           **{n: base + 2 * o for n, o in offs.items()})

    def run(self, h: torch.Tensor, weights, out: torch.Tensor | None = None) -> torch.Tensor:
        """h [B, L, d] -> the block's output, into ``out`` (which may be ``h``).  ``weights``: addresses in the order of
        ``WEIGHTS``."""
        assert h.is_contiguous() and h.dtype == torch.bfloat16
        if out is None:
            out = torch.empty(self.shape, dtype=torch.bfloat16, device=h.device)
        a = self.args
        for n, p in zip(WEIGHTS, weights):
            setattr(a, n, p)
        a.h_in, a.h_out = _lib.ptr(h).value, _lib.ptr(out).value
        rc = _lib.lib().dz_opt_block(ctypes.byref(a), _lib.stream_ptr())
        _lib.check(rc, "dz_opt_block")
        _lib.launch_count += 6                               # seven kernels; check() counted one
        return out
