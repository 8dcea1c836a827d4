"""A whole decoder block as one native call (``csrc/block_forward.cu``): the host cost of a block is one call instead of
seven or more.  The same kernels run in the same order on the same operands as in ``OPTModel._layer_forward`` and
``LlamaModel._layer_forward``."""
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


LLAMA_WEIGHTS = ("ln1_w", "qkv_w", "out_w", "ln2_w", "gu_w", "down_w")


class _LlamaBlock(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_int) for n in ("B", "L", "d", "F", "H", "Hkv", "pos0", "n_pos")] +
                [("eps", ctypes.c_float), ("scale", ctypes.c_float)] +
                [(n, ctypes.c_void_p) for n in LLAMA_WEIGHTS] +
                [(n, ctypes.c_void_p) for n in ("h_in", "h_out", "h_mid", "xn", "qkv", "ctx", "f", "raw", "rope_cs",
                                                "pad_left", "err")] +
                [("fused_rope", ctypes.c_int), ("fused_swiglu", ctypes.c_int)])


class _Runner:
    """Workspaces and constant arguments of the blocks of one forward (B sequences of L tokens, bf16 CUDA)."""

    weights: tuple
    entry: str

    def _workspaces(self, B: int, L: int, d: int, sizes, pad_left: torch.Tensor | None, device) -> dict:
        M = B * L
        self.shape = (B, L, d)
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
        return dict(B=B, L=L, d=d, pad_left=_lib.ptr(pad_left).value, err=_lib.ptr(self._err).value,
                    **{n: base + 2 * o for n, o in offs.items()})

    def run(self, h: torch.Tensor, weights, out: torch.Tensor | None = None) -> torch.Tensor:
        """h [B, L, d] -> the block's output, into ``out`` (which may be ``h``).  ``weights``: addresses in the order of
        ``self.weights``."""
        assert h.is_contiguous() and h.dtype == torch.bfloat16
        if out is None:
            out = torch.empty(self.shape, dtype=torch.bfloat16, device=h.device)
        a = self.args
        for n, p in zip(self.weights, weights):
            setattr(a, n, p)
        a.h_in, a.h_out = _lib.ptr(h).value, _lib.ptr(out).value
        rc = getattr(_lib.lib(), self.entry)(ctypes.byref(a), _lib.stream_ptr())
        _lib.check(rc, self.entry)
        _lib.launch_count += self.kernels - 1                # check() counted one
        return out


class BlockRunner(_Runner):
    """OPT blocks."""

    weights, entry, kernels = WEIGHTS, "dz_opt_block", 7

    def __init__(self, B: int, L: int, d: int, F: int, H: int, pre_norm: bool, act: int, eps: float,
                 pad_left: torch.Tensor | None, device):
        ws = self._workspaces(B, L, d, (("h_mid", d), ("xn", d), ("qkv", 3 * d), ("ctx", d), ("f", F)), pad_left, device)
        self.args = _Block(F=F, H=H, pre_norm=int(pre_norm), act=act, eps=eps, scale=(d // H) ** -0.5, **ws)


class LlamaBlockRunner(_Runner):
    """LLaMA-family blocks; ``rope``: the (cos, sin) table, row m at position ``pos0 + m % L``."""

    weights, entry = LLAMA_WEIGHTS, "dz_llama_block"

    def __init__(self, B: int, L: int, d: int, F: int, H: int, Hkv: int, eps: float, pos0: int, rope: torch.Tensor,
                 pad_left: torch.Tensor | None, device, fused_rope: bool = True, fused_swiglu: bool = True):
        hd = d // H
        fused = _lib.lib().dz_llama_block_fused(B * L, H, Hkv, hd, F, int(fused_rope), int(fused_swiglu))
        sizes = [("h_mid", d), ("xn", d), ("qkv", 3 * d), ("ctx", d), ("f", F)]
        raw = max(0 if fused & 1 else (H + 2 * Hkv) * hd, 0 if fused & 2 else 2 * F)
        if raw:
            sizes.append(("raw", raw))
        ws = self._workspaces(B, L, d, sizes, pad_left, device)
        self._rope = rope
        self.kernels = 7 + (not fused & 1) + (not fused & 2)
        self.args = _LlamaBlock(F=F, H=H, Hkv=Hkv, pos0=pos0, n_pos=rope.shape[0], eps=eps, scale=hd ** -0.5,
                                rope_cs=_lib.ptr(rope).value, fused_rope=int(fused_rope), fused_swiglu=int(fused_swiglu),
                                **ws)
