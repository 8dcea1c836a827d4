"""Generation-time ops: single-token attention over a KV cache, token sampling, whole decoding steps.

CUDA tensors run ``csrc/decode_kernels.cu``; CPU tensors the PyTorch statements
(``attention.decode_attention_reference`` and ``sample_reference`` below)."""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from .attention import decode_attention_reference

ll = ctypes.c_longlong


def decode_attention(q, k_cache, v_cache, kv_len, n_heads, pad_left=None, prefix_k=None, prefix_v=None,
                     scale=None):
    """q [B, d] against k_cache / v_cache [B, Lmax, d] (first ``kv_len`` rows valid) -> [B, d]."""
    if not q.is_cuda:
        return decode_attention_reference(q, k_cache, v_cache, kv_len, n_heads, pad_left, prefix_k, prefix_v, scale)
    B, d = q.shape
    hd = d // n_heads
    scale = scale if scale is not None else hd ** -0.5
    out = torch.empty((B, d), dtype=torch.bfloat16, device=q.device)
    npre = prefix_k.shape[0] if prefix_k is not None else 0
    assert q.stride(-1) == 1 and k_cache.stride(-1) == 1 and v_cache.stride(-1) == 1
    assert k_cache.stride() == v_cache.stride()
    # the kernel reads rows in 16-byte vectors: rows that start elsewhere are copied
    if (k_cache.data_ptr() | v_cache.data_ptr()) & 15:
        k_cache, v_cache = (t.clone(memory_format=torch.contiguous_format) for t in (k_cache, v_cache))
    if prefix_k is not None and (prefix_k.data_ptr() | prefix_v.data_ptr()) & 15:
        prefix_k, prefix_v = (t.clone(memory_format=torch.contiguous_format) for t in (prefix_k, prefix_v))
    rc = _lib.lib().dz_decode_attn(
        _lib.ptr(q), ll(q.stride(0)), _lib.ptr(k_cache), _lib.ptr(v_cache), ll(k_cache.stride(0)),
        ll(k_cache.stride(1)), _lib.ptr(prefix_k), _lib.ptr(prefix_v),
        ll(prefix_k.stride(0) if prefix_k is not None else 0), npre, _lib.ptr(pad_left), int(kv_len), B,
        n_heads, hd, ctypes.c_float(scale), _lib.ptr(out), ll(out.stride(0)), _lib.stream_ptr())
    _lib.check(rc, "dz_decode_attn")
    return out


def sample_reference(logits, temperature=1.0, top_k=None, top_p=None, do_sample=True, generator=None):
    from ..models.generate import filter_logits
    if not do_sample:
        return logits.argmax(dim=-1)
    probs = torch.softmax(filter_logits(logits.float(), temperature, top_k, top_p), dim=-1)
    return torch.multinomial(probs, 1, generator=generator).squeeze(1)


def sample(logits: torch.Tensor, temperature: float = 1.0, top_k: int | None = None,
           top_p: float | None = None, do_sample: bool = True, seed: int = 0, offset: int = 0) -> torch.Tensor:
    """One token id per row of fp32 ``logits`` [B, V] (int64).  ``offset`` distinguishes the
    draws of successive decoding steps under one ``seed``."""
    if not logits.is_cuda:
        g = torch.Generator().manual_seed((seed * 1000003 + offset) & (2 ** 63 - 1))
        return sample_reference(logits, temperature, top_k, top_p, do_sample, g)
    return sample_step(logits, temperature, top_k, top_p, do_sample, seed, offset).long()


def sample_step(logits: torch.Tensor, temperature: float = 1.0, top_k: int | None = None,
                top_p: float | None = None, do_sample: bool = True, seed: int = 0, offset: int = 0,
                done: torch.Tensor | None = None, eos: torch.Tensor | None = None, pad_id: int = 0) -> torch.Tensor:
    """The draws of :func:`sample` as int32 on the device.  With ``done`` (int32 [B]) finished rows give ``pad_id`` and
    rows that draw an id of ``eos`` (int32) are marked finished, all in the sampling kernel (CUDA only)."""
    assert logits.dtype == torch.float32 and logits.stride(-1) == 1
    B, V = logits.shape
    out = torch.empty(B, dtype=torch.int32, device=logits.device)
    rc = _lib.lib().dz_sample_step(
        _lib.ptr(logits), ll(logits.stride(0)), B, V, ctypes.c_float(temperature or 1.0), int(top_k or 0),
        ctypes.c_float(top_p if top_p is not None else 1.0), int(do_sample), ctypes.c_uint64(seed),
        ctypes.c_uint64(offset), _lib.ptr(done), _lib.ptr(eos), eos.numel() if eos is not None else 0, int(pad_id),
        _lib.ptr(out), _lib.stream_ptr())
    _lib.check(rc, "dz_sample_step")
    return out


# ---------------------------------------------------------------------------------- whole decoding steps
_LAYER_FIELDS = ("ln1_w", "ln1_b", "qkv_w", "qkv_b", "out_w", "out_b", "ln2_w", "ln2_b", "up_w", "up_b", "down_w",
                 "down_b", "prefix_k", "prefix_v")


class _Layer(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in _LAYER_FIELDS]


class _Config(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_int) for n in ("layers", "B", "d", "F", "H", "Hkv", "hd", "n_prefix", "rms", "pre_norm",
                                             "act", "rope_n_pos", "cache_rows")] +
                [("eps", ctypes.c_float), ("scale", ctypes.c_float)] +
                [(n, ctypes.c_longlong) for n in ("ld_prefix", "ld_seq", "ld_row")] +
                [(n, ctypes.c_void_p) for n in ("rope_cs", "h", "h2", "xn", "qkv", "ctx", "f", "err")])


MAX_STEP_ROWS = 64       # sequences a DecodePlan takes (the row limit of the skinny GEMM)


class DecodePlan:
    """All blocks of one decoding step as a single native call (``csrc/decode_step.cu``).

    ``layers``: per block a dict of the names in ``_LAYER_FIELDS`` -> bf16 CUDA tensor or None; the plan keeps them and
    its workspaces alive.  ``h`` [B, d] holds the embedded tokens before :meth:`step` and the last block's output after.
    The caches are bf16 [B, cache_rows, d] per layer; a step at or past ``cache_rows`` is refused."""

    def __init__(self, layers: list[dict], B: int, d: int, F: int, H: int, Hkv: int, act: int, rms: bool,
                 pre_norm: bool, eps: float, cache_rows: int, rope: torch.Tensor | None = None):
        self._handle = ctypes.c_void_p()
        self._free = _lib.lib().dz_decode_plan_free      # held here: module globals may be gone when the plan is
        dev = layers[0]["qkv_w"].device
        hd = d // H
        ws = lambda n: torch.empty((B, n), dtype=torch.bfloat16, device=dev)          # noqa: E731
        self.h, self._ws = ws(d), [ws(d), ws(d), ws((H + 2 * Hkv) * hd), ws(d), ws(F)]
        self._keep = (layers, rope)
        self._kernels = 7 * len(layers)
        self._cache_rows = cache_rows
        pk = layers[0].get("prefix_k")
        for w in layers:
            for n in _LAYER_FIELDS:
                x = w.get(n)
                assert x is None or (x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous()), n
        arr = (_Layer * len(layers))(*[_Layer(*[_lib.ptr(w.get(n)).value for n in _LAYER_FIELDS]) for w in layers])
        p = lambda t: _lib.ptr(t).value                                               # noqa: E731
        cfg = _Config(layers=len(layers), B=B, d=d, F=F, H=H, Hkv=Hkv, hd=hd, n_prefix=0 if pk is None else pk.shape[0],
                      rms=int(rms), pre_norm=int(pre_norm), act=act, rope_n_pos=0 if rope is None else rope.shape[0],
                      eps=eps, scale=hd ** -0.5, ld_prefix=0 if pk is None else pk.stride(0),
                      ld_seq=cache_rows * d, ld_row=d, cache_rows=cache_rows, rope_cs=p(rope), h=p(self.h),
                      h2=p(self._ws[0]), xn=p(self._ws[1]), qkv=p(self._ws[2]), ctx=p(self._ws[3]), f=p(self._ws[4]),
                      err=p(_lib.err_word(dev)))
        _lib.check(_lib.lib().dz_decode_plan_create(ctypes.byref(cfg), arr, ctypes.byref(self._handle)),
                   "dz_decode_plan_create")

    def caches(self, k: list[torch.Tensor], v: list[torch.Tensor]):
        """Pointer arrays of the per-layer caches for :meth:`step` (kept by the caller beside the tensors)."""
        n, shape = len(self._keep[0]), (self.h.shape[0], self._cache_rows, self.h.shape[1])
        assert len(k) == n == len(v)
        for t in (*k, *v):
            assert t.shape == shape and t.is_contiguous() and t.dtype == torch.bfloat16 and t.device == self.h.device
        return tuple((ctypes.c_void_p * n)(*[_lib.ptr(t).value for t in ts]) for ts in (k, v))

    def step(self, caches, t: int, pad_left: torch.Tensor) -> torch.Tensor:
        rc = _lib.lib().dz_decode_step(self._handle, caches[0], caches[1], int(t), _lib.ptr(pad_left),
                                       _lib.stream_ptr())
        _lib.check(rc, "dz_decode_step")
        _lib.launch_count += self._kernels - 1               # check() counted one
        return self.h

    def __del__(self):
        if getattr(self, "_handle", None):
            self._free(self._handle)
            self._handle = None
