"""Host side of decoding: the caches of a run."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from dizo_b200.models.generate import _Decoder, _PPDecoder, _TPDecoder
from dizo_b200.models.opt import OPTConfig, OPTModel
from dizo_b200.ops import _lib


def test_each_cache_owns_its_memory():
    """Reordering beams replaces the caches one by one: what is replaced can go back at once only if no other cache is a
    view of the same allocation."""
    m = OPTModel(OPTConfig(vocab_size=60, hidden_size=32, num_hidden_layers=3, ffn_dim=64, num_attention_heads=2,
                           max_position_embeddings=64), "cpu", torch.float32)
    dec = _Decoder(m, 4, 10)
    for _ in range(2):
        tensors = dec.k + dec.v
        assert len({t.untyped_storage().data_ptr() for t in tensors}) == len(tensors) == 6
        assert all(t.untyped_storage().nbytes() == 4 * 10 * 32 * 4 for t in tensors)
        dec.reorder(torch.tensor([1, 0, 3, 3]))


@pytest.mark.parametrize("cls", [_Decoder, _TPDecoder, _PPDecoder])
def test_every_decoder_reorders_its_caches(cls):
    m = SimpleNamespace(config=SimpleNamespace(hidden_size=16, num_hidden_layers=2), device=torch.device("cpu"),
                        dtype=torch.float32, tp=2, lo=0, hi=2)
    dec = cls(m, 3, 5)
    for i, t in enumerate(dec.k + dec.v):
        t.copy_(torch.arange(3.0).view(3, 1, 1) + 10 * i)
    dec.reorder(torch.tensor([2, 0]))
    for i, t in enumerate(dec.k + dec.v):
        assert t.shape[:2] == (2, 5) and t[:, 0, 0].tolist() == [10 * i + 2, 10 * i]


@pytest.mark.skipif(not _lib.available() or torch.cuda.is_available(), reason="host checks alone: library built, no GPU")
@pytest.mark.parametrize("which", range(4))
def test_decode_attention_refuses_rows_off_a_16_byte_boundary(which):
    """Keys, values and prefix rows are read in 16-byte vectors: the entry point says so before anything is launched."""
    rows = [4096 * (i + 2) for i in range(4)]                    # addresses that are never followed
    rows[which] += 8
    kc, vc, pk, pv = (ctypes.c_void_p(r) for r in rows)
    ll = ctypes.c_longlong
    rc = _lib.lib().dz_decode_attn(ctypes.c_void_p(4096), ll(64), kc, vc, ll(640), ll(64), pk, pv, ll(64), 2, None, 8, 1, 1,
                                   64, ctypes.c_float(1.0), ctypes.c_void_p(4096), ll(64), None)
    assert rc == 2
