"""Whole blocks as one native call: the same kernels on the same operands as ``_layer_forward``, so the same bits."""
import pytest
import torch

from dizo_b200.data.synthetic import synthetic_batch
from dizo_b200.models.llama import LlamaConfig, LlamaModel
from dizo_b200.models.opt import OPTConfig, OPTModel, Transform
from dizo_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _model(pre: bool, mode: str = "full", d: int = 256) -> OPTModel:
    cfg = OPTConfig(vocab_size=520, hidden_size=d, num_hidden_layers=3, ffn_dim=520, num_attention_heads=4,
                    max_position_embeddings=160, do_layer_norm_before=pre, word_embed_proj_dim=d if pre else 64)
    return OPTModel(cfg, "cuda", torch.bfloat16, mode=mode).init_random_fast(5, std=0.05)


@pytest.mark.parametrize("pre", [True, False])
@pytest.mark.parametrize("mode,d", [("full", 256), ("full", 192), ("head", 256)])      # d 192: q | k | v biases not adjacent
@pytest.mark.parametrize("B,L", [(1, 9), (3, 130)])
def test_native_blocks_equal_layer_forward(pre, mode, d, B, L, monkeypatch):
    m = _model(pre, mode, d)
    b = synthetic_batch(1, B, L, 520, cand_ids=(9, 372)).to("cuda")
    b.pad_left = torch.arange(B, dtype=torch.int32, device="cuda")
    alpha = torch.full((max(len(m.dizo_include_names()), 1),), 0.7, device="cuda")

    def results():
        out = [m.hidden_states(b), m.hidden_states(b, Transform(seed=3, coef=1e-2), rows=b.rows), *m.loss_pair(b, 7, 1e-2)]
        if mode == "full":
            out.append(m.hidden_states(b, Transform(alpha=alpha)))        # stages q | k | v only
        _lib.check_device_errors()
        return out

    if mode == "full":
        m.arena.set_dizo(m.dizo_include_names())
        m.arena.sweep(seed1=9, c1=0.05)
    if d != 192:
        assert m._block_weights(0, None, 0, True) is not None
    native = results()
    monkeypatch.setattr(OPTModel, "_block_runner", lambda self, batch: None)
    for x, y in zip(native, results()):
        assert torch.equal(x, y)


@pytest.mark.parametrize("heads,kv,d", [(4, 2, 512), (8, 8, 256)])          # head dims 128 and 32
@pytest.mark.parametrize("mode", ["full", "head"])
@pytest.mark.parametrize("B,L", [(1, 9), (3, 130), (16, 200)])
def test_native_llama_blocks_equal_layer_forward(heads, kv, d, mode, B, L, monkeypatch):
    cfg = LlamaConfig(vocab_size=520, hidden_size=d, num_hidden_layers=3, intermediate_size=712, num_attention_heads=heads,
                      num_key_value_heads=kv, max_position_embeddings=256)
    m = LlamaModel(cfg, "cuda", torch.bfloat16, mode=mode).init_random_fast(5, std=0.05)
    b = synthetic_batch(1, B, L, 520, cand_ids=(9, 372)).to("cuda")
    b.pad_left = torch.arange(B, dtype=torch.int32, device="cuda") % 5
    assert m._block_runner(b) is not None and m._block_weights(0, None, 0, True) is not None

    def results():
        out = [m.hidden_states(b), m.hidden_states(b, Transform(seed=3, coef=1e-2), rows=b.rows), *m.loss_pair(b, 7, 1e-2)]
        _lib.check_device_errors()
        return out

    native = results()
    monkeypatch.setattr(LlamaModel, "_block_runner", lambda self, batch: None)
    for x, y in zip(native, results()):
        assert torch.equal(x, y)


def test_native_block_does_not_overwrite_its_input():
    m = _model(True)
    b = synthetic_batch(2, 2, 40, 520, cand_ids=(9, 372)).to("cuda")
    r = m._block_runner(b)
    h = torch.randn(2, 40, 256, device="cuda").bfloat16()
    keep = h.clone()
    ptrs = m._block_weights(1, None, 0, True)
    y = r.run(h, ptrs)
    assert torch.equal(h, keep)
    z = r.run(h, ptrs, out=h)
    assert z.data_ptr() == h.data_ptr() and torch.equal(z, y)


@pytest.mark.parametrize("family", ["opt", "opt-post", "llama"])
@pytest.mark.parametrize("B,L", [(1, 9), (3, 40)])           # the last block's tail has 1 and 3 rows: register products
def test_staged_weights_in_a_chain_equal_a_synchronised_one(family, B, L, monkeypatch):
    """Every block reads weights that the sweep in front of it has just written into a reused buffer.  A chain of dependent
    launches gives the bits of the same kernels with the device idle before each of them."""
    if family == "llama":
        m = LlamaModel(LlamaConfig(vocab_size=520, hidden_size=256, num_hidden_layers=6, intermediate_size=712,
                                   num_attention_heads=4, num_key_value_heads=2, max_position_embeddings=256), "cuda",
                       torch.bfloat16).init_random_fast(5, std=0.05)
    else:
        m = OPTModel(OPTConfig(vocab_size=520, hidden_size=256, num_hidden_layers=6, ffn_dim=520, num_attention_heads=4,
                               max_position_embeddings=160, do_layer_norm_before=family == "opt",
                               word_embed_proj_dim=256 if family == "opt" else 64), "cuda",
                     torch.bfloat16).init_random_fast(5, std=0.05)
    b = synthetic_batch(1, B, L, 520, cand_ids=(9, 372)).to("cuda")

    def results():
        out = []
        for seed in range(4):
            out += [*m.loss_pair(b, seed, 0.3), m.hidden_states(b, Transform(seed=seed, coef=0.3), rows=b.rows)]
        _lib.check_device_errors()
        return out

    chained = results()
    check = _lib.check

    def waiting(rc, name):
        torch.cuda.synchronize()
        check(rc, name)

    monkeypatch.setattr(_lib, "check", waiting)
    monkeypatch.setattr(type(m), "_block_runner", lambda self, batch: None)       # one Python call a kernel
    for x, y in zip(chained, results()):
        assert torch.equal(x, y)
