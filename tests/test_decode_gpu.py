"""Decoding kernels: native decoding steps against the block-by-block path, the sampler's two forms."""
import math

import numpy as np
import pytest
import torch

from dizo_b200.models.generate import _Decoder, generate
from dizo_b200.models.llama import LlamaConfig, LlamaModel
from dizo_b200.models.opt import OPTConfig, OPTModel, make_batch
from dizo_b200.ops import _lib, philox
from dizo_b200.ops import decode as decode_ops
from dizo_b200.ops import llama as llama_ops
from dizo_b200.ops.attention import decode_attention_reference

pytestmark = pytest.mark.gpu


def _models(**kw):
    opt = dict(vocab_size=520, hidden_size=160, num_hidden_layers=3, ffn_dim=328, max_position_embeddings=256) | kw
    lla = dict(vocab_size=520, hidden_size=512, num_hidden_layers=2, intermediate_size=712, max_position_embeddings=256) | kw
    return {
        "opt": lambda: OPTModel(OPTConfig(num_attention_heads=2, **opt), "cuda", torch.bfloat16),
        "opt-post": lambda: OPTModel(OPTConfig(num_attention_heads=10, do_layer_norm_before=False, word_embed_proj_dim=64,
                                               **opt), "cuda", torch.bfloat16),
        "opt-adapters": lambda: OPTModel(OPTConfig(num_attention_heads=2, **opt), "cuda", torch.bfloat16,
                                         mode="lora+prefix"),
        "llama": lambda: LlamaModel(LlamaConfig(num_attention_heads=4, num_key_value_heads=2, **lla), "cuda",
                                    torch.bfloat16),
        "llama-prefix": lambda: LlamaModel(LlamaConfig(num_attention_heads=16, num_key_value_heads=16, **lla), "cuda",
                                           torch.bfloat16, mode="prefix"),
    }


@pytest.mark.parametrize("name", ["opt", "opt-post", "opt-adapters", "llama", "llama-prefix"])
@pytest.mark.parametrize("B,L", [(1, 3), (5, 130), (40, 17)])
def test_native_step_equals_block_by_block(name, B, L):
    m = _models()[name]().init_random_fast(3, std=0.05)
    for n in m.trainable_names:
        if "lora_B" in n:
            m.param(n).normal_(0, 0.05)
    g = torch.Generator().manual_seed(B * L)
    ids = torch.randint(4, 500, (B, L), generator=g)
    mask = torch.ones_like(ids)
    for i in range(1, B):
        mask[i, :min(i, L - 1)] = 0
    batch = make_batch(ids, mask).to("cuda")
    decs = [_Decoder(m, B, L + 8) for _ in range(2)]
    assert decs[0].native
    decs[1].native = False
    first = [d.prefill(batch) for d in decs]
    assert torch.equal(first[0], first[1])
    pos = (mask.sum(1).cuda() + 2).to(torch.int32)
    for t in range(3):
        tok = torch.full((B,), 7 + t, dtype=torch.int32, device="cuda")
        a, b = (d.step(tok, pos + t, batch.pad_left) for d in decs)
        _lib.check_device_errors()
        # the same operands in another order of fp32 sums: the newest key comes from registers instead of the cache, a step of
        # up to four sequences takes its products (LLaMA's SwiGLU among them) through gemv.cu, others split K differently
        assert ((a - b).norm() / b.norm()).item() < 2 * 2.0 ** -8
        for x, y in zip(decs[0].k + decs[0].v, decs[1].k + decs[1].v):
            x, y = x[:, :L + t + 1].float(), y[:, :L + t + 1].float()
            assert ((x - y).norm() / y.norm()).item() < 2 * 2.0 ** -8
    index = torch.arange(B - 1, -1, -1, device="cuda")
    for d in decs:
        d.reorder(index)
    a, b = (d.step(tok, pos + 3, batch.pad_left[index]) for d in decs)
    assert ((a - b).norm() / b.norm()).item() < 2 * 2.0 ** -8


@pytest.mark.parametrize("name", ["opt", "opt-adapters", "llama", "llama-prefix"])
@pytest.mark.parametrize("B,L", [(1, 600), (2, 330), (3, 330), (4, 700), (7, 301), (64, 70)])
def test_step_attends_to_all_keys(name, B, L):
    """The attention inside a step (cache append, keys shared by up to 8 CTAs, products for 1 to 4 rows in registers) against
    the fp32 statement over the cache it leaves, with padding longer than one CTA's share."""
    m = _models(num_hidden_layers=1, max_position_embeddings=1024)[name]().init_random_fast(3, std=0.2)
    cfg, P = m.config, m.num_prefix
    d, H = cfg.hidden_size, cfg.num_attention_heads
    mask = torch.ones(B, L, dtype=torch.long)
    for i in range(B):
        mask[i, :i * L // (B + 1)] = 0
    batch = make_batch(torch.randint(4, 500, (B, L), generator=torch.Generator().manual_seed(B * L)), mask).to("cuda")
    dec = _Decoder(m, B, L + 3)
    dec.prefill(batch)
    pos = (mask.sum(1).cuda() + 2).to(torch.int32)
    for t in range(L, L + 2):
        dec.step(torch.arange(B, device="cuda", dtype=torch.int32) + t, pos + t - L, batch.pad_left)
        _lib.check_device_errors()
        _, _, qkv, ctx, _ = (w.float().cpu() for w in dec.plan._ws)
        if isinstance(m, LlamaModel):
            qkv = llama_ops.rope_qkv_reference(qkv, 1, P + t, H, cfg.num_key_value_heads, d // H, cfg.rope_theta)
            qkv = qkv.bfloat16().float()
        k, v = dec.k[0].float().cpu(), dec.v[0].float().cpu()
        # a rotated value may fall on the other side of a rounding to bf16 (2^-7 of it at most); v and unrotated k are copies
        tol = 2.0 ** -7 if isinstance(m, LlamaModel) else 0.0
        assert ((k[:, t] - qkv[:, d:2 * d]).abs() <= tol * k[:, t].abs() + tol * 1e-3).all()
        assert torch.equal(v[:, t], qkv[:, 2 * d:])
        w = m._layer_weights(0, m._resolver(0, None, None, 0))
        pk, pv = (None, None) if w.prefix_k is None else (w.prefix_k.float().cpu(), w.prefix_v.float().cpu())
        ref = decode_attention_reference(qkv[:, :d], k, v, t + 1, H, batch.pad_left.cpu(), pk, pv)
        # one rounding to bf16 (at most 2^-8 of a value) and, where q is rotated, its own
        assert ((ctx - ref).norm() / ref.norm()).item() < 2.0 ** -7


@pytest.mark.parametrize("name", ["opt", "llama"])
def test_step_past_the_caches_is_refused(name):
    m = _models()[name]().init_random_fast(3, std=0.05)
    batch = make_batch(torch.arange(4, 16).view(2, 6)).to("cuda")
    dec = _Decoder(m, 2, 7)
    dec.prefill(batch)
    tok = torch.full((2,), 7, dtype=torch.int32, device="cuda")
    pos = torch.full((2,), 8, dtype=torch.int32, device="cuda")
    dec.step(tok, pos, batch.pad_left)
    before = [x.clone() for x in dec.k + dec.v]
    with pytest.raises((_lib.KernelError, IndexError)):
        dec.step(tok, pos + 1, batch.pad_left)
    _lib.check_device_errors()
    assert dec.len == 7 and all(torch.equal(x, y) for x, y in zip(before, dec.k + dec.v))


def test_step_after_a_reorder_to_fewer_sequences():
    m = _models()["opt"]().init_random_fast(3, std=0.05)
    batch = make_batch(torch.arange(4, 28).view(4, 6)).to("cuda")
    tok = torch.full((4,), 7, dtype=torch.int32, device="cuda")
    pos = torch.full((4,), 8, dtype=torch.int32, device="cuda")
    index = torch.tensor([2], device="cuda")
    out = []
    for native in (True, False):
        dec = _Decoder(m, 4, 16)
        dec.native = native
        dec.prefill(batch)
        dec.step(tok, pos, batch.pad_left)
        dec.reorder(index)
        out.append(dec.step(tok[:1], pos[:1] + 1, batch.pad_left[index]))
    _lib.check_device_errors()
    assert ((out[0] - out[1]).norm() / out[1].norm()).item() < 2 * 2.0 ** -8


@pytest.mark.parametrize("shift", [0, 4, 1])
def test_decode_attention_over_rows_off_a_16_byte_boundary(shift):
    """Caches and prefix rows may start anywhere: the values are those of the aligned ones, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(shift)
    B, n, H, hd, P = 2, 37, 3, 64, 5

    def rows(*shape):
        flat = torch.randn(math.prod(shape) + shift, device="cuda", generator=g).bfloat16()
        return flat[shift:].view(shape)

    q, k, v, pk, pv = rows(B, H * hd), rows(B, n, H * hd), rows(B, n, H * hd), rows(P, H * hd), rows(P, H * hd)
    y = decode_ops.decode_attention(q, k, v, n - 1, H, None, pk, pv)
    ref = decode_ops.decode_attention(q, k.clone(), v.clone(), n - 1, H, None, pk.clone(), pv.clone())
    _lib.check_device_errors()
    assert torch.equal(y, ref)


@pytest.mark.parametrize("B,H,hd", [(16, 19, 64), (31, 10, 80), (64, 5, 128)])
@pytest.mark.parametrize("n", [1, 7, 59, 60, 400])
def test_decode_attention_of_many_heads(B, H, hd, n):
    """More (sequence, head) pairs than run at once, around the number of keys (64, prefix rows among them) up to which a CTA
    has four warps."""
    g = torch.Generator(device="cuda").manual_seed(n + hd)
    q, k, v = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((B, H * hd), (B, n, H * hd), (B, n, H * hd)))
    pk, pv = (torch.randn(5, H * hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    pad = torch.randint(0, n, (B,), device="cuda", dtype=torch.int32, generator=g)
    y = decode_ops.decode_attention(q, k, v, n, H, pad, pk, pv)
    _lib.check_device_errors()
    ref = decode_attention_reference(q.float(), k.float(), v.float(), n, H, pad, pk.float(), pv.float())
    # one rounding to bf16 (at most 2^-8 of a value) beside fp32 sums and exponentials
    assert ((y.float() - ref).norm() / ref.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("V", [1024, 4096, 32768, 65536])
def test_draw_without_filters_walks_the_mass_in_order(V):
    """Equal logits: every probability is 2^-k, every partial sum is exact, and the token follows from the Philox word."""
    logits = torch.zeros(3, V, device="cuda")
    for off in range(8):
        got = decode_ops.sample_step(logits, seed=11, offset=off).tolist()
        for row, tok in enumerate(got):
            word = int(philox.philox4x32(row, off, 0, 3, 11, 0)[0])
            u = np.float32(np.float32((word >> 8) + 0.5) * np.float32(2.0 ** -24))
            assert tok == math.ceil(float(u) * V) - 1


@pytest.mark.parametrize("V", [1, 3, 4, 511, 2048, 32003])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_greedy_token_is_the_first_of_the_largest(V, shift):
    g = torch.Generator(device="cuda").manual_seed(V)
    flat = torch.randint(-9, 10, (4 * (V + 5) + shift,), device="cuda", generator=g).float()
    logits = flat[shift:].view(4, V + 5)[:, :V]
    got = decode_ops.sample_step(logits, do_sample=False).tolist()
    assert got == [r.index(max(r)) for r in logits.tolist()]


@pytest.mark.parametrize("V", [7, 512, 2049, 32000, 51200])
@pytest.mark.parametrize("top_k,top_p", [(None, None), (40, None), (None, 0.9), (300, 0.6)])
def test_sampler_forms_agree(V, top_k, top_p):
    """The shared-memory form and the form for vocabularies beyond it draw the same tokens: columns of -inf that push the
    row over the limit add exact zeros to every sum."""
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = torch.randn(6, V, device="cuda", generator=g) * 3
    logits[5] = 0.0
    wide = torch.full((6, 51300), float("-inf"), device="cuda")
    wide[:, :V] = logits
    for off in range(4):
        a = decode_ops.sample(logits, 0.8, top_k, top_p, True, seed=11, offset=off)
        b = decode_ops.sample(wide, 0.8, top_k, top_p, True, seed=11, offset=off)
        assert torch.equal(a, b)
        p = torch.softmax(logits / 0.8, -1)
        assert (p.gather(1, a[:, None]) > 0).all()
    assert torch.equal(decode_ops.sample(logits, do_sample=False), logits.argmax(-1))


def test_sample_step_marks_finished_rows():
    logits = torch.full((3, 100), -5.0, device="cuda")
    logits[0, 9], logits[1, 4], logits[2, 50] = 5.0, 5.0, 5.0
    done = torch.tensor([0, 0, 1], dtype=torch.int32, device="cuda")
    eos = torch.tensor([4, 60], dtype=torch.int32, device="cuda")
    out = decode_ops.sample_step(logits, do_sample=False, done=done, eos=eos, pad_id=1)
    assert out.tolist() == [9, 4, 1] and done.tolist() == [0, 1, 1]


@pytest.mark.parametrize("sample", [False, True])
def test_generate_stops_rows_at_an_end_of_sequence_id(sample):
    """Rows end with their first EOS id."""
    m = _models()["opt"]().init_random_fast(3, std=0.05)
    g = torch.Generator().manual_seed(4)
    ids = torch.randint(4, 500, (3, 20), generator=g)
    mask = torch.ones_like(ids)
    mask[1, :7] = 0
    kw = dict(max_new_tokens=9, do_sample=sample, top_p=0.9, seed=3)
    free = generate(m, ids, mask, **kw)
    for stop in ({free[0][21]}, {row[-3] for row in free}):
        got = generate(m, ids, mask, eos_token_id=sorted(stop), pad_token_id=1, **kw)
        for row, prompt, out in zip(free, (20, 13, 20), got):
            end = next((i + 1 for i in range(prompt, len(row)) if row[i] in stop), len(row))
            assert out == row[:end]
    assert generate(m, ids, mask, max_new_tokens=0) == [r[k.bool()].tolist() for r, k in zip(ids, mask)]


@pytest.mark.parametrize("name", ["opt", "llama"])
def test_generate_queues_no_step_behind_the_last_token(name, monkeypatch):
    m = _models()[name]().init_random_fast(3, std=0.05)
    ids = torch.randint(4, 500, (2, 20), generator=torch.Generator().manual_seed(4))
    steps = []
    step = decode_ops.DecodePlan.step
    monkeypatch.setattr(decode_ops.DecodePlan, "step", lambda self, *a: (steps.append(1), step(self, *a))[1])
    kw = dict(max_new_tokens=9, do_sample=True, seed=3)
    free = generate(m, ids, **kw)
    assert len(steps) == 8 and all(len(r) == 29 for r in free)
    stop = {r[20 + i] for i, r in enumerate(free)}                 # the rows end with their first and second token at latest
    del steps[:]
    got = generate(m, ids, eos_token_id=sorted(stop), **kw)
    assert len(steps) == max(len(r) for r in got) - 21
    assert all(r == f[:len(r)] and r[-1] in stop for r, f in zip(got, free))


def test_generate_takes_end_of_sequence_ids_outside_the_vocabulary():
    m = _models()["opt"]().init_random_fast(3, std=0.05)
    ids = torch.arange(4, 16).view(2, 6)
    assert generate(m, ids, max_new_tokens=3, eos_token_id=[-1, 520, 2 ** 40]) == generate(m, ids, max_new_tokens=3)
