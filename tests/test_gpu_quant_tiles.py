"""Edges of the tiled kernels of the quantized path, bit for bit against the oracle: exact-order attention of portions and
single rows for every grouping of heads."""
import numpy as np
import pytest

import oracle as O
from gpu_common import assert_bit_equal, backend  # noqa: F401
from orangu_b200 import LlamaModel, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim", [(4, 4, 64), (4, 2, 128), (6, 2, 128), (16, 4, 80), (8, 1, 64), (16, 2, 16)])
def test_exact_attention_of_portions_and_rows(backend, heads, kv_heads, dim):
    cfg = dict(n_vocab=256, n_embd=256, n_layer=2, n_head=heads, n_head_kv=kv_heads, head_dim=dim, n_ff=512, rope_freq_base=10000.0, rms_eps=1e-5)
    tensors = synth.model_tensors(cfg, seed=heads)
    model, ref = LlamaModel(backend, cfg, tensors, max_seq_len=640, max_batch_tokens=150), O.Model(cfg, tensors)
    kv, rkv = model.new_kv_cache(600), ref.new_kv(600, f16=True)
    at = 0
    rng = np.random.default_rng(dim)
    for n in (150, 1, 64, 7, 33, 1, 130, 140, 1):  # portions that begin and end inside tiles and pages, single rows between them
        toks = rng.integers(0, cfg["n_vocab"], n).astype(np.uint32)
        assert_bit_equal(model.forward(kv, toks, at), ref.forward(rkv, toks, at), f"{n} tokens at {at}")
        at += n
    model.close()


@pytest.mark.parametrize("dim", [64, 96])
def test_head_norms_biases_and_rotations(backend, dim):
    """One warp per head: dimensions that fill its lanes and that do not, heads that fill a CTA and that do not, several tokens."""
    cfg = dict(n_vocab=256, n_embd=256, n_layer=2, n_head=8, n_head_kv=1, head_dim=dim, n_ff=512, rope_freq_base=10000.0, rms_eps=1e-5, rope_neox=True)
    tensors = synth.add_qwen_extras(cfg, synth.model_tensors(cfg, seed=3), seed=3)
    model, ref = LlamaModel(backend, cfg, tensors, max_seq_len=64, max_batch_tokens=32), O.Model(cfg, tensors)
    kv, rkv = model.new_kv_cache(64), ref.new_kv(64, f16=True)
    toks = np.arange(40, dtype=np.uint32)
    for at, n in ((0, 29), (29, 1), (30, 10)):
        assert_bit_equal(model.forward(kv, toks[at:at + n], at), ref.forward(rkv, toks[at:at + n], at), f"{n} tokens at {at}")
    model.close()
