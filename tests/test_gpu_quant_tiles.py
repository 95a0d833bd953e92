"""Edges of the tiled kernels of the quantized path, bit for bit against the oracle: products of a few and of many tokens at the ends of
their tiles, blocks at the limit of what one accumulator holds, exact-order attention of portions and single rows for every grouping of heads."""
import numpy as np
import pytest

import oracle as O
from gpu_common import assert_bit_equal, backend  # noqa: F401
from orangu_b200 import LlamaModel, QuantMatrix, synth

pytestmark = pytest.mark.gpu
Q4_K, Q6_K = 12, 14


def both_orders(backend, w, x, n):
    shape = (w.ggml_type(), w.in_dim, w.out_dim)
    assert_bit_equal(backend.matmul(x, n, w).reshape(-1), O.matmul(x, n, w.raw, *shape).reshape(-1), f"prefill order, {n} tokens")
    assert_bit_equal(backend.matmul_decode(x, n, w).reshape(-1), O.matmul_decode(x, n, w.raw, *shape).reshape(-1), f"decode order, {n} tokens")


# rows: not a multiple of 16 or 128; columns: one super-block, fewer than the warps that share a sum, more than a buffer of mins (16)
@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("rows,cols", [(2100, 256), (1030, 768), (2100, 4608)])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 31, 33, 48, 49, 64, 65, 96, 97, 113, 129, 200])
def test_products_at_the_edges_of_tiles(backend, t, rows, cols, n):
    w = QuantMatrix(synth.matrix(t, rows, cols, 5)["data"], t, cols, rows)
    both_orders(backend, w, synth.normal(n * cols, 6 + n), n)


@pytest.mark.parametrize("few", [True, False])
def test_sums_beyond_one_accumulator(backend, few):
    """Rows whose every code is 15 and every scale 63 against activations of the largest code: halves of 15.4e6 and sums of 30.7e6, above
    2^24; among rows of ordinary blocks, in some tiles of 128 rows and not in others, few of them or many."""
    rows, cols = 2100, 512
    blocks = synth.matrix(Q4_K, rows, cols, 9)["data"].reshape(rows, -1, 144).copy()
    full = np.r_[3:5, 130, 2099] if few else np.r_[3:5, 130, 700:900, 2099]
    blocks[full, :, 4:12] = 0xff  # scales and mins 63, their upper bits too
    blocks[full, :, 12:16] = 0xff
    blocks[full, :, 16:] = 0xff
    blocks[full[::2], :, 20:21] = 0x3e  # not all alike: odd sums as well
    w = QuantMatrix(blocks.reshape(-1), Q4_K, cols, rows)
    for n in (16, 40, 130):
        x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
        x[::3] = 1.5
        x[1::6] = np.where(np.arange(cols) % 7 == 0, -1.5, 1.5)
        both_orders(backend, w, x.reshape(-1), n)


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
