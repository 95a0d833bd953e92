"""Which kernels a product takes, and what the host knows of them afterwards."""
import numpy as np
import pytest

import oracle as O
from gpu_common import assert_bit_equal, backend, kernels_run  # noqa: F401
from orangu_b200 import LlamaModel, QuantMatrix, capi, synth
from q4k_make import q4k_blocks

pytestmark = pytest.mark.gpu
Q8_0, Q4_K, Q6_K = 8, 12, 14


def own(names):
    return [k for k in names if "Memcpy" not in k and "Memset" not in k]


# tiles without and with wide rows, a few tokens, tokens taken in several launches
@pytest.mark.parametrize("rows,cols,n,wide", [(18894, 2304, 64, []), (18894, 2304, 64, [3, 900]), (700, 768, 5, [3]), (64, 66048, 7, [])])
def test_launches_are_counted(backend, rows, cols, n, wide):
    w = QuantMatrix(q4k_blocks(rows, cols, 3, np.array(wide, int)).reshape(-1), Q4_K, cols, rows)
    x = synth.normal(n * cols, 4)
    for run in (backend.matmul, backend.matmul_decode):
        run(x, n, w)
        before = backend.launch_count()
        names = own(kernels_run(lambda: run(x, n, w)))
        assert backend.launch_count() - before == len(names), names


def test_long_rows_of_many_tokens_take_the_tiles(backend):
    """Prefill order, rows of 112 super-blocks: the few-token kernel holds the terms of 8 tokens at a time, not of 16, and is the slower."""
    rows, cols, n = 4096, 28672, 48
    w = QuantMatrix(q4k_blocks(rows, cols, 3, np.r_[0:0]).reshape(-1), Q4_K, cols, rows)
    x = synth.normal(n * cols, 4)
    assert any("gemm_tc5_q4k_kernel" in k for k in kernels_run(lambda: backend.matmul(x, n, w)))
    assert_bit_equal(backend.matmul(x, n, w), O.matmul(x, n, w.raw, Q4_K, cols, rows), "48 tokens")


# 7104 and 9472 rows are three and four tiles of 16 rows an SM; the kernels of prefill order, of decode order
@pytest.mark.parametrize("t,rows,cols,n,prefill,decode", [
    (Q4_K, 7104, 768, 2, "few", "few"), (Q4_K, 7105, 768, 2, "gemv", "few"), (Q4_K, 7105, 4096, 2, "gemv", "gemv"), (Q4_K, 9473, 768, 2, "gemv", "gemv"),
    (Q4_K, 9472, 768, 3, "few", "few"), (Q4_K, 9473, 768, 3, "gemv", "gemv"), (Q4_K, 9473, 768, 4, "few", "few"),
    (Q6_K, 9472, 768, 2, "few", "few"), (Q6_K, 9473, 768, 2, "few", "gemv"), (Q6_K, 9473, 768, 3, "few", "few")])
def test_two_and_three_tokens(backend, t, rows, cols, n, prefill, decode):
    w = QuantMatrix(synth.matrix(t, rows, cols, 5)["data"], t, cols, rows)
    x = synth.normal(n * cols, 6)
    for run, want, oracle in ((backend.matmul, prefill, O.matmul), (backend.matmul_decode, decode, O.matmul_decode)):
        names = kernels_run(lambda: run(x, n, w))
        assert any({"few": "gemm_few_kernel", "gemv": "gemv_kernel"}[want] in k for k in names), names
        assert_bit_equal(run(x, n, w), oracle(x, n, w.raw, t, cols, rows), "products")


def test_f16_codes_are_held_only_for_q4k_weights(backend):
    """The tiles of Q4_K read activations in a form of their own, 2.2 bytes an entry; a model without Q4_K weights holds none of it."""
    import torch

    cfg = dict(n_vocab=256, n_embd=256, n_layer=1, n_head=4, n_head_kv=2, head_dim=64, n_ff=8192, rope_freq_base=10000.0, rms_eps=1e-5)
    names = ("token_embd", "output", "attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    used = {}
    for t in (Q4_K, Q6_K):
        tensors = synth.model_tensors(cfg, seed=3, types={name: t for name in names})
        before = torch.cuda.mem_get_info()[0]
        model = LlamaModel(backend, cfg, tensors, max_seq_len=4096, max_batch_tokens=4096, exact_attention_max_pos=64)
        used[t] = before - torch.cuda.mem_get_info()[0]
        model.close()
    entries = 4096 * (256 + 256 + 8192)
    assert used[Q4_K] - used[Q6_K] > 1.9 * entries, used  # (weights of Q6_K are the larger, by 4.5 MB)


@pytest.mark.parametrize("t,n_seq", [(Q4_K, 16), (Q8_0, 16)])
def test_a_wait_that_ran_out_in_a_replayed_step_is_reported(backend, t, n_seq):
    """The steps of a decode loop are captured at its first call and only replayed afterwards; the status that their products leave is read
    after every call."""
    cfg = dict(n_vocab=256, n_embd=1280, n_layer=1, n_head=10, n_head_kv=5, head_dim=128, n_ff=9472, rope_freq_base=10000.0, rms_eps=1e-5)
    tensors = synth.model_tensors(cfg, seed=3, types={name: t for name in ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down", "output")})
    model = LlamaModel(backend, cfg, tensors, max_seq_len=64, max_batch_tokens=16, kv_pool_tokens=2048)
    kvs = [model.new_kv_cache(48) for _ in range(n_seq)]
    first = list(range(n_seq))
    tile = "gemm_tc5_q4k" if t == Q4_K else "gemm_tc5_q8"
    assert any(tile in k for k in kernels_run(lambda: model.decode_loop(kvs, first, 2)))
    model.decode_loop(kvs, first, 2)
    capi.check(backend._h, backend._lib.ob_tile_wait_selftest(backend._h))
    with pytest.raises(capi.OranguError, match="gave up a bounded wait"):
        model.decode_loop(kvs, first, 2)
    model.decode_loop(kvs, first, 2)  # reported once
    model.close()
