"""Edges of the tiled kernels of the quantized path, bit for bit against the oracle: products of a few and of many tokens at the ends of
their tiles and over several tiles per CTA, blocks at the limit of what one accumulator holds and above it, exact-order attention of portions and
single rows for every grouping of heads."""
import numpy as np
import pytest

import oracle as O
from gpu_common import assert_bit_equal, backend, kernels_run  # noqa: F401
from orangu_b200 import LlamaModel, QuantMatrix, synth
from q4k_make import SUM24, code_bytes, q4k_blocks, scale_bytes, sums

pytestmark = pytest.mark.gpu
Q4_K, Q6_K = 12, 14


def both_orders(backend, w, x, n):
    shape = (w.ggml_type(), w.in_dim, w.out_dim)
    assert_bit_equal(backend.matmul(x, n, w).reshape(-1), O.matmul(x, n, w.raw, *shape).reshape(-1), f"prefill order, {n} tokens")
    assert_bit_equal(backend.matmul_decode(x, n, w).reshape(-1), O.matmul_decode(x, n, w.raw, *shape).reshape(-1), f"decode order, {n} tokens")


# rows: not a multiple of 16 or 128; columns: one super-block, fewer than the warps that share a sum, more than a buffer of mins (16).  Mostly the
# few-token kernel; tiles of 16 and 32 tokens from some 100 tokens on.
@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("rows,cols", [(2100, 256), (1030, 768), (2100, 4608)])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 31, 33, 48, 49, 64, 65, 96, 97, 113, 129, 200])
def test_products_at_the_edges_of_tiles(backend, t, rows, cols, n):
    w = QuantMatrix(synth.matrix(t, rows, cols, 5)["data"], t, cols, rows)
    both_orders(backend, w, synth.normal(n * cols, 6 + n), n)


@pytest.mark.parametrize("few", [True, False])
def test_sums_beyond_one_accumulator(backend, few):
    """Rows whose every code is 15 and every scale 63 against activations of the largest code: halves of 15.4e6 and sums of 30.7e6, above
    2^24; among rows of ordinary blocks, few of them or many.  (These sizes take the few-token kernel, whose sums are integers.)"""
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


# ---- the tcgen05 tiles of Q4_K
def extreme_rows(n, cols):
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    x[::3] = 1.5  # every code 127
    x[1::6] = np.where(np.arange(cols) % 7 == 0, -1.5, 1.5)
    x[2::6] = np.where(np.arange(cols) % 256 < 128, 1.5, -1.5)  # large sums that cancel
    return x.reshape(-1)


def routes(backend, w, x, n, prefill, decode):
    """Both orders bit for bit, and the kernels that ran: `prefill` and `decode` are what their names have to contain."""
    for run, want in ((backend.matmul, prefill), (backend.matmul_decode, decode)):
        names = [k for k in kernels_run(lambda: run(x, n, w)) if "gemm" in k or "gemv" in k]
        assert len(names) == len(want) and all(any(part in k for k in names) for part in want), (names, want)
    both_orders(backend, w, x, n)


@pytest.fixture(scope="module")
def tall_matrices():
    """296 tiles of 128 rows, the last one ragged, so that CTAs take several tiles, and nine super-blocks, an odd number for the two warps that
    issue.  Without wide rows, with a few (which a kernel of their own computes), with more than one in 128 (halves apart)."""
    rows, cols = 296 * 128 - 50, 9 * 256
    few = np.r_[0, 3:5, 130, 5000, rows - 1]
    return {kind: QuantMatrix(q4k_blocks(rows, cols, 9, wide).reshape(-1), Q4_K, cols, rows)
            for kind, wide in (("none", np.r_[0:0]), ("few", few), ("many", np.r_[few, 9000:9400]))}


# widths of tile that the rule takes: prefill order, decode order; the same with halves apart
@pytest.mark.parametrize("n,plain,apart", [(13, (16, 16), (16, 16)), (31, (32, 32), (32, 32)), (47, (64, 48), (64, 32)), (61, (64, 32), (64, 32)),
                                           (95, (96, 48), (64, 32)), (200, (96, 48), (64, 32))])
@pytest.mark.parametrize("wide", ["none", "few", "many"])
def test_tiles_of_every_width(backend, tall_matrices, n, plain, apart, wide):
    w = tall_matrices[wide]
    two, widths = ("true", apart) if wide == "many" else ("false", plain)
    rows_apart = ["gemm_few_kernel"] if wide == "few" else []
    routes(backend, w, extreme_rows(n, w.in_dim), n, [f"gemm_tc5_q4k_kernel<true, {two}, {widths[0]}>"] + rows_apart,
           [f"gemm_tc5_q4k_kernel<false, {two}, {widths[1]}>"] + rows_apart)


def test_token_scales_of_one_tile_at_a_time(backend):
    """Rows of 112 super-blocks: the scales of two tiles do not fit beside tiles of 96 tokens."""
    rows, cols, n = 4700, 28672, 520
    w = QuantMatrix(q4k_blocks(rows, cols, 4, np.r_[0:0]).reshape(-1), Q4_K, cols, rows)
    x = synth.normal(n * cols, 5)
    assert any("gemm_tc5_q4k_kernel<true, false, 96>" in k for k in kernels_run(lambda: backend.matmul(x, n, w)))
    assert_bit_equal(backend.matmul(x, n, w).reshape(-1), O.matmul(x, n, w.raw, Q4_K, cols, rows).reshape(-1), "prefill order")


@pytest.mark.parametrize("above", [0, 1])
def test_sums_at_the_limit_of_an_accumulator(backend, above):
    """Blocks whose scales times codes are the largest that is taken for one accumulator, or one or a few less, so that sums against the largest
    activations are whole numbers, odd ones too, up to 2^24 - 8; and one more, which makes their rows wide."""
    rows, cols, n = 4000, 9 * 256, 200
    rng = np.random.default_rng(7)
    blocks = q4k_blocks(rows, cols, 2, np.r_[0:0])
    at = np.r_[0:40, 127:129, 3000:3040, rows - 1]
    for r in at:
        for b in range(blocks.shape[1]):
            if rng.random() < 0.3:
                continue
            # 120960 in four sub-blocks of the largest codes, 11088 in one, what is left in one of scale 1, in any order
            sc, codes = np.array([63, 63, 63, 63, 63, 1, 40, 7]), np.zeros((8, 32), np.int64)
            codes[:4] = 15
            codes[4, :12] = [15] * 11 + [11]
            left = SUM24 - 120960 - 63 * 176 + (above if r in at[::4] and b % 2 else -int(rng.integers(0, 4)))
            codes[5, :left // 8] = 8
            codes[5, left // 8] = left % 8
            order = rng.permutation(8)
            sub = np.array([rng.permutation(c) for c in codes])
            blocks[r, b, 4:16] = scale_bytes(sc[None, order], rng.integers(0, 64, (1, 8)))[0]
            blocks[r, b, 16:] = code_bytes(sub[None, order])[0]
    s = sums(blocks)
    assert s.max() == SUM24 + above and ((s > SUM24).any(1).sum() > 0) == bool(above)
    w = QuantMatrix(blocks.reshape(-1), Q4_K, cols, rows)
    x = extreme_rows(n, cols).reshape(n, cols)
    x[3::6] = -1.5
    assert (s > SUM24).any(1).sum() <= rows // 128
    rows_apart = ["gemm_few_kernel"] if above else []
    routes(backend, w, x.reshape(-1), n, ["gemm_tc5_q4k_kernel<true"] + rows_apart, ["gemm_tc5_q4k_kernel<false"] + rows_apart)


def test_wide_rows_in_a_step_of_a_model(backend):
    """Three matrices of different heights in one launch, some with wide rows and some without; products added to the residual stream that they are
    written to; the same in a captured decode step."""
    cfg = dict(n_vocab=256, n_embd=1280, n_layer=2, n_head=10, n_head_kv=5, head_dim=128, n_ff=9472, rope_freq_base=10000.0, rms_eps=1e-5)
    tensors = synth.model_tensors(cfg, seed=5, types={"attn_v": Q4_K})
    for i in range(2):
        for name, wide in (("attn_q", np.r_[0:0]), ("attn_k", np.r_[1, 255]), ("attn_v", np.r_[130]), ("attn_output", np.r_[7, 1279]), ("ffn_gate", np.r_[5, 3000:3020]),
                           ("ffn_up", np.r_[0:0]), ("ffn_down", np.r_[0, 128])):
            t = tensors[f"blk.{i}.{name}.weight"]
            t["data"] = q4k_blocks(t["out_dim"], t["in_dim"], 31 * i + len(name), wide).reshape(-1)
    model, ref = LlamaModel(backend, cfg, tensors, max_seq_len=512, max_batch_tokens=300, kv_pool_tokens=4096), O.Model(cfg, tensors)
    rng = np.random.default_rng(1)
    toks = rng.integers(0, cfg["n_vocab"], 300).astype(np.uint32)
    kv, rkv = model.new_kv_cache(320), ref.new_kv(320, f16=True)
    want, hidden = ref.forward(rkv, toks, 0, want_hidden=True)
    got = []
    names = kernels_run(lambda: got.append(model.forward(kv, toks, 0)))
    # attention's three, its output, gate and up, down: all on tiles, each with a kernel for every matrix that has wide rows
    assert sum("gemm_tc5_q4k_kernel" in k for k in names) == 8 and sum("gemm_few_kernel" in k for k in names) >= 2 * 5, names
    assert_bit_equal(got[0], want, "prefill logits")
    assert_bit_equal(model.last_hidden(300), hidden, "residual stream")
    kvs, rkvs, first = [], [], []
    for s in range(16):
        kvs.append(model.new_kv_cache(32))
        rkvs.append(ref.new_kv(32, f16=True))
        toks = rng.integers(0, cfg["n_vocab"], 3 + s % 4).astype(np.uint32)
        assert_bit_equal(model.forward(kvs[s], toks, 0), ref.forward(rkvs[s], toks, 0), f"sequence {s}")
        first.append(int(toks[0]))
    out = []
    names = kernels_run(lambda: out.append(model.decode_loop(kvs, first, 6)))
    assert any("gemm_tc5_q4k_kernel<false, false, 16>" in k for k in names) and any("gemm_few_kernel" in k for k in names), names
    for s in range(16):
        tok, at = first[s], 3 + s % 4
        for i in range(6):
            tok = O.argmax(ref.forward(rkvs[s], [tok], at + i))
            assert out[0][i][s] == tok, (s, i)
    model.close()


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
