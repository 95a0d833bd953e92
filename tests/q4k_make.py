"""Q4_K blocks made to measure: which rows hold sums that one fp32 accumulator cannot."""
import numpy as np

from orangu_b200 import synth

Q4_K = 12
SUM24 = (2 ** 24 - 1) // 127  # scales times codes of a block that fit one accumulator whatever the activations


def scale_bytes(sc, m):
    """Eight 6-bit scales and mins of each block as its twelve bytes."""
    sc, m = np.asarray(sc, np.uint8), np.asarray(m, np.uint8)
    return np.concatenate([sc[:, :4] | (sc[:, 4:] >> 4 << 6), m[:, :4] | (m[:, 4:] >> 4 << 6), (sc[:, 4:] & 15) | (m[:, 4:] & 15) << 4], axis=1)


def code_bytes(codes):
    """[blocks][8][32] codes as the 128 bytes of each block: sub-blocks 2 g and 2 g + 1 are the low and high nibbles of group g."""
    c = np.asarray(codes, np.uint8)
    return (c[:, 0::2] | c[:, 1::2] << 4).reshape(len(c), 128)


def sums(blocks):
    """Scales times codes of every block."""
    b = blocks.reshape(-1, 144)
    s, q = b[:, 4:16].astype(np.int64), b[:, 16:].reshape(-1, 4, 32).astype(np.int64)
    sc = np.concatenate([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], axis=1)
    return (sc[:, 0::2] * (q & 15).sum(2) + sc[:, 1::2] * (q >> 4).sum(2)).sum(1).reshape(blocks.shape[:2])


def q4k_blocks(rows, cols, seed, wide=()):
    """Blocks of a matrix whose wide rows are the ones named: scales and mins 63 and codes 15, halves of 15.4e6 and sums of 30.7e6 against
    the largest activations, above 2^24."""
    blocks = synth.matrix(Q4_K, rows, cols, seed)["data"].reshape(rows, -1, 144).copy()
    blocks[sums(blocks) > SUM24, 4:8] &= 0x0f
    blocks[wide, :, 4:] = 0xff
    blocks[wide[::2], :, 20:21] = 0x3e  # not all alike: odd sums as well
    assert ((sums(blocks) > SUM24).any(1).nonzero()[0] == np.sort(wide)).all()
    return blocks
