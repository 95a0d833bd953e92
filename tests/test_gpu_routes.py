"""Which kernels a product takes, and what the host knows of them afterwards."""
import numpy as np
import pytest

from gpu_common import backend, kernels_run  # noqa: F401
from orangu_b200 import LlamaModel, QuantMatrix, synth
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
