"""Column maxima that are exactly zero: the sign is that of the last zero, wherever in the column it lies, and finding it costs
a small part of the column, on every path of the plan (one block, a cluster, a second pass, super-rows of one and of more rows)."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from test_kernels_gpu import _to_dev, _to_host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 20000, 16), (1, 4096, 512), (2, 3001, 129), (1, 9001, 1024), (1, 4001, 1023), (1, 5003, 2049), (3, 700, 4100), (1, 64, 9001),
          (5, 31, 24), (300, 64, 64), (1, 2000, 3), (2, 1000, 64)]


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("A,B,C", SHAPES)
def test_sign_of_the_last_zero_in_any_row(A, B, C, dt):
    from byteir_b200 import ops
    rng = np.random.default_rng(A + B + C)
    x = -rng.random((A, B, C), dtype=np.float32) - 0.5
    first, second = np.sort(rng.integers(0, B, (2, A, C)), axis=0)  # up to two zeros per column, of either sign
    first[:, ::7], second[:, ::7] = 0, 0                            # ... and some with one zero in the first row
    first[:, 1::7], second[:, 1::7] = 0, B - 1
    a, c = np.meshgrid(np.arange(A), np.arange(C), indexing="ij")
    x[a, first, c] = np.where(rng.random((A, C)) < 0.5, -0.0, 0.0)
    x[a, second, c] = np.where(rng.random((A, C)) < 0.5, -0.0, 0.0)
    want = x[a, second, c]
    x = x.astype(np.float16) if dt == "f16" else x if dt == "f32" else O.f32_to_bf16(x)
    for head in (0, 1):
        xd = _to_dev(np.concatenate([x.reshape(-1)[:head], x.reshape(-1)]))[head:].view(A, B, C)
        got = O.to_f32(_to_host(ops.reduce_max(xd, [1]))).reshape(A, C)
        assert np.array_equal(got, want) and np.array_equal(np.signbit(got), np.signbit(want))


# one zero in the first of 200000 rows: a walk over all of them, one load after the other, takes 36 ms
def test_a_zero_in_front_does_not_cost_a_walk_over_all_rows():
    from byteir_b200 import ops
    x = torch.full((200000, 16), -1.0, device="cuda", dtype=torch.float16)
    x[0] = -0.0
    ops.reduce_max(x, [0])
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    got = ops.reduce_max(x, [0])
    end.record()
    end.synchronize()
    assert bool((got == 0).all()) and bool(torch.signbit(got).all())
    assert start.elapsed_time(end) < 5.0
