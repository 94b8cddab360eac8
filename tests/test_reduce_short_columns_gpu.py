"""Column reductions with few rows or many columns: a thread per vector or element of the output, eight warps per group of
columns, and the sizes where one gives way to the other; outputs off the 16-byte boundary, f32 results of 16-bit values.
And infinities and NaN on every path of rows and columns, against the oracle."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from test_kernels_gpu import _assert_max_equal, _make, _to_dev, _to_host

pytestmark = pytest.mark.gpu
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}

# units: A * C / 4 or / 8 where C is whole vectors, else A * C; a thread per unit from 1184 B or 200 B of them on
CASES = [
    # A, B, C
    (1, 2, 8), (2, 7, 24), (5, 8, 40), (5, 9, 40), (2, 16, 4736), (4, 16, 37888), (1, 32, 64), (1, 33, 64), (3, 31, 1000), (70, 20, 16),
    (9, 40, 21200), (20, 66, 16000), (2, 3, 3), (7, 2, 881), (1, 15, 977), (1, 16, 33), (1, 17, 33), (90, 17, 23), (1, 32, 33), (3, 20, 17),
    (1, 33, 6601), (1, 33, 6599), (1, 64, 1001), (1, 65, 1001), (3, 65, 803), (2, 100, 10001), (2, 100, 9999), (1, 300, 60001), (1, 300, 22201),
    (1, 300, 22199), (1, 300, 1023),
]


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("op", ["sum", "max", "f32"])
@pytest.mark.parametrize("A,B,C", CASES)
def test_short_columns(A, B, C, op, dt):
    from byteir_b200 import ops
    rng = np.random.default_rng(A * 7 + B * 3 + C)
    x = _make(rng, (A, B, C), dt, "normal")
    if op == "max":  # a quarter of the columns with zeros of either sign as their maximum
        m = -np.abs(O.to_f32(x)) - 0.125
        z = rng.random((A, B, (C + 3) // 4))
        m[:, :, ::4] = np.where(z < 0.3, np.where(z < 0.15, -0.0, 0.0), m[:, :, ::4])
        x = m.astype(np.float16) if dt == "f16" else m.astype(np.float32) if dt == "f32" else O.f32_to_bf16(m.astype(np.float32))
    for head in (0, 1):  # elements that input and output begin behind the boundary
        xd = _to_dev(np.concatenate([x.reshape(-1)[:head], x.reshape(-1)]))[head:].view(A, B, C)
        out = torch.empty(A * C + head, device="cuda", dtype=torch.float32 if op == "f32" else TORCH[dt])[head:]
        fn = {"sum": ops.reduce_sum, "max": ops.reduce_max, "f32": ops.reduce_sum_to_f32}[op]
        got = _to_host(fn(xd, [1], out=out)).reshape(-1)
        if op == "max":
            _assert_max_equal(got, O.reduce("max", x, A, B, C))
            continue
        # f32 sums: at most B / 8 + 8 additions in a chain, then one rounding to the output type
        ref = O.reduce_sum_f64(x, A, B, C)
        mag = np.abs(O.to_f32(x).astype(np.float64)).sum(axis=1).reshape(-1)
        ulp = 0.0 if op == "f32" else {"f32": 0.0, "f16": 2.0**-11, "bf16": 2.0**-8}[dt]
        bound = ulp * np.abs(ref) * 1.001 + 2.0**-24 * (B / 8 + 12) * mag + (2.0**-25 if dt == "f16" and op == "sum" else 0)
        assert np.all(np.abs(O.to_f32(got).astype(np.float64) - ref) <= bound)


# rows: whole vectors, odd pitch in shared memory, odd pitch by lanes, segments; columns: a thread per unit, eight warps, super-rows
# of one and of several rows, a cluster, a second pass over them
SPECIAL = [(70, 64, 1), (300, 33, 1), (700, 385, 1), (2, 100003, 1), (3, 7, 40), (2, 30, 40), (2, 60, 129), (64, 100, 129), (1, 4100, 1024),
           (1, 3001, 1023), (1, 20000, 3), (1, 2000, 2049)]


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("A,B,C", SPECIAL)
def test_infinities_and_nan_on_every_path(A, B, C, dt):
    from byteir_b200 import ops
    rng = np.random.default_rng(B + C)
    x = O.to_f32(_make(rng, (A, B, C), dt, "normal"))
    flat = x.transpose(0, 2, 1).reshape(-1, B)  # one row per result
    n = flat.shape[0]
    flat[0::5] = -np.inf                                             # nothing but the least value
    flat[1::5][np.arange(len(flat[1::5])), rng.integers(0, B, len(flat[1::5]))] = np.nan
    flat[2::5][np.arange(len(flat[2::5])), rng.integers(0, B, len(flat[2::5]))] = np.inf
    x = np.ascontiguousarray(flat.reshape(A, C, B).transpose(0, 2, 1))
    x = x.astype(np.float16) if dt == "f16" else x if dt == "f32" else O.f32_to_bf16(x)
    xd = _to_dev(x)
    _assert_max_equal(_to_host(ops.reduce_max(xd, [1])).reshape(-1), O.reduce("max", x, A, B, C))
    got = O.to_f32(_to_host(ops.reduce_sum(xd, [1]))).reshape(-1)
    kind = np.arange(n) % 5
    assert np.all(got[kind == 0] == -np.inf) and np.all(np.isnan(got[kind == 1])) and np.all(got[kind == 2] == np.inf)
    assert np.all(np.isfinite(got[kind > 2]))
