"""Row gather in output order (rows that are no multiple of 32 bytes, or off the 16-byte boundary): units of every width, blocks
that end inside a row and rows longer than a block, the front dimension, indices out of range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TORCH = {1: torch.uint8, 2: torch.float16, 4: torch.float32, 8: torch.int64}


# row lengths around a unit of 16, 8, 4, 2 and 1 bytes, and around the 2048 units of a block
@pytest.mark.parametrize("elt,feature", [(2, 1), (2, 24), (2, 33), (4, 3), (4, 20), (4, 733), (8, 1), (8, 3), (1, 7), (1, 2047), (1, 2048), (1, 2049),
                                         (2, 5001), (4, 4100)])
@pytest.mark.parametrize("A,n,index", [(1, 1, torch.int64), (1, 700, torch.int32), (3, 129, torch.int64)])
def test_every_unit_width(elt, feature, A, n, index):
    from byteir_b200 import ops
    rng = np.random.default_rng(feature * 5 + n)
    rows = 97
    ids = rng.integers(0, rows, n)
    for head in (0, 1):  # elements that the table and the output begin behind the boundary
        raw = rng.integers(0, 256, (A * rows * feature + head) * elt, dtype=np.uint8)
        table = torch.from_numpy(raw).cuda().view(TORCH[elt])[head:].view(A, rows, feature)
        out = torch.zeros(A * n * feature + head + 1, dtype=TORCH[elt], device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        idx = torch.from_numpy(ids).to(index).cuda()
        ops.index_select(table, idx, 1, out=out[head:-1].view(A, n, feature), status=status)
        got = out[head:-1].view(A, n, feature).cpu().view(torch.uint8).numpy()
        want = raw.reshape(-1)[head * elt:].reshape(A, rows, feature * elt)[:, ids]
        assert np.array_equal(got.reshape(want.shape), want) and int(status) == 0
        assert int(out[-1:].view(torch.uint8).sum()) == 0  # nothing behind the end
        bad = idx.clone()
        bad[n // 2] = rows
        ops.index_select(table, bad, 1, out=out[head:-1].view(A, n, feature), status=status)
        want = want.copy()
        want[:, n // 2] = 0
        got = out[head:-1].view(A, n, feature).cpu().view(torch.uint8).numpy()
        assert np.array_equal(got.reshape(want.shape), want) and int(status) == 1
