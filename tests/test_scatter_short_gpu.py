"""Scatter-add of short lists, which one block sorts by itself.  The values are small whole numbers, so that every sum is
exact in any order and the result equals the plain loop's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# lengths around a warp's round, the rounds per warp, the largest list of one block (4096 in place, else 8192); row counts around one, two and three
# digits of 8 bits; ids that repeat, ids that are all the same, ids in falling order
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 4096, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("rows", [1, 2, 255, 256, 257, 65535, 65537, 200000])
def test_short_lists(n, rows):
    from byteir_b200 import ops
    rng = np.random.default_rng(n * 7 + rows)
    for feature, ids in ((8, rng.integers(0, rows, n)), (3, np.full(n, rows - 1)), (16, (rows - 1) - np.arange(n) % rows)):
        table, upd = rng.integers(-8, 8, (rows, feature)).astype(np.float32), rng.integers(-8, 8, (n, feature)).astype(np.float32)
        want = table.copy()
        np.add.at(want, ids, upd)
        t, i, u = torch.from_numpy(table).cuda(), torch.from_numpy(ids.astype(np.int64)).cuda(), torch.from_numpy(upd).cuda()
        assert np.array_equal(ops.index_put_add(t, i, u).cpu().numpy(), want)
        assert np.array_equal(ops.index_put_add(t, i, u, out=t).cpu().numpy(), want)


# beside a table copy one block sorts 5120 entries, and 8192 from 40 MB of table on
@pytest.mark.parametrize("rows,feature", [(9000, 33), (156249, 64), (156250, 64)])
@pytest.mark.parametrize("n", [5120, 5121, 8192, 8193])
def test_lists_around_the_most_that_one_block_sorts(n, rows, feature):
    from byteir_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(n + rows)
    table, upd = (torch.randint(-8, 8, (k, feature), generator=gen, device="cuda").float() for k in (rows, n))
    ids = torch.randint(0, rows, (n,), generator=gen, device="cuda")
    ids[: n // 4] = ids[0]
    assert torch.equal(ops.index_put_add(table, ids, upd), table.index_add(0, ids, upd))
