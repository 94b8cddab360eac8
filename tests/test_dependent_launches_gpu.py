"""Kernels launched early (programmatic dependent launch) one behind the other, in a stream and as a captured graph: what a
kernel leaves has to be complete when the next one reads it.  Every pass has other inputs in the same buffers, so that a
value left over from the pass before is a wrong one."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from test_flash_attn_gpu import _dev, _host, _mk

pytestmark = pytest.mark.gpu


def _passes(fill, chain, check, graph):
    """`fill(i)` brings pass i's inputs, `chain()` enqueues the kernels and names their outputs, `check(i, copies)`"""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        fill(0)
        chain()  # the allocator's blocks and the kernels are there before a capture
        if graph:
            stream.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                outs = chain()
        for i in range(4):
            fill(i)
            if graph:
                g.replay()
            else:
                outs = chain()
            copies = [o.clone() for o in outs]
            stream.synchronize()
            check(i, copies)


# every sequence at most one step of 64 keys, in a cache large enough for equal shares: no row has two partial results and
# every block of the merge has nothing to merge
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("b,h,hk,d,cap", [(8, 32, 8, 128, 4000), (64, 16, 4, 64, 1200)])
def test_short_sequences_then_dependents_of_the_decode_step(b, h, hk, d, cap, graph):
    from byteir_b200 import ops
    rng = np.random.default_rng(b)

    def cache():  # only the rows that can be in use have values
        c = np.zeros((b, cap, hk, d), np.uint16)
        c[:, :64] = _mk(rng, (b, 64, hk, d), "bf16")
        return c

    ins = [[_mk(rng, (b, 1, h, d), "bf16"), cache(), cache(), _mk(rng, (b, 1, hk, d), "bf16"), _mk(rng, (b, 1, hk, d), "bf16"),
            rng.integers(0, 63, b).astype(np.int32)] for _ in range(4)]
    bufs = [_dev(t) for t in ins[0][:5]] + [torch.from_numpy(ins[0][5]).cuda()]
    src = [[_dev(t) for t in one[:5]] + [torch.from_numpy(one[5]).cuda()] for one in ins]
    ids = torch.arange(b - 1, -1, -1, device="cuda")
    q, kc, vc, kn, vn, lens = bufs
    out, lse = torch.empty_like(q), torch.empty((b, h, 1), dtype=torch.float32, device="cuda")

    def fill(i):
        for dst, s in zip(bufs, src[i]):
            dst.copy_(s)

    def chain():
        ops.flash_attn_kvcache(q, kc, vc, kn, vn, lens, out=out, lse=lse)
        rows = out.view(b, h * d)
        return (ops.index_select(rows, ids, 0), ops.transpose(rows, [1, 0]), ops.reduce_max(lse.view(b, h), [1]),
                ops.index_select(kc.view(b, -1), ids, 0))

    def check(i, got):
        want_k, want_v = ins[i][1].copy(), ins[i][2].copy()
        want, want_lse = O.flash_attn_kvcache(ins[i][0], want_k, want_v, ins[i][3], ins[i][4], ins[i][5], d ** -0.5, True)
        w = O.to_f32(want).reshape(b, h * d)
        np.testing.assert_allclose(O.to_f32(_host(got[0])), w[::-1], rtol=2e-2, atol=1e-2)
        np.testing.assert_allclose(O.to_f32(_host(got[1])), w.T, rtol=2e-2, atol=1e-2)
        np.testing.assert_allclose(got[2].cpu().numpy(), want_lse.reshape(b, h).max(1), rtol=1e-3, atol=1e-3)
        assert np.array_equal(_host(got[3]).reshape(want_k.shape), want_k[::-1])

    _passes(fill, chain, check, graph)


# the backward's passes share the row sums, which another kernel leaves, and the caller's buffers of the pass before
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("b,sq,sk,h,hk,d,window", [(2, 300, 420, 8, 4, 128, (-1, -1)), (1, 1100, 1100, 16, 16, 64, (200, 0)),
                                                   (3, 2048, 2048, 24, 8, 128, (-1, -1))])
def test_backward_passes_in_the_same_buffers(b, sq, sk, h, hk, d, window, graph):
    from byteir_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(sq)
    shapes = [(b, sq, h, d), (b, sk, hk, d), (b, sk, hk, d), (b, sq, h, d)]
    src = [[torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in shapes] for _ in range(4)]
    bufs = [torch.empty_like(t) for t in src[0]]
    q, k, v, do = bufs
    o, lse, dsum = torch.empty_like(q), torch.empty((b, h, sq), device="cuda"), torch.empty((b, h, (sq + 127) // 128 * 128), device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]

    def step(q, k, v, do, **kw):
        fwd, bwd = ({n: kw[n] for n in names if n in kw} for names in (("out", "lse"), ("dq", "dk", "dv", "d_softmax_sum")))
        out, l2 = ops.flash_attn_fwd(q, k, v, d ** -0.5, True, window, **fwd)
        return (out, l2) + tuple(ops.flash_attn_bwd(do, q, k, v, out, l2, d ** -0.5, True, window, **bwd))

    want = []
    for one in src:
        want.append(step(*one))
        torch.cuda.synchronize()

    def fill(i):
        for dst, s in zip(bufs, src[i]):
            dst.copy_(s)

    def chain():
        got = step(q, k, v, do, out=o, lse=lse, dq=grads[0], dk=grads[1], dv=grads[2], d_softmax_sum=dsum)
        return got[:2] + tuple(ops.transpose(t, [0, 2, 1, 3]) for t in got[2:])

    def check(i, got):
        for g, w in zip(got, want[i][:2] + tuple(t.transpose(1, 2) for t in want[i][2:])):
            assert torch.equal(g, w.contiguous())

    _passes(fill, chain, check, graph)


# dQ in the place of Q or dO: the dK/dV pass has read them before it is written
@pytest.mark.parametrize("over", ["q", "dout"])
def test_dq_in_the_place_of_an_input(over):
    from byteir_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn((2, 1500, 20, 128), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4))
    out, lse = ops.flash_attn_fwd(q, k, v, 128 ** -0.5, True)
    want = ops.flash_attn_bwd(do, q, k, v, out, lse, 128 ** -0.5, True)
    torch.cuda.synchronize()
    for _ in range(3):
        q2, do2 = q.clone(), do.clone()
        got = ops.flash_attn_bwd(do2, q2, k, v, out, lse, 128 ** -0.5, True, dq=q2 if over == "q" else do2)
        assert all(torch.equal(g, w) for g, w in zip(got, want))
