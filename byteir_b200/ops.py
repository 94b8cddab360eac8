"""Host-side mirror of the ByRE compute ops of the default CUDA provider, over
torch CUDA tensors.  torch supplies device memory and the current stream only;
every op runs the sm_100a kernels through the C ABI.  The steps of a call
(checks, output and workspace memory, launch) are native: csrc/pyext/ops_ext.cc.

Semantics follow the reference op kernels
(runtime/lib/backends/cuda/providers/default/{reduction,indexing,
tensor_manipulate}): ReduceSumOp / ReduceMaxOp with a `dimensions` attribute
(consecutive dims), IndexSelectOp / IndexPutOp with `dim`, TransposeOp with
`permutation`.
"""
import ctypes as C

import torch

from . import _native as N

_X = N.ops_ext()
_DT = {torch.float32: N.F32, torch.float16: N.F16, torch.bfloat16: N.BF16}


def _dt(t):
    try:
        return _DT[t.dtype]
    except KeyError:
        raise TypeError(f"unsupported element type {t.dtype}") from None


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _need_cuda(*ts):
    for t in ts:
        if not t.is_cuda:
            raise ValueError("byteir_b200 ops take CUDA tensors; there is no CPU path")
        if not t.is_contiguous():
            raise ValueError("tensors must be contiguous (ByRE memrefs are)")


def reduce_sum(x, dimensions, out=None, workspace=None):
    return _X.reduce(N.REDUCE_SUM, x, dimensions, out, workspace)


def reduce_max(x, dimensions, out=None, workspace=None):
    return _X.reduce(N.REDUCE_MAX, x, dimensions, out, workspace)


def reduce_sum_to_f32(x, dimensions, out=None, workspace=None):
    """Unrounded f32 partial of a sum (the operand of a later all-reduce)."""
    return _X.reduce_sum_to_f32(x, dimensions, out, workspace)


def cast_from_f32(x, dtype, out=None):
    _need_cuda(x)
    if out is None:
        out = torch.empty(x.shape, dtype=dtype, device=x.device)
    N.check(N.lib().b200_cast_from_f32(_DT[dtype], x.data_ptr(), out.data_ptr(), x.numel(), _stream()),
            "b200_cast_from_f32")
    return out


def index_select(x, index, dim, out=None, status=None, path=0):
    return _X.index_select(x, index, dim, out, status, path)


def index_put_add(x, index, update, dim=0, out=None, workspace=None, status=None):
    """out = x; out[index[i], ...] += update[i, ...] (IndexPutOp, accumulate)."""
    return _X.index_put_add(x, index, update, dim, out, workspace, status)


def transpose(x, permutation, out=None):
    return _X.transpose(x, permutation, out)


def transpose_batched(x, out=None, path=0):
    """[batch, rows, cols] -> [batch, cols, rows]"""
    return _X.transpose_batched(x, out, path)


def flash_attn_fwd(q, k, v, softmax_scale, causal=True, window=(-1, -1), out=None, lse=None):
    """q, k, v: [B, S, H, D] (last dim contiguous), f16 or bf16.  Returns (out, softmax_lse[B, H, Sq])."""
    return _X.flash_attn_fwd(q, k, v, softmax_scale, causal, window, out, lse)


def flash_attn_bwd(dout, q, k, v, out, lse, softmax_scale, causal=True, window=(-1, -1),
                   dq=None, dk=None, dv=None, d_softmax_sum=None):
    """Gradients of flash_attn_fwd.  Returns (dq, dk, dv); dq/dk/dv share the strides of q/k/v."""
    return _X.flash_attn_bwd(dout, q, k, v, out, lse, softmax_scale, causal, window, dq, dk, dv, d_softmax_sum)


def kvcache_params(q, kcache, vcache, knew, vnew, out, softmax_scale, causal=True, window=(-1, -1)):
    """The packed arguments of run_flash_attn_kvcache for tensors laid out [B, S, H, D]."""
    p = N.FlashKvCacheParams()
    for name, t in (("q", q), ("k", kcache), ("v", vcache), ("knew", knew), ("vnew", vnew), ("o", out)):
        bs, rs, hs = (t.stride(0), t.stride(1), t.stride(2)) if t is not None else (0, 0, 0)
        setattr(p, name + "_batch_stride", bs)
        setattr(p, name + "_row_stride", rs)
        setattr(p, name + "_head_stride", hs)
    p.b, p.seqlen_q, p.h, p.d = q.shape
    p.seqlen_k, p.h_k = kcache.shape[1], kcache.shape[2]
    p.seqlen_knew = knew.shape[1] if knew is not None else 0
    p.d_rounded = (p.d + 31) // 32 * 32
    p.seqlen_q_rounded = (p.seqlen_q + 127) // 128 * 128
    p.seqlen_k_rounded = (p.seqlen_k + 127) // 128 * 128
    p.softmax_scale = softmax_scale
    p.window_size_left = window[0]
    p.window_size_right = 0 if causal else window[1]
    return p


def flash_attn_kvcache(q, kcache, vcache, knew=None, vnew=None, seqlens_k=None, softmax_scale=None,
                       causal=True, window=(-1, -1), out=None, lse=None, workspace=None):
    """One decode step: append knew/vnew [B, S_new, H_k, D] to the caches [B, S_max, H_k, D] at row
    seqlens_k[b] (i32 [B]; None = the cache is full and nothing is appended) and attend q [B, Sq, H, D]
    to the rows in use.  The caches are updated in place.  Returns (out, softmax_lse[B, H, Sq]).

    Where blocks share the keys of the batch equally (large caches, head dims 64 and 128) the parts in which a
    sequence is summed follow from the lengths of all sequences.  The same batch gives the same bits; the same
    sequence beside others gives the same result to within the rounding of 16-bit probabilities."""
    return _X.flash_attn_kvcache(q, kcache, vcache, knew, vnew, seqlens_k, softmax_scale, causal, window, out, lse,
                                 workspace)


class ShardedSum:
    """Exchange step of a sum whose reduced axis is sharded over ranks (one kernel over NVLink peer
    memory instead of all-reduce + cast).  `peer_inbox` / `peer_flags`: device addresses per rank of
    memory all ranks can write (e.g. from torch symmetric memory), `counter`: a zeroed device uint32."""

    def __init__(self, rank, world, n, peer_inbox, peer_flags, counter, status=None):
        self.rank, self.world, self.n = rank, world, n
        self._inbox = (C.c_void_p * world)(*peer_inbox)
        self._flags = (C.c_void_p * world)(*peer_flags)
        self._counter, self._status = counter, status

    def __call__(self, partial, out):
        rc = N.lib().b200_sharded_sum_finish(
            _dt(out), partial.data_ptr(), self._inbox, self._flags, self.rank, self.world, self.n,
            self._counter.data_ptr(), out.data_ptr(),
            self._status.data_ptr() if self._status is not None else None, _stream())
        N.check(rc, "b200_sharded_sum_finish")
        return out


class ShardedSumSwitch:
    """The same exchange with the sum taken inside the NVSwitch (multimem.ld_reduce over a multicast
    mapping of symmetric memory).  `own_slots`: this rank's float[2][n] in symmetric memory;
    `multicast_slots`: the multicast address of the same range; `peer_flags`, `counter` as above."""

    def __init__(self, rank, world, n, own_slots, multicast_slots, peer_flags, counter, status=None):
        self.rank, self.world, self.n = rank, world, n
        self._own, self._mc = own_slots, multicast_slots
        self._flags = (C.c_void_p * world)(*peer_flags)
        self._counter, self._status = counter, status

    def __call__(self, partial, out):
        rc = N.lib().b200_sharded_sum_finish_nvls(
            _dt(out), partial.data_ptr(), self._own, self._mc, self._flags, self.rank, self.world, self.n,
            self._counter.data_ptr(), out.data_ptr(),
            self._status.data_ptr() if self._status is not None else None, _stream())
        N.check(rc, "b200_sharded_sum_finish_nvls")
        return out
