"""What the entry points refuse before they touch a device: no GPU is needed, and none is used where there is one."""
import ctypes as C

import pytest


@pytest.mark.parametrize("elt_bytes", [-1, 0, 3, 6, 16, 32])
@pytest.mark.parametrize("shape,perm", [((2, 3, 5, 8), (2, 1, 0, 3)), ((2, 3, 5, 8), (3, 1, 2, 0)), ((4, 6), (1, 0)), ((7, 4, 6), (0, 2, 1))])
def test_permute_refuses_other_element_sizes(shape, perm, elt_bytes):
    from byteir_b200 import _native as N
    n = len(shape)
    rc = N.lib().b200_permute(elt_bytes, 0x10000, 0x20000, n, (C.c_int64 * n)(*shape), (C.c_int64 * n)(*perm), None)
    assert rc == -2  # B200_ERR_UNSUPPORTED


# the fixed block of b200_reduce_no_alloc: shapes whose plan would like more of it are served with fewer splits or none
NO_ALLOC = [(1, 27423, 628, "f16"), (20, 161, 21895, "f32"), (20, 161, 21895, "f16"), (53, 37, 1490, "f32"), (64, 128, 1025, "f16"),
            (1, 256, 33001, "f16"), (64, 512, 4097, "f32"), (1, 32768, 1023, "bf16")]


@pytest.mark.parametrize("A,B,C,dt,served", [s + (True,) for s in NO_ALLOC] + [(580, 64, 256, "f16", False), (590, 200, 256, "f16", False)])
def test_no_alloc_serves_by_shape(A, B, C, dt, served):
    from byteir_b200 import _native as N
    # without tensors a shape that is served gets as far as the check for them (or for a device)
    rc = N.lib().b200_reduce_no_alloc(0, {"f32": N.F32, "f16": N.F16, "bf16": N.BF16}[dt], None, None, A, B, C, None)
    assert (rc != -3) == served, rc  # B200_ERR_WORKSPACE


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["sum", "max"])
@pytest.mark.parametrize("A,B,C,dt", NO_ALLOC)
def test_no_alloc_results(A, B, C, dt, op):
    import torch
    from byteir_b200 import _native as N
    t = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dt]
    gen = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randn((A, B, C), generator=gen, device="cuda").to(t)
    if op == "max":
        x = -x.abs() - 0.25  # no zeros but the planted ones: a normal value rounds to zero now and then
        x[:, B // 3, ::5] = 0.0
        x[:, B // 2, ::10] = -0.0
    got = torch.empty((A, C), device="cuda", dtype=t)
    N.check(N.lib().b200_reduce_no_alloc(N.REDUCE_SUM if op == "sum" else N.REDUCE_MAX, {"f32": N.F32, "f16": N.F16, "bf16": N.BF16}[dt],
                                         x.data_ptr(), got.data_ptr(), A, B, C, torch.cuda.current_stream().cuda_stream), "no_alloc")
    if op == "max":
        want = x.amax(1)
        want[:, ::5] = 0.0
        want[:, ::10] = -0.0
        assert torch.equal(got, want) and torch.equal(torch.signbit(got), torch.signbit(want))
        return
    # one rounding to the type, and f32 sums of at most B / 8 additions in a chain, then a tree
    want, mag = torch.zeros((A, C), dtype=torch.float64, device="cuda"), torch.zeros((A, C), dtype=torch.float64, device="cuda")
    for i in range(0, B, 256):
        want += x[:, i:i + 256].double().sum(1)
        mag += x[:, i:i + 256].double().abs().sum(1)
    bound = {"f32": 0.0, "f16": 2.0**-11, "bf16": 2.0**-8}[dt] * want.abs() * 1.001 + 2.0**-24 * (B / 8 + 32) * mag
    assert bool(((got.double() - want).abs() <= bound).all())


# a module's reduction takes the scratch that its launch uses: none where the splits fold through distributed shared memory
@pytest.mark.gpu
@pytest.mark.parametrize("shape,used", [((64, 1000, 256), False), ((1, 32768, 1024), True)])
def test_module_takes_the_scratch_that_its_launch_uses(shape, used):
    import torch
    from byteir_b200 import _native as N, brt
    from test_brt_host import reduce_mlir
    sizes = []

    def alloc(size):
        sizes.append(size)
        return torch.cuda.caching_allocator_alloc(max(size, 1))

    declared = N.lib().b200_reduce_workspace_bytes(N.REDUCE_SUM, N.F16, *shape)
    assert declared > 0
    out_shape = (shape[0], shape[2])
    s = brt.Session("cuda", alloc_func=alloc, free_func=torch.cuda.caching_allocator_delete)
    s.load_from_memory(reduce_mlir("ReduceSumOp_f16_f16", "f16", shape, out_shape, "dense<1> : tensor<1xi64>"))
    x, out = torch.randn(shape, device="cuda").half(), torch.empty(out_shape, device="cuda", dtype=torch.float16)
    request = s.new_request(torch.cuda.current_stream().cuda_stream)
    request.bind_args([(0, x.data_ptr()), (1, out.data_ptr())])
    request.finish_io_binding()
    request.run()
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), x.float().sum(1), rtol=2e-2, atol=1e-2)
    assert sum(sizes) == ((declared + 255) // 256 * 256 if used else 0)
    request.close()
    s.close()
