"""The quantisers that do more than one thing in a launch, against the calls that they stand for: the one-launch NVFP4 quantiser and
the three operands of an attention layer (bit for bit), at the sizes where tiles, slots and shares of the grid change; K less its mean
in one launch.  That a call takes the one launch is asserted, by the debug-hook build's count of them or by the library's rule."""
import ctypes

import pytest
import torch

from tests.helpers import dynamic_nvfp4, gaussian, hooks_library, takes_one_launch

pytestmark = pytest.mark.gpu


def _u8(t):
    return t.view(torch.uint8)


def _reference(x, cross, reduce, swizzle, layout):
    """global scale and quantiser as two calls of the direct interface"""
    from ac4k_kernel_b200.ops.quant import Ac4kQuantizeOp
    return Ac4kQuantizeOp()(x, cross, reduce, swizzle=swizzle, sf_layout=layout)


def _same(got, want):
    return torch.equal(got[0], want[0]) and torch.equal(_u8(got[1]), _u8(want[1])) and torch.equal(got[2].view(torch.int32), want[2].view(torch.int32))


@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("m,k", [(148, 8192), (257, 8192), (2048, 4160), (4096, 4096), (4097, 4112), (1000, 16384), (12345, 2064), (33000, 1024), (40000, 128),
                                 (8192, 8192)])
def test_rows_of_every_route(m, k, layout):
    """two launches up to 2^24 elements and beyond 2^25, one launch"""
    from ac4k_kernel_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randn((m, k), generator=g, device="cuda", dtype=torch.bfloat16)
    x[m // 2, k // 3] = -77.0                                      # the maximum, once
    assert _same(ops.quantize(x, 0, 1, sf_layout=layout), _reference(x, 0, 1, False, layout))


@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("shape", [
    (520, 8192), (1030, 4800), (1900, 4112), (2048, 4096), (64, 48, 1024), (3, 5, 130, 1280),      # four to seven tiles an SM, ragged along either dimension
    (4097, 4096), (4097, 4112), (5003, 4096), (12345, 2064),      # 14 tiles fit: a few more, each slot used again once
    (8192, 4096), (32000, 1032), (300001, 64), (1100000, 16),     # and up to four times; rows shorter than a tile
])
def test_one_launch_rows(shape, layout):
    hooks = hooks_library()
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)
    x[..., shape[-2] // 2, shape[-1] // 3].flatten()[-1] = -77.0      # the maximum, once
    cross, reduce = len(shape) - 2, len(shape) - 1
    launches = hooks.ac4k_debug_one_launches()
    got = dynamic_nvfp4(hooks, x, cross, reduce, False, layout)
    assert hooks.ac4k_debug_one_launches() == launches + 1
    assert _same(got, _reference(x, cross, reduce, False, layout))


@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("swizzle", [False, True])
@pytest.mark.parametrize("shape", [(1, 700, 3, 128), (2, 1031, 5, 64), (1, 5000, 16, 72), (1, 9000, 16, 128), (3, 130, 1, 8)])
def test_one_launch_columns(shape, swizzle, layout):
    from ac4k_kernel_b200 import ops
    hooks = hooks_library()
    x = (gaussian(shape, seed=shape[1]) * 2).bfloat16().cuda()
    x[0, shape[1] - 1, 0, 1] = 50.0
    launches = hooks.ac4k_debug_one_launches()
    assert _same(dynamic_nvfp4(hooks, x, 3, 1, swizzle, layout), _reference(x, 3, 1, swizzle, layout))
    assert hooks.ac4k_debug_one_launches() == launches + 1
    assert _same(ops.quantize(x, 3, 1, swizzle=swizzle, sf_layout=layout), _reference(x, 3, 1, swizzle, layout))


@pytest.mark.parametrize("fill", [0.0, float("nan"), float("inf"), float("-inf"), 1e-38, -0.0])
@pytest.mark.parametrize("shape,cross,reduce,swizzle", [((2048, 4096), 0, 1, False), ((4100, 4096), 0, 1, False), ((20000, 1032), 0, 1, False),
                                                        ((1000, 4808), 0, 1, False), ((1, 700, 3, 128), 3, 1, True), ((1, 5000, 16, 72), 3, 1, False)])
def test_one_launch_odd_values(shape, cross, reduce, swizzle, fill):
    from ac4k_kernel_b200 import ops
    assert takes_one_launch(shape, cross, reduce, swizzle, torch.cuda.get_device_properties(0).multi_processor_count)
    x = torch.full(shape, fill, device="cuda", dtype=torch.bfloat16)
    assert _same(ops.quantize(x, cross, reduce, swizzle=swizzle), _reference(x, cross, reduce, swizzle, "ac4k"))
    part = tuple(slice(n // 3, None) for n in shape[:-1])
    x[part] = gaussian(tuple(x[part].shape), seed=2).bfloat16().cuda()
    x.view(-1)[5::1001] = fill                                     # blocks with one such value
    assert _same(ops.quantize(x, cross, reduce, swizzle=swizzle), _reference(x, cross, reduce, swizzle, "ac4k"))


@pytest.mark.parametrize("shape,cross,reduce,swizzle", [((2000, 4096), 0, 1, False), ((4100, 4096), 0, 1, False), ((1, 9000, 16, 128), 3, 1, True)])
def test_one_launch_replayed_and_on_two_streams(shape, cross, reduce, swizzle):
    """through the operator: scratch is the allocator's"""
    from ac4k_kernel_b200 import _lib, ops
    assert takes_one_launch(shape, cross, reduce, swizzle, torch.cuda.get_device_properties(0).multi_processor_count)
    xs = [torch.randn(shape, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    want = [_reference(x, cross, reduce, swizzle, "ac4k") for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(ops.quantize(xs[i], cross, reduce, swizzle=swizzle))
    torch.cuda.synchronize()
    assert all(_same(t, want[i]) for i in range(2) for t in got[i])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.quantize(xs[0], cross, reduce, swizzle=swizzle)
    for scale in (1.0, -3.0, 0.5):
        xs[0].copy_(xs[1] * scale)
        graph.replay()
        torch.cuda.synchronize()
        assert _same(out, _reference(xs[0], cross, reduce, swizzle, "ac4k"))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("shape,cross,reduce,swizzle", [((3000, 2048), 0, 1, False), ((4100, 4096), 0, 1, False), ((1, 9000, 16, 128), 3, 1, True)])
def test_one_launch_meets_over_any_scratch(shape, cross, reduce, swizzle):
    """The CTAs' words lie in scratch that holds anything, also what a call before left there, and may begin on any multiple of 4; on
    two streams at once; and in a graph, which is replayed with the words' tag of its capture."""
    hooks = hooks_library()
    xs = [(gaussian(shape, seed=i) * (1 + 3 * i)).cuda() for i in range(2)]
    want = [_reference(x, cross, reduce, swizzle, "ac4k") for x in xs]
    launches, calls = hooks.ac4k_debug_one_launches(), 0
    g = torch.Generator().manual_seed(1)
    for fill in (torch.zeros(1024, dtype=torch.int32), torch.full((1024,), -1, dtype=torch.int32),
                 torch.randint(-2 ** 31, 2 ** 31 - 1, (1024,), generator=g, dtype=torch.int32)):
        for offset in (0, 1):
            scratch = torch.zeros(1026, dtype=torch.int32, device="cuda")
            scratch[offset:offset + 1024] = fill.cuda()
            for i in (0, 1, 0):
                assert _same(dynamic_nvfp4(hooks, xs[i], cross, reduce, swizzle, scratch=scratch[offset:].data_ptr()), want[i])
                calls += 1
            assert scratch[offset + 1024:].sum() == 0 and (offset == 0 or scratch[0] == 0)
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(dynamic_nvfp4(hooks, xs[i], cross, reduce, swizzle))
                calls += 1
    torch.cuda.synchronize()
    assert all(_same(t, want[i]) for i in range(2) for t in got[i])
    x = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = [dynamic_nvfp4(hooks, x, cross, reduce, swizzle) for _ in range(3)]
    calls += 3
    for i in (0, 1, 1, 0):
        x.copy_(xs[i])
        for _ in range(10):
            graph.replay()
        torch.cuda.synchronize()
        assert all(_same(t, want[i]) for t in outs)
    assert hooks.ac4k_debug_one_launches() == launches + calls        # none took another route


def _attention_operands(q, k, v, h_dim, n_dim, lib=None):
    from ac4k_kernel_b200._lib import LIB, last_error
    lib = lib or LIB
    b, h, d, dv = q.shape[0], q.shape[h_dim], q.shape[3], v.shape[3]
    nq, nkv = q.shape[n_dim], k.shape[n_dim]
    dev = {"device": "cuda"}
    made, kp = [], (nkv + 63) // 64 * 64
    for m, c in ((nq, (d + 63) // 64 * 64), (nkv, (d + 63) // 64 * 64), (dv, kp)):
        made.append((torch.empty((b, h, m, c // 2), dtype=torch.uint8, **dev),
                     torch.empty((b, h, (m + 127) // 128, c // 64, 32, 4, 4), dtype=torch.float8_e4m3fn, **dev),
                     torch.empty((), dtype=torch.float32, **dev)))
    scratch = torch.empty(1024, dtype=torch.int32, **dev)
    pointers = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])
    strides = (ctypes.c_int64 * 12)(*[t.stride(i) for t in (q, k, v) for i in (0, h_dim, n_dim, 3)])
    rc = lib.ac4k_attention_quantize_nvfp4(pointers([m[0] for m in made]), pointers([m[1] for m in made]), pointers([m[2] for m in made]),
                                           scratch.data_ptr(), pointers([q, k, v]), strides, b, h, nq, nkv, d, dv,
                                           torch.cuda.current_stream().cuda_stream)
    assert rc == 0, last_error()
    return made


@pytest.mark.parametrize("layout", ["BNHD", "BHND"])
@pytest.mark.parametrize("b,h,nq,nkv,d,dv", [
    (1, 1, 1, 1, 64, 64), (2, 8, 104, 104, 128, 128), (1, 3, 1000, 77, 96, 128), (1, 16, 3000, 4000, 128, 128),
    (1, 1, 130, 129, 80, 72), (3, 5, 65, 257, 40, 128),
    (2, 3, 100, 100, 100, 65),                                      # no tensor map for these strides: a call each
])
def test_attention_operands(layout, b, h, nq, nkv, d, dv):
    n_dim, h_dim = (1, 2) if layout == "BNHD" else (2, 1)
    shape = lambda n, c: (b, n, h, c) if layout == "BNHD" else (b, h, n, c)
    q, k, v = ((gaussian(shape(n, c), seed=n + c + i) * (1 + i)).bfloat16().cuda() for i, (n, c) in enumerate(((nq, d), (nkv, d), (nkv, dv))))
    got = _attention_operands(q, k, v, h_dim, n_dim)
    for t, (x, cross, reduce, swizzle) in zip(got, ((q, n_dim, 3, False), (k, n_dim, 3, False), (v, 3, n_dim, True))):
        assert _same(t, _reference(x, cross, reduce, swizzle, "128x4"))


@pytest.mark.parametrize("fill", [0.0, float("nan"), float("inf"), float("-inf"), 1e-38])
@pytest.mark.parametrize("n,nkv,d", [(130, 200, 128), (6000, 5000, 128), (1000, 900, 40)])
def test_attention_operands_odd_values_on_two_streams(n, nkv, d, fill):
    """one launch for the three, asserted; n = 6000 uses slots again"""
    hooks = hooks_library()
    q, k, v = gaussian((1, n, 16, d), seed=1).cuda(), gaussian((1, nkv, 16, d), seed=2).cuda(), gaussian((1, nkv, 16, d), seed=3).cuda()
    k[:, nkv // 2:] = fill
    v[:, :nkv // 3] = fill
    q.view(-1)[5::1001], k.view(-1)[3::1001], v.view(-1)[7::1001] = fill, fill, fill
    sets = [(q, k, v), (v.clone(), q[:, :nkv].contiguous() if n >= nkv else k, k.clone())]
    want = [[_reference(x, *dims, "128x4") for x, dims in zip(s, ((1, 3, False), (1, 3, False), (3, 1, True)))] for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    launches = hooks.ac4k_debug_one_launches()
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(10):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(_attention_operands(*sets[i], 2, 1, hooks))
    torch.cuda.synchronize()
    assert hooks.ac4k_debug_one_launches() == launches + 20
    assert all(_same(t, w) for i in range(2) for made in got[i] for t, w in zip(made, want[i]))


@pytest.mark.parametrize("d,taken", [(128, True), (100, False), (65, False)])
def test_attention_operands_of_a_fused_projection(d, taken):
    """q, k and v as views into one tensor: right where one launch takes them, refused where the calls it stands for would have taken
    the maximum of other elements"""
    qkv = (gaussian((2, 130, 3, 5, d), seed=d) * torch.tensor([1.0, 4.0, 9.0]).view(1, 1, 3, 1, 1)).bfloat16().cuda()
    views = [qkv[:, :, i] for i in range(3)]
    if not taken:
        with pytest.raises(AssertionError, match="is not dense"):
            _attention_operands(*views, 2, 1)
        return
    for t, want in zip(_attention_operands(*views, 2, 1), _attention_operands(*[v.contiguous() for v in views], 2, 1)):
        assert _same(t, want)


@pytest.mark.parametrize("view", ["one past the start", "every other row", "a head for all", "turned"])
def test_attention_operands_that_are_no_dense_tensors(view):
    """the check for a dense operand, against views of every kind with strides that no tensor map takes"""
    x = gaussian((2, 66, 6, 70), seed=1).cuda()
    dense = gaussian((2, 33, 3, 36), seed=2).cuda()
    v = {"one past the start": x.flatten()[1:1 + dense.numel()].view(dense.shape), "every other row": x[:, ::2, :3, :36],
         "a head for all": dense[:, :, :1].expand(-1, -1, 3, -1), "turned": dense.transpose(1, 2).contiguous().transpose(1, 2)}[view]
    if view in ("one past the start", "turned"):
        got = _attention_operands(v, v, v, 2, 1)
        want = _attention_operands(*[v.clone(memory_format=torch.contiguous_format)] * 3, 2, 1)
        assert all(_same(a, b) for a, b in zip(got, want))
    else:
        with pytest.raises(AssertionError, match="is not dense"):
            _attention_operands(v, v, v, 2, 1)


@pytest.mark.parametrize("layout", ["BNHD", "BHND"])
@pytest.mark.parametrize("b,h,n,d", [(1, 1, 1, 1), (2, 3, 100, 65), (1, 2, 127, 128), (3, 2, 128, 128), (1, 2, 129, 66), (1, 4, 640, 100),
                                     (2, 1, 1000, 96), (1, 3, 1024, 128)])
def test_keys_less_their_mean(layout, b, h, n, d):
    """against the quantiser with a given mean.  With means that are exact, bit for bit.  Else the two means are fp32 sums in different
    orders, so that a mean (of 2 to 4) may differ by an ulp of bf16, 2^-6, and a difference (below 16) that it is taken off by one of
    2^-4 more: `moved`, the bound of what an element of either changes by, and a block's maximum with it"""
    from ac4k_kernel_b200._lib import LIB
    n_dim, h_dim = (1, 2) if layout == "BNHD" else (2, 1)
    shape = (b, n, h, d) if layout == "BNHD" else (b, h, n, d)
    for exact in (True, False):
        k = gaussian(shape, seed=n + d).cuda()
        k = ((k * 8).round() if exact else k * 2 + 3).bfloat16()      # (sums of whole numbers are exact in any order)
        q, v = k.clone(), k.clone()
        mean = k.double().mean(dim=n_dim, keepdim=True).float().bfloat16() if exact else k.mean(dim=n_dim, keepdim=True)
        made = []
        for given in (mean, None):
            outs = []
            for m, block in ((n, 64), (n, 128)):
                outs += [torch.empty((b, h, m, (d + 15) // 16 * 16), dtype=torch.int8, device="cuda"),
                         torch.empty((b, h, (m + block - 1) // block), device="cuda")]
            outs += [torch.empty((b, h, d, (n + 15) // 16 * 16), dtype=torch.uint8, device="cuda"), torch.zeros((b, h, (d + 15) // 16 * 16), device="cuda")]
            st = lambda t: (ctypes.c_int64 * 4)(*[t.stride(i) for i in (0, h_dim, n_dim, 3)])
            ms = (ctypes.c_int64 * 2)(mean.stride(0), mean.stride(h_dim))
            rc = LIB.ac4k_attention_quantize_int8(*[t.data_ptr() for t in outs], q.data_ptr(), st(q), k.data_ptr(), st(k), v.data_ptr(), st(v),
                                                  given.data_ptr() if given is not None else None, ms, b, h, n, n, d, d,
                                                  torch.cuda.current_stream().cuda_stream)
            assert rc == 0
            made.append(outs)
        torch.cuda.synchronize()
        for i in (0, 1, 4, 5):                                       # q and v: the same calls
            assert torch.equal(made[0][i], made[1][i])
        if exact:
            assert torch.equal(made[0][2], made[1][2]) and torch.equal(made[0][3], made[1][3])
        else:
            moved = 2.0 ** -6 + 2.0 ** -4
            assert ((made[0][3] - made[1][3]).abs() <= moved / 127).all()
            rows = made[0][3].repeat_interleave(128, dim=2)[:, :, :n, None]
            assert ((made[0][2].int() - made[1][2].int()).abs() <= 1 + 2 * moved / rows.clamp(min=1e-30)).all()


@pytest.mark.parametrize("fill", [float("nan"), float("inf"), float("-inf"), 3.3895e38, -3.3895e38, 1e-38])
@pytest.mark.parametrize("n,d", [(100, 65), (640, 128)])
def test_keys_less_their_mean_odd_values(n, d, fill):
    """the mean and the codes of a channel with such values, against torch's mean and the quantiser that is given it, bit for bit (the other
    means are exact)"""
    from ac4k_kernel_b200 import _cuda_ops
    from ac4k_kernel_b200.ops.attention import _int8_quantize
    k = (gaussian((2, n, 3, d), seed=n) * 8).round().bfloat16().cuda()
    k[0, n // 3, 1, 5], k[0, n - 1, 1, 5], k[1, 0, 2, d - 1], k[1, n // 2] = fill, fill, fill, fill
    made = []
    for m, block in ((n, 64), (n, 128)):
        made += [torch.empty((2, 3, m, (d + 15) // 16 * 16), dtype=torch.int8, device="cuda"), torch.empty((2, 3, (m + block - 1) // block), device="cuda")]
    made += [torch.empty((2, 3, d, (n + 15) // 16 * 16), dtype=torch.float8_e4m3fn, device="cuda"), torch.empty((2, 3, (d + 15) // 16 * 16), device="cuda")]
    _cuda_ops.attention_quantize_int8(*made, k, k, k, "BNHD")
    codes, scales = _int8_quantize(k, "BNHD", 1, BLOCK_SIZE=128, sub=k.mean(dim=1, keepdim=True))
    assert torch.equal(made[2], codes) and torch.equal(made[3].view(torch.int32), scales.view(torch.int32))
