"""The routes that small and odd-sized calls take, at the sizes where they change: the quantisers' single-launch kernels,
the block quantiser on odd head dimensions, the decode GEMM's division of the activation rows among K slices, and the
operators' native host side.  Quantisers are compared bit for bit."""
import pytest
import torch

from oracle import emulation as E
from tests.helpers import gaussian


def _u8(t):
    return t.view(torch.uint8)


def _two_calls(x, cross, reduce, swizzle, layout):
    """global scale and quantiser as two calls of the direct interface"""
    from ac4k_kernel_b200.ops.quant import Ac4kQuantizeOp
    return Ac4kQuantizeOp()(x, cross, reduce, swizzle=swizzle, sf_layout=layout)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("shape,cross,reduce,swizzle", [
    ((1, 16), 0, 1, False), ((1, 8192), 0, 1, False), ((3, 2064), 0, 1, False),      # one CTA; K not a multiple of 64
    ((16, 8192), 0, 1, False), ((17, 8192), 0, 1, False),                            # the last of one cluster, the first of two launches
    ((50, 8192), 0, 1, False), ((666, 4096), 0, 1, False), ((129, 80), 0, 1, False),
    ((4096, 2560), 0, 1, False), ((2049, 4096), 0, 1, False),                        # tiled, with and without a ragged tile
    ((4100, 4096), 0, 1, False),                                                     # above 2^24 elements: atomic maximum
    ((2, 5, 3, 64), 1, 3, False), ((2, 300, 3, 128), 1, 3, False), ((1, 2000, 16, 128), 1, 3, False),
    ((2, 100, 3, 128), 3, 1, True), ((1, 64, 2, 80), 3, 1, True),                    # rows contiguous along the cross dimension
    ((2, 33, 3, 65), 3, 1, True), ((7, 33), 0, 1, False), ((9, 40), 1, 0, False),    # strided kernel
])
def test_scale_and_codes_in_one_call(shape, cross, reduce, swizzle, layout):
    from ac4k_kernel_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16) * 3
    want = _two_calls(x, cross, reduce, swizzle, layout)
    got = ops.quantize(x, cross, reduce, swizzle=swizzle, sf_layout=layout)
    torch.cuda.synchronize()
    assert got[2].shape == want[2].shape == () and torch.equal(got[2], want[2])
    assert got[0].shape == want[0].shape and torch.equal(got[0], want[0])
    assert got[1].shape == want[1].shape and torch.equal(_u8(got[1]), _u8(want[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [0.0, float("nan"), float("inf"), 1e-38])
@pytest.mark.parametrize("rows", [2, 40])
def test_odd_values_in_one_call(rows, fill):
    from ac4k_kernel_b200 import ops
    for whole in (True, False):
        x = torch.full((rows, 8192), fill, device="cuda", dtype=torch.bfloat16)
        if not whole:
            x[:, 100:] = gaussian((rows, 8092), seed=3).cuda()
        want = _two_calls(x, 0, 1, False, "ac4k")
        got = ops.quantize(x, 0, 1)
        assert torch.equal(got[2].view(torch.int32), want[2].view(torch.int32))
        assert torch.equal(got[0], want[0]) and torch.equal(_u8(got[1]), _u8(want[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp8e4m3", "int8"])
@pytest.mark.parametrize("b,k,h,d", [(1, 1, 1, 1), (2, 15, 3, 65), (2, 16, 1, 64), (1, 17, 2, 63), (1, 100, 12, 65), (1, 128, 2, 128),
                                     (1, 512, 2, 64), (1, 1023, 1, 100), (1, 1024, 2, 17), (1, 1025, 2, 65), (1, 1025, 2, 66),
                                     (300, 20, 1, 17), (300, 130, 1, 17), (40, 64, 1, 63), (8, 64, 1, 63),       # one launch; a warp a row; one; a warp a row
                                     (150, 16, 4, 640), (3, 770, 1, 5000), (1, 1024, 1, 13000)])                 # four launches, one, four
def test_columns_contiguous(b, k, h, d, precision):
    """[B, N, H, D] along N: one launch over a short N where there are columns for its CTAs and not too many, else four launches,
    or, where D is odd, a warp for each row"""
    from ac4k_kernel_b200 import ops
    x = (gaussian((b, k, h, d), seed=k + d) * 2).bfloat16().cuda()
    x[:, :, :, d // 2] = 0                                             # a column of zeros: 0 * inf
    if precision == "int8":
        y, s = ops.quantize(x, 3, 1, precision="int8")
        ry, rs = E.quantize_int8_ref(x.cpu(), 3, 1)
    else:
        y, s = ops.quantize(x, 3, 1, swizzle=True, max_scale=2.25, precision="fp8e4m3")
        ry, rs = E.quantize_fp8_ref(x.cpu(), 3, 1, 2.25, swizzle=True)
    assert y.shape == ry.shape and torch.equal(_u8(y).cpu(), _u8(ry))
    assert torch.equal(s.cpu(), rs)


@pytest.mark.gpu
@pytest.mark.parametrize("b,n,h,d,layout,block", [(11, 100, 12, 65, "BNHD", 128), (1, 129, 2, 1, "BHND", 64), (1, 130, 1, 127, "BNHD", 16),
                                                 (1, 65, 2, 131, "BHND", 128), (2, 40, 1, 66, "BNHD", 32),
                                                 (1, 1007, 5, 66, "BNHD", 16), (2, 1000, 5, 131, "BHND", 32)])     # four warps a block
def test_block_quantiser_any_head_dimension(b, n, h, d, layout, block):
    from ac4k_kernel_b200.ops.attention import _int8_quantize
    x = (gaussian((b, n, h, d) if layout == "BNHD" else (b, h, n, d), seed=n + d) * 3).bfloat16().cuda()
    dim = 1 if layout == "BNHD" else 2
    mean = x.mean(dim=dim, keepdim=True)
    for sub in (None, mean):
        y, s = _int8_quantize(x, layout, dim, BLOCK_SIZE=block, sub=sub)
        ry, rs = E.quantize_int8_block_ref(x if sub is None else x - sub, layout, block)
        assert torch.equal(s, rs) and torch.equal(y, ry)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["ac4k", "128x4"])
@pytest.mark.parametrize("m,n,k", [(1, 128, 1024), (3, 200, 4096), (5, 136, 8192), (13, 512, 2048), (16, 8192, 1024), (17, 512, 4096),
                                   (31, 8192, 8192), (33, 264, 4096), (50, 8192, 8192), (63, 384, 4096), (64, 20000, 1024)])
def test_decode_rows_over_slices(m, n, k, layout):
    """4, 2 or 1 K slices, activation rows that do not divide among them"""
    from ac4k_kernel_b200 import ops
    a, b = gaussian((m, k), seed=m).cuda(), (gaussian((n, k), seed=n) * 0.05).bfloat16().cuda()
    qa, qb = ops.quantize(a, 0, 1, sf_layout=layout), ops.quantize(b, 0, 1, sf_layout=layout)
    bias = gaussian((1, n), seed=5).cuda()
    out = torch.full((m, n), float("nan"), device="cuda")
    assert ops.linear(*qa, *qb, bias=bias, out=out) is out
    want = E.dequantize_nvfp4_ref(*qa).double() @ E.dequantize_nvfp4_ref(*qb).double().T + bias.double()
    # fp32 sums of k products: a few 2^-24 of their size each
    assert float((out.double() - want).norm() / want.norm()) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["int8+fp8e4m3", "nvfp4"])
@pytest.mark.parametrize("nq,nkv,d", [(256, 515, 128), (300, 1100, 128), (130, 640, 64)])
def test_one_or_two_query_tiles_per_block(nq, nkv, d, precision):
    """160 heads take two query tiles per block, two of them alone one: the same arithmetic per row, so the same bits.
    (Several key tiles: warps of a group may run a tile ahead of one another.)"""
    from ac4k_kernel_b200 import _cuda_ops, ops
    from ac4k_kernel_b200.ops.attention import _int8_quantize
    h = 160
    q, k, v = (gaussian((1, n, h, d), seed=n + i).cuda() for i, n in enumerate((nq, nkv, nkv)))
    if precision == "nvfp4":
        args = [*ops.quantize(q, 1, 3, sf_layout="128x4"), *ops.quantize(k, 1, 3, sf_layout="128x4"),
                *ops.quantize(v, 3, 1, swizzle=True, sf_layout="128x4")]
        kernel = _cuda_ops.mha_nvfp4_fwd
    else:
        v8, vs = ops.quantize(v, 3, 1, swizzle=True, max_scale=2.25, precision="fp8e4m3")
        args = [*_int8_quantize(q, "BNHD", 1, BLOCK_SIZE=64), 64, *_int8_quantize(k, "BNHD", 1, BLOCK_SIZE=128), 128, v8, vs]
        kernel = _cuda_ops.mha_int8_x_fp8_fwd

    def run(heads):
        cut = [t[:, :heads].contiguous() if isinstance(t, torch.Tensor) and t.dim() >= 3 else t for t in args]
        o = torch.full((1, heads, nq, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        kernel(o, *cut, d ** -0.5)
        return o

    many = [run(h) for _ in range(5)]
    few = run(2)
    assert all(torch.equal(many[0], m) for m in many)
    assert torch.equal(many[0][:, :2], few) and not bool(torch.isnan(few.float()).any())


@pytest.mark.gpu
@pytest.mark.parametrize("d", [128, 96, 80, 72, 512, 1024, 1032])
def test_rope_near_rounding_boundaries(d):
    """Values whose products land on and beside the boundaries between two bf16 values, tiny and huge ones, zeros,
    infinities and NaN: all bits as the fp64 arithmetic gives them."""
    from ac4k_kernel_b200 import ops
    s, n = 40, 3
    g = torch.Generator().manual_seed(d)
    x = torch.randn((1, s, n, d), generator=g).bfloat16()
    x[0, 0] = 0
    x[0, 1, 0, :8] = torch.tensor([1e-38, -1e-38, 3e38, -3e38, float("inf"), float("nan"), 1e-30, 0.0]).bfloat16()
    freqs = E.rope_params_ref(64, d)
    freqs[3] = torch.complex(torch.full((d // 2,), 1 + 2.0 ** -9, dtype=torch.float64), torch.zeros(d // 2, dtype=torch.float64))
    freqs[4] = freqs[3] * (1 + 2.0 ** -40)                             # beside a tie: fp32 cannot tell
    freqs[5] = torch.complex(torch.full((d // 2,), 1e-42, dtype=torch.float64), torch.full((d // 2,), 1e300, dtype=torch.float64))
    grid = torch.tensor([[s, 1, 1]], dtype=torch.int32)
    got = ops.rope3d(x.cuda(), grid.cuda(), freqs.cuda()).cpu()
    want = E.rope3d_ref(x, grid, freqs)
    nan = torch.isnan(want.float())
    assert torch.equal(nan, torch.isnan(got.float()))
    assert torch.equal(got.view(torch.int16)[~nan], want.view(torch.int16)[~nan])


@pytest.mark.gpu
@pytest.mark.parametrize("d", [128, 72, 512, 1032])
def test_rope_zero_pairs(d):
    """Pairs of zeros of either sign beside others, under usual, negative, zero, tiny, infinite and NaN factors"""
    from ac4k_kernel_b200 import ops
    s, n = 12, 5
    g = torch.Generator().manual_seed(d)
    x = torch.randn((1, s, n, d), generator=g).bfloat16()
    pairs = torch.rand((1, s, n, d // 2, 1), generator=g) < 0.6
    zero = torch.where(torch.rand(x.shape, generator=g) < 0.5, 0.0, -0.0).bfloat16()
    x = torch.where(pairs.expand(-1, -1, -1, -1, 2).reshape(x.shape), zero, x)
    x[0, :, 0], x[0, :, 1, ::2] = zero[0, :, 0], zero[0, :, 1, ::2]      # whole heads; single zeros
    freqs = E.rope_params_ref(s, d)
    for row, f in enumerate((-1 + 0j, 0j, complex(-0.0, -0.0), 1e-35 - 1e-42j, complex(float("inf"), 1), complex(float("nan"), 0), -1e-320 + 1j)):
        freqs[row + 1] = torch.full((d // 2,), f, dtype=torch.complex128)
    grid = torch.tensor([[s, 1, 1]], dtype=torch.int32)
    got = ops.rope3d(x.cuda(), grid.cuda(), freqs.cuda()).cpu()
    want = E.rope3d_ref(x, grid, freqs)
    nan = torch.isnan(want.float())
    assert bool(nan.any()) and torch.equal(nan, torch.isnan(got.float()))
    assert torch.equal(got.view(torch.int16)[~nan], want.view(torch.int16)[~nan])


def _milliseconds(fn):
    """median of nine single calls on the device"""
    t = []
    for i in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        if i >= 3:
            t.append(a.elapsed_time(b))
    return sorted(t)[4]


@pytest.mark.gpu
def test_rope_zeros_take_no_longer():
    """Zeros took the fp32 and the fp64 form one after the other: 1.7 times the time of other values, not 1.0"""
    from ac4k_kernel_b200 import ops
    grid, freqs = torch.tensor([[21, 30, 40]], dtype=torch.int32, device="cuda"), E.rope_params_ref(64, 128).cuda()
    x = torch.randn((1, 25200, 40, 128), device="cuda", dtype=torch.bfloat16)
    usual = _milliseconds(lambda: ops.rope3d(x, grid, freqs))
    x[..., 4::8], x[..., 5::8] = 0, 0                                    # a pair of every vector of eight
    assert _milliseconds(lambda: ops.rope3d(x, grid, freqs)) < 1.35 * usual


@pytest.mark.gpu
@pytest.mark.parametrize("s,n,d", [(1, 128, 256), (3, 40, 128), (100, 33, 256), (2, 40, 40), (1500, 8, 64), (1, 60, 304), (5, 9, 1024), (2, 1, 8)])
def test_rope_few_positions(s, n, d):
    """One to eight warps per position, by the number of positions and of vectors in one"""
    from ac4k_kernel_b200 import ops
    x = gaussian((2, s, n, d), seed=s + d)
    grid = torch.tensor([[s, 1, 1], [max(1, s // 2), 1, 1]], dtype=torch.int32)
    freqs = E.rope_params_ref(s, d)
    got = ops.rope3d(x.cuda(), grid.cuda(), freqs.cuda()).cpu()
    assert torch.equal(got.view(torch.int16), E.rope3d_ref(x, grid, freqs).view(torch.int16))


def _graph_microseconds(fn, calls=20):
    """median time of one of `calls` calls replayed from a graph"""
    fn()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(calls):
            fn()
    return _milliseconds(g.replay) / calls * 1e3


@pytest.mark.gpu
def test_rope_few_positions_take_few_rounds():
    """16 positions of 128 heads x 256 took 0.57 of the time of 1000 when a position had one warp; 0.22 with eight"""
    from ac4k_kernel_b200 import ops
    t, freqs = [], E.rope_params_ref(1024, 256).cuda()
    for s in (16, 1000):
        x, grid = gaussian((1, s, 128, 256), seed=s).cuda(), torch.tensor([[s, 1, 1]], dtype=torch.int32, device="cuda")
        t.append(_graph_microseconds(lambda: ops.rope3d(x, grid, freqs)))
    assert t[0] < 0.4 * t[1]


@pytest.mark.gpu
def test_decode_rows_of_one_slice_take_no_longer():
    """64 activation rows against one, one K slice: 1.4 times the time, 1.7 with the rows stored one at a time"""
    from ac4k_kernel_b200 import ops
    w = ops.quantize((gaussian((512, 512), seed=1) * 0.05).bfloat16().cuda(), 0, 1, sf_layout="128x4")
    t = []
    for m in (64, 1):
        a = ops.quantize(gaussian((m, 512), seed=m).cuda(), 0, 1, sf_layout="128x4")
        t.append(_graph_microseconds(lambda: ops.linear(*a, *w), calls=100))
    assert t[0] < 1.58 * t[1]


@pytest.mark.gpu
def test_short_token_blocks_take_no_longer():
    """[1, 4096, 16, 66] in blocks of 16 tokens against blocks of 128: twice the time with sixteen warps a block, 1.1 with four"""
    from ac4k_kernel_b200.ops.attention import _int8_quantize
    x = gaussian((1, 4096, 16, 66), seed=1).cuda()
    t = [_graph_microseconds(lambda: _int8_quantize(x, "BNHD", 1, BLOCK_SIZE=block)) for block in (16, 128)]
    assert t[0] < 1.5 * t[1]


@pytest.mark.gpu
def test_one_column_takes_no_cta_of_64():
    """A column of 1024 values by itself: as long as 64 of them when a CTA walked it alone, a third of that with a warp"""
    from ac4k_kernel_b200 import ops
    t = []
    for m in (1, 64):
        x = gaussian((1024, m), seed=m).cuda()
        t.append(_graph_microseconds(lambda: ops.quantize(x, 1, 0, precision="fp8e4m3")))
    assert t[0] < 0.6 * t[1]


@pytest.mark.gpu
def test_query_tiles_by_the_time_they_take():
    """190 heads of three query tiles against four: 1.02 of the time with one tile per block, 0.89 with two"""
    from ac4k_kernel_b200 import _cuda_ops, ops
    from ac4k_kernel_b200.ops.attention import _int8_quantize
    t = []
    for nq in (384, 512):
        q, k, v = (gaussian((1, n, 190, 128), seed=n + i).cuda() for i, n in enumerate((nq, 1024, 1024)))
        v8, vs = ops.quantize(v, 3, 1, swizzle=True, max_scale=2.25, precision="fp8e4m3")
        args = [*_int8_quantize(q, "BNHD", 1, BLOCK_SIZE=64), 64, *_int8_quantize(k, "BNHD", 1, BLOCK_SIZE=128), 128, v8, vs]
        o = torch.empty((1, 190, nq, 128), dtype=torch.bfloat16, device="cuda")
        t.append(_graph_microseconds(lambda: _cuda_ops.mha_int8_x_fp8_fwd(o, *args, 128 ** -0.5), calls=5))
    assert t[0] < 0.95 * t[1]


@pytest.mark.gpu
def test_narrow_rows_fill_the_chip():
    """q of attention, rows of 128 features, against as many bytes in long rows: 1.16 - 1.19 of the time with four CTAs of the
    narrow tiles on an SM, 1.09 - 1.10 with five"""
    from ac4k_kernel_b200 import _cuda_ops, ops
    t = []
    for shape, cross, reduce in (((1, 75600, 40, 128), 1, 3), ((75600, 5120), 0, 1)):
        x = torch.randn(shape, device="cuda", dtype=torch.bfloat16)
        q, sf, g = ops.quantize(x, cross, reduce, sf_layout="128x4")
        t.append(min(_graph_microseconds(lambda: _cuda_ops.quantize_nvfp4(q, sf, x, g, cross, reduce, False), calls=5) for _ in range(3)))
    assert t[0] < 1.14 * t[1]


@pytest.mark.gpu
def test_native_host_side_is_the_python_path():
    """Attention's results are the wrappers' own, given an output or not, and so are some refusals (all operators and options:
    test_host_calls.py)"""
    from ac4k_kernel_b200 import ops
    from ac4k_kernel_b200.native import host_calls
    import sys
    assert host_calls is not None, "the native host side is not built"
    py = sys.modules["ac4k_kernel_b200.ops.attention"]
    q, k, v = (gaussian((2, 70, 3, 80), seed=i).cuda() for i in range(3))
    for precision, fn in (("nvfp4", py._nvfp4_attention), ("int8+fp8e4m3", py._int8_x_fp8_attention)):
        for layout in ("BNHD", "BHND"):
            t = [x if layout == "BNHD" else x.transpose(1, 2).contiguous() for x in (q, k, v)]
            out = torch.empty_like(t[0])
            assert ops.attention(*t, layout=layout, precision=precision, out=out) is out
            assert torch.equal(out, fn(*t, layout)) and torch.equal(out, ops.attention(*t, layout=layout, precision=precision))
    x = gaussian((20, 256), seed=9).cuda()
    assert host_calls.quantize(x.t(), 0, 1, None, "nvfp4", False, "ac4k") is None          # not contiguous
    assert host_calls.quantize(x, 0, 0, None, "nvfp4", False, "ac4k") is None
    assert host_calls.quantize(x, 0, 1, None, "nvfp4", False, "other") is None
    with pytest.raises(RuntimeError, match="contiguous"):
        ops.quantize(x.t(), 0, 1)
    with pytest.raises(AssertionError):
        ops.quantize(x, 0, 0)
    w = ops.quantize(gaussian((64, 128), seed=1).cuda(), 0, 1)
    with pytest.raises(RuntimeError, match="B size"):
        ops.linear(*ops.quantize(x, 0, 1), *w)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 50, 300])
def test_captured(m):
    """quantise (one cluster, flat, flat with a ragged tile) and GEMM replayed from a graph on new inputs"""
    from ac4k_kernel_b200 import ops
    w = ops.quantize((gaussian((512, 1024), seed=1) * 0.05).bfloat16().cuda(), 0, 1)
    x = gaussian((m, 1024), seed=2).cuda()
    ops.linear(*ops.quantize(x, 0, 1), *w)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = ops.linear(*ops.quantize(x, 0, 1), *w)
    for seed in (3, 4):
        x.copy_(gaussian((m, 1024), seed=seed).cuda() * seed)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, ops.linear(*ops.quantize(x, 0, 1), *w))


def test_native_host_side_leaves_other_tensors_to_python():
    from ac4k_kernel_b200.native import host_calls
    if host_calls is None:
        pytest.skip("the native host side is not built")
    x = torch.zeros((16, 64), dtype=torch.bfloat16)
    assert host_calls.quantize(x, 0, 1, None, "nvfp4", False, "ac4k") is None
    assert host_calls.quantize("x", 0, 1, None, "nvfp4", False, "ac4k") is None
    assert host_calls.linear(x, x, x, x, x, x, None, None) is None
    assert host_calls.attention(x, x, x, "BNHD", "nvfp4", None) is None
    assert host_calls.rope3d(x, x, x, None) is None
