"""MXFP8 host-side arithmetic (pure PyTorch, no GPU): block scales, quantisation error, the scale layout the
tensor core reads.  The GPU kernels are checked against these functions in the gpu-marked tests."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from mintccl_b200.ops import mxfp8 as mx


def test_scale_is_the_smallest_power_of_two_without_saturation():
    g = torch.Generator().manual_seed(0)
    amax = torch.cat([torch.rand(2000, generator=g) * 10 ** torch.randint(-6, 7, (2000,), generator=g).float(),
                      torch.tensor([448.0, 448.0001, 447.9999, 1.75, 1.7500001, 2.0 ** -20, 3.0e4])])
    s = mx.scale_to_float(mx.scale_for_amax(amax))
    assert bool(((torch.log2(s) % 1) == 0).all())                    # powers of two
    assert bool((amax / s <= 448.0).all())                           # the block's largest value fits e4m3
    assert bool((amax / (s / 2) > 448.0).all())                      # and half the scale would not


def test_zero_block_and_roundtrip_shapes():
    x = torch.zeros(64)
    d, s = mx.quantize_mxfp8(x)
    assert d.dtype == torch.uint8 and s.dtype == torch.uint8 and d.numel() == 64 and s.numel() == 2
    assert int(s[0]) == 127 - 8 and bool((mx.dequantize_mxfp8(d, s) == 0).all())
    with pytest.raises(Exception):
        mx.quantize_mxfp8(torch.zeros(33))                           # blocks of 32


@pytest.mark.parametrize("spread", [1.0, 1e-3, 1e3])
def test_quantisation_error_is_bounded_by_the_block_maximum(spread):
    g = torch.Generator().manual_seed(3)
    x = torch.randn(4096, generator=g) * spread * torch.logspace(-2, 2, 4096 // 32).repeat_interleave(32)
    d, s = mx.quantize_mxfp8(x)
    dq = mx.dequantize_mxfp8(d, s)
    assert bool(torch.isfinite(dq).all())                            # e4m3fn has no infinity; NaN would mean saturation
    amax = x.view(-1, 32).abs().amax(dim=1, keepdim=True)
    err = (dq - x).view(-1, 32).abs()
    # 3 mantissa bits: half an ulp is 2^-4 of the value's binade, at most 2^-4 of the block maximum
    assert bool((err <= amax * 2.0 ** -4 + 1e-30).all())
    # elements near the block maximum keep 2^-4 relative accuracy
    big = x.view(-1, 32).abs() >= amax / 2
    assert bool((err[big] <= x.view(-1, 32).abs()[big] * 2.0 ** -4 * 1.0001).all())


def test_quantise_rows_keeps_blocks_inside_rows():
    g = torch.Generator().manual_seed(5)
    x = torch.randn(8, 96, generator=g)
    x[3] *= 1000.0                                                   # one loud row must not change its neighbours' scales
    d, s = mx.quantize_rows_mxfp8(x)
    assert d.shape == (8, 96) and s.shape == (8, 3)
    d2, s2 = mx.quantize_rows_mxfp8(x[2:3])
    assert torch.equal(d[2:3], d2) and torch.equal(s[2:3], s2)


@pytest.mark.parametrize("rows,k", [(128, 128), (256, 384), (384, 1024)])
def test_tiled_scale_layout_matches_the_documented_formula(rows, k):
    """[rows / 128][K / 128][512] bytes with byte (r % 32) * 16 + ((r % 128) / 32) * 4 + kb % 4 for row r and
    32-element block kb: what tcgen05.cp moves into TMEM for kind::mxf8f6f4.block_scale."""
    kb = k // 32
    scale = torch.arange(rows * kb, dtype=torch.int64).remainder(251).to(torch.uint8).view(rows, kb)
    tiled = mx.tile_scales(scale)
    assert tiled.numel() == rows * kb
    g = torch.Generator().manual_seed(rows + k)
    for _ in range(300):
        r = int(torch.randint(0, rows, (1,), generator=g))
        b = int(torch.randint(0, kb, (1,), generator=g))
        off = ((r // 128) * (k // 128) + b // 4) * 512 + (r % 32) * 16 + ((r % 128) // 32) * 4 + b % 4
        assert int(tiled[off]) == int(scale[r, b]), (r, b)
    with pytest.raises(ValueError):
        mx.tile_scales(torch.zeros(100, 4, dtype=torch.uint8))


def test_sum_of_quantised_tensors_requantises_once():
    """The oracle of the block-scaled all-reduce: dequantise every rank's tensor, add in fp32, quantise the sum
    once.  Its error against the exact sum is that of ONE quantisation of the sum plus the inputs' own."""
    g = torch.Generator().manual_seed(9)
    xs = [torch.randn(2048, generator=g) * (r + 1) for r in range(8)]
    qs = [mx.quantize_mxfp8(x) for x in xs]
    total = sum(mx.dequantize_mxfp8(d, s) for d, s in qs)
    d, s = mx.quantize_mxfp8(total)
    out = mx.dequantize_mxfp8(d, s)
    amax = total.view(-1, 32).abs().amax(dim=1, keepdim=True)
    assert bool(((out - total).view(-1, 32).abs() <= amax * 2.0 ** -4).all())
    exact = sum(xs)
    rel = ((out - exact).norm() / exact.norm()).item()
    assert rel < 0.05


class _Sub(torch.Tensor):
    pass


class _Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.fixture
def no_kernels(monkeypatch):
    """The device condition lifted, and a kernel launch an error: what reaches it on the GPU would read raw memory."""
    def launch(*a):
        raise AssertionError("a kernel was launched on a tensor that is not its own memory")
    monkeypatch.setattr(mx, "_plain_cuda", mx._is_plain)
    monkeypatch.setattr(mx, "_on_device", launch)
    with pytest.raises(AssertionError):
        mx.quantize_mxfp8(torch.randn(64))                           # the condition is lifted: a plain tensor gets there
    with pytest.raises(AssertionError):
        mx.tile_scales(torch.zeros(128, 4, dtype=torch.uint8))


def test_traced_encoding_replays_on_other_inputs(no_kernels):
    """A trace of these functions holds the operations, not an empty tensor that a kernel once filled."""
    g = torch.Generator().manual_seed(5)
    x, y = torch.randn(128, 128, generator=g), torch.randn(128, 128, generator=g) * 40.0
    sx, sy = (torch.randint(0, 256, (128, 8), generator=g, dtype=torch.uint8) for _ in range(2))
    from torch.fx.experimental.proxy_tensor import make_fx
    for got, want in zip(make_fx(mx.quantize_rows_mxfp8)(x)(y), mx._torch_quantize(y)):
        assert torch.equal(got.reshape(-1), want)
    for f in (make_fx(mx.tile_scales)(sx), torch.jit.trace(mx.tile_scales, sx, check_trace=False)):
        assert torch.equal(f(sy), mx._torch_tile_scales(sy))
    with pytest.raises(RuntimeError, match="aten::view"):            # torch.jit cannot record the view of e4m3 as bytes
        torch.jit.trace(mx.quantize_rows_mxfp8, x, check_trace=False)


@pytest.mark.parametrize("form", ["subclass", "mode", "functional", "functionalize", "zero", "jvp", "fake"])
def test_encoding_of_tensors_that_are_not_plain_memory(form, no_kernels):
    x = torch.randn(64, generator=torch.Generator().manual_seed(6))
    want = mx._torch_quantize(x)
    if form == "subclass":
        got = mx.quantize_mxfp8(x.as_subclass(_Sub))
    elif form == "mode":
        with _Mode():
            got = mx.quantize_mxfp8(x)
    elif form == "functional":
        got = mx.quantize_mxfp8(torch._to_functional_tensor(x))
        want = tuple(map(torch.Tensor.tolist, want))
        got = tuple(map(torch.Tensor.tolist, got))
        assert got == want
        return
    elif form == "functionalize":
        got = torch.func.functionalize(mx.quantize_mxfp8)(x)
    elif form == "zero":
        got, want = mx.quantize_mxfp8(torch._efficientzerotensor(64)), mx._torch_quantize(torch.zeros(64))
    elif form == "jvp":
        got, _ = torch.func.jvp(lambda t: tuple(o.float() for o in mx.quantize_mxfp8(t)), (x,), (torch.ones_like(x),))
        want = tuple(o.float() for o in want)
    else:
        from torch._subclasses.fake_tensor import FakeTensorMode
        with FakeTensorMode() as m:
            d, s = mx.quantize_mxfp8(m.from_tensor(x))
            assert tuple(d.shape) == (64,) and tuple(s.shape) == (2,)
        return
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("lifted", [False, True], ids=["cpu", "device_lifted"])
def test_tile_scales_under_vmap(lifted, monkeypatch):
    """A batched tensor has no address to ask for."""
    if lifted:
        monkeypatch.setattr(mx, "_plain_cuda", mx._is_plain)
    s = torch.randint(0, 256, (3, 128, 8), generator=torch.Generator().manual_seed(7), dtype=torch.uint8)
    assert torch.equal(torch.vmap(mx.tile_scales)(s), torch.stack([mx._torch_tile_scales(t) for t in s]))


def test_gemm_refuses_tensors_on_the_cpu(monkeypatch):
    """Host addresses must not reach a kernel: the call ends before the native library is asked for anything."""
    from mintccl_b200 import _native as N

    def launch():
        raise AssertionError("launched")
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 0)
    monkeypatch.setattr(N, "lib", launch)
    d, s, w = torch.zeros(128, 128, dtype=torch.uint8), torch.zeros(128, 4, dtype=torch.uint8), torch.zeros(256, 128, dtype=torch.uint8)
    with pytest.raises(ValueError, match="CUDA"):
        mx.gemm_mxfp8(d, s, w, torch.zeros(256, 4, dtype=torch.uint8))
