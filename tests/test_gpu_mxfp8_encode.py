"""The MXFP8 encoding kernels give the bytes of the torch expressions they stand in for."""
import pytest
import torch

from mintccl_b200.ops import mxfp8 as mx

pytestmark = pytest.mark.gpu


def _special(n, dtype):
    """Magnitudes over the whole range of the type, ties of e4m3, zeros, infinities, NaN and all-zero blocks."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, generator=g, device="cuda")
    lo, hi = (-44.0, 38.0) if dtype is not torch.float16 else (-7.0, 4.5)
    e = torch.rand(n // 32, generator=g, device="cuda") * (hi - lo) + lo
    x = (x.view(-1, 32) * (10.0 ** e.double()[:, None])).float()
    x[::7, 3] = 0.0
    x[1::11] = -0.0
    x[2::13, 5] = float("inf")
    x[3::13, 6] = float("-inf")
    x[4::17, 7] = float("nan")
    x[5::19] = torch.arange(32, device="cuda") * 15.0 - 16.0       # 448, 464: halves of the last steps
    x[6::23] = torch.finfo(dtype).max
    x[7::29] = torch.finfo(dtype).smallest_normal * torch.finfo(dtype).eps
    return x.reshape(-1).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("blocks", [0, 1, 31, 33, 1023, 40_000])
def test_quantise_kernel_gives_the_bytes_of_the_torch_path(dtype, blocks):
    x = _special(blocks * 32, dtype) if blocks else torch.empty(0, device="cuda", dtype=dtype)
    d, s = mx.quantize_mxfp8(x)
    td, ts = mx._torch_quantize(x)
    assert torch.equal(s, ts)
    assert torch.equal(d, td)


def test_quantise_kernel_takes_any_layout():
    g = torch.Generator(device="cuda").manual_seed(1)
    base = torch.randn(4 * 96 * 64 + 8, generator=g, device="cuda").to(torch.bfloat16)
    for x in (base[1:1 + 64 * 96].view(64, 96), base[:96 * 64].view(64, 96).t(), base[:4 * 96 * 64].view(4, 96, 64)[::2, :, ::2]):
        for got, want in zip(mx.quantize_mxfp8(x), mx._torch_quantize(x)):
            assert torch.equal(got, want)
    with pytest.raises(RuntimeError):
        mx.quantize_mxfp8(base[:33])


@pytest.mark.parametrize("rows,kb", [(128, 4), (256, 124), (128, 128), (384, 132), (1024, 36)])
def test_tile_kernel_gives_the_bytes_of_the_torch_path(rows, kb):
    g = torch.Generator(device="cuda").manual_seed(rows + kb)
    s = torch.randint(0, 256, (rows, kb), generator=g, device="cuda", dtype=torch.uint8)
    assert torch.equal(mx.tile_scales(s), mx._torch_tile_scales(s))
    off = torch.cat([s.new_zeros(1), s.reshape(-1)])[1:].view(rows, kb)      # not on a 4-byte boundary
    assert torch.equal(mx.tile_scales(off), mx._torch_tile_scales(s))


def test_traced_encoding_replays_on_other_inputs():
    """A recorded graph of the encoding on CUDA tensors holds the operations: it gives other inputs their own bytes."""
    from torch.fx.experimental.proxy_tensor import make_fx
    g = torch.Generator(device="cuda").manual_seed(3)
    x, y = (torch.randn(128, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    sx, sy = mx.quantize_rows_mxfp8(x)[1].repeat(1, 2), mx.quantize_rows_mxfp8(y * 40)[1].repeat(1, 2)
    for got, want in zip(make_fx(mx.quantize_rows_mxfp8)(x)(y), mx._torch_quantize(y)):
        assert torch.equal(got.reshape(-1), want)
    assert torch.equal(torch.jit.trace(mx.tile_scales, sx, check_trace=False)(sy), mx._torch_tile_scales(sy))
