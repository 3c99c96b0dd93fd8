"""The codec kernels' two access widths, bit-exact against the oracle (no tolerance): sizes around a block and a lane's
four elements, buffers off the 16-byte boundary, columns that are and are not a multiple of 4, values on and next to
the boundaries between codes (where the encoder divides instead of multiplying)."""
import pytest
import torch

from oracle import came_oracle as orc

pytestmark = pytest.mark.gpu


def _boundary_values(n, qmax, seed):
    g = torch.Generator().manual_seed(seed)
    a = 0.7310585975646973
    k = torch.randint(-int(qmax), int(qmax), (n,), generator=g).float() + 0.5
    x = (k / qmax) * a
    step = torch.randint(-2, 3, (n,), generator=g).to(torch.int32)
    x = (x.view(torch.int32) + step).view(torch.float32)      # up to two representable values off the boundary
    x[::256] = a
    return x


def _same(a, b):
    return torch.equal(a.cpu().contiguous().view(torch.int32), b.contiguous().view(torch.int32))


@pytest.mark.parametrize("n", [3, 252, 259, 2047, 2048, 2304 + 8])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("signed", [True, False])
def test_blockwise(n, shift, signed):
    from came_b200 import quant
    x = _boundary_values(n + shift, 127.0 if signed else 255.0, n)
    q, a = quant.quantize_blockwise(x.cuda()[shift:], signed=signed)
    qo, ao = orc.quantize_blockwise(x[shift:], signed=signed)
    assert torch.equal(q.cpu(), qo) and _same(a, ao)
    wide = torch.zeros(n + shift, dtype=q.dtype, device="cuda")
    wide[shift:] = q
    assert _same(quant.dequantize_blockwise(wide[shift:], a, signed=signed), orc.dequantize_blockwise(qo, ao, signed=signed))


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 48])
@pytest.mark.parametrize("cols", [1, 4, 12, 17, 124, 128, 129, 132, 260])
@pytest.mark.parametrize("shift", [0, 1])
def test_tile(rows, cols, shift):
    from came_b200 import quant
    n = rows * cols
    x = _boundary_values(n + shift, 127.0, n)
    q, a = quant.quantize_tile16(x.cuda()[shift:].view(rows, cols))
    qo, ao = orc.quantize_tile16(x[shift:].view(rows, cols))
    assert torch.equal(q.cpu(), qo) and _same(a, ao)
    assert _same(quant.dequantize_tile16(q, a), orc.dequantize_tile16(qo, ao))
