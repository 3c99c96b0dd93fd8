"""Tensors made of small matrices (the kernels that take chunks of 256 or more matrices into shared memory) at the edges
of their range: one matrix more or less than a chunk, a short last group of four, run-time shapes up to 8 x 8, the first
shapes beyond it, buffers off the 16-byte boundary.  Tolerances and presets as in tests/test_gpu_nd.py."""
import pytest
import torch

from oracle import came_oracle as orc
from tests.parity_util import run_pair
from tests.test_gpu_parity import H_LLAMA, H_NOWD, _check_8bit, _check_fp, _dt

pytestmark = pytest.mark.gpu

SHAPES = [(257, 1, 3, 3), (85, 3, 3, 3), (1, 2, 3, 3), (683, 3, 1, 1), (2049, 1, 1, 1), (5, 1, 1), (301, 5, 5), (43, 3, 7, 7),
          (257, 8, 8), (259, 1, 16), (258, 16, 1), (300, 64, 1), (300, 1, 65), (31, 9, 9)]


@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_8bit(dtype):
    import came_b200
    out, opt, _ = run_pair(came_b200.CAME8bitFull, lambda dim: orc.FLAT8_CPU, SHAPES, _dt(dtype), 4, H_LLAMA, seed=61)
    _check_8bit(out, _dt(dtype))
    assert all(plan.status() == 0 for plan in opt._engine.plans.values())


@pytest.mark.parametrize("cls_name,preset", [("CAME", orc.CAME), ("CAMECUDA", orc.CUDAFP_GENERIC)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_fp32_states(cls_name, preset, dtype):
    import came_b200
    out, _, _ = run_pair(getattr(came_b200, cls_name), lambda dim: preset, SHAPES, _dt(dtype), 4, H_NOWD, seed=62)
    _check_fp(out, _dt(dtype))


@pytest.mark.parametrize("shift", [1, 4])
def test_unaligned_buffers_step_like_aligned_ones(shift):
    """Same arithmetic, other access widths: bit for bit."""
    import came_b200
    shape, n = (86, 3, 3, 3), 86 * 27
    gen = torch.Generator().manual_seed(shift)
    p0, g0 = torch.randn(n, generator=gen), torch.randn(n, generator=gen) * 1e-3
    results = []
    for off in (0, shift):
        p, g = (torch.zeros(n + off, device="cuda", dtype=torch.float16) for _ in range(2))
        p[off:] = p0.half().cuda()
        g[off:] = g0.half().cuda()
        param = torch.nn.Parameter(p[off:].view(shape))
        param.grad = g[off:].view(shape)
        opt = came_b200.CAME8bitFull([param], lr=1e-3, weight_decay=0.1)
        for _ in range(2):
            opt.step()
        results.append([param.data.clone()] + [v.clone() for k, v in sorted(opt.state[param].items()) if torch.is_tensor(v)])
    assert all(torch.equal(a, b) for a, b in zip(*results))
