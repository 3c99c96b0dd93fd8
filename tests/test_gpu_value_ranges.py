"""Values at the ends of their ranges in the whole-step and small kernels."""
import pytest
import torch

from tests.parity_util import make_inputs

pytestmark = pytest.mark.gpu

H = dict(lr=1e-3, eps=(1e-30, 1e-16), clip_threshold=1.0, betas=(0.9, 0.999, 0.9999), weight_decay=1e-2)
SHAPES = [(33, 770), (64, 48), (257, 17), (300,), (6, 3, 3), (5, 2, 40, 24)]


def _final(cls, shapes, grads, params0, scale, dtype):
    ps = [torch.nn.Parameter(p.cuda()) for p in params0]
    opt = cls(ps, **H)
    opt.param_groups[0]["grad_scale"] = scale
    for gs in grads:
        for p, g in zip(ps, gs):
            p.grad = (g.float() / scale).to(dtype).cuda()
        opt.step()
    return [p.data for p in ps] + [v for p in ps for _, v in sorted(opt.state[p].items()) if torch.is_tensor(v)]


@pytest.mark.parametrize("cls_name", ["CAME8bit", "CAME8bitFull", "CAMECUDA"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("power", [80, -64])
def test_unscaled_gradients_whose_squares_leave_the_range(cls_name, dtype, power):
    """grad_scale is a power of two, which commutes with every rounding: the same bytes as without it.  (Gradients of
    about 1e-3 times 2^-64 square to zero; their smallest entries, above 2^-60 among 40 000, stay normal numbers.)"""
    import came_b200
    cls = getattr(came_b200, cls_name)
    params0, grads = make_inputs(SHAPES, dtype, 3, seed=5)
    want = _final(cls, SHAPES, grads, params0, 1.0, dtype)
    got = _final(cls, SHAPES, grads, params0, 2.0 ** -power, dtype)
    for a, b in zip(want, got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cls_name", ["CAMECUDA", "CAME8bitFull"])
@pytest.mark.parametrize("n", [1, 255, 257, 5000])
def test_vector_whose_clip_divisor_is_infinite(cls_name, n):
    """beta2 = 1 keeps the second moment at zero: the clamped 1e-30 makes u = 1e15 g, whose squares overflow, and a finite
    u over an infinite divisor is zero (CAMECUDA.py:262-269, came_kernels.cu:1509-1516): the parameter stays."""
    import came_b200
    p = torch.nn.Parameter(torch.linspace(-1, 1, n, device="cuda"))
    p.grad = torch.linspace(1e5, 2e5, n, device="cuda")
    before = p.data.clone()
    opt = getattr(came_b200, cls_name)([p], lr=1e-2, betas=(0.9, 1.0, 0.999))
    for _ in range(2):
        opt.step()
    assert torch.equal(p.data, before)
