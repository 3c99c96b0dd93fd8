"""Values at the ends of their ranges in the whole-step and small kernels."""
import pytest
import torch

from oracle import came_oracle as orc
from tests.parity_util import make_inputs, run_pair
from tests.test_gpu_parity import _check_8bit, _check_fp

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


PRESETS = [("CAME8bit", lambda dim: orc.TILE8 if dim == 2 else orc.FLAT8), ("CAME8bitFull", lambda dim: orc.FLAT8),
           ("CAMECUDA", lambda dim: orc.CUDAFP)]
MATRICES = [(256, 512), (130, 1088), (33, 77), (16, 8), (300,)]


@pytest.mark.parametrize("cls_name,preset", PRESETS)
def test_gradients_that_are_all_zero(cls_name, preset, route):
    import came_b200
    out, _, _ = run_pair(getattr(came_b200, cls_name), preset, MATRICES, torch.float32, 3, H, seed=6, grad_scale=0.0)
    (_check_fp if cls_name == "CAMECUDA" else _check_8bit)(out, torch.float32)


@pytest.mark.parametrize("cls_name", ["CAME8bit", "CAME8bitFull", "CAMECUDA"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_poisoned_gradient_stays_in_its_tensor(cls_name, value, route):
    """Every wait ends, and the other tensors get the bytes they get without it."""
    import came_b200
    shapes = MATRICES + [(6, 3, 3), (5, 2, 40, 24)]
    params0, grads = make_inputs(shapes, torch.bfloat16, 2, seed=7)
    results = []
    for bad in range(-1, len(shapes)):
        ps = [torch.nn.Parameter(p.cuda()) for p in params0]
        opt = getattr(came_b200, cls_name)(ps, **H)
        for gs in grads:
            for i, (p, g) in enumerate(zip(ps, gs)):
                p.grad = g.cuda()
                if i == bad:
                    p.grad.view(-1)[p.numel() // 2] = value
            opt.step()
        assert all(plan.status() == 0 for plan in opt._engine.plans.values())
        results.append([p.data for p in ps])
        for i, (a, b) in enumerate(zip(results[0], results[-1])):
            assert bool(b.isfinite().all()) == (i != bad), (i, bad)
            assert i == bad or torch.equal(a, b), (i, bad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_flat_layout_off_the_16_byte_boundary(dtype):
    """Parameters and gradients at odd elements of larger buffers: the same bytes as on the boundary (odd widths: the same
    arithmetic), and nothing is written beside them."""
    import came_b200
    shapes = [(37, 201), (64, 777), (100, 21), (9, 31), (257, 5)]
    params0, grads = make_inputs(shapes, dtype, 3, seed=8)
    finals = []
    for shift in (0, 1, 3):
        def place(t):
            big = torch.full((t.numel() + 8,), 7.0, dtype=dtype, device="cuda")
            view = big[shift:shift + t.numel()].view(t.shape)
            view.copy_(t)
            return big, view
        placed = [place(p) for p in params0]
        ps = [torch.nn.Parameter(v) for _, v in placed]
        opt = came_b200.CAME8bitFull(ps, **H)
        for gs in grads:
            for p, g in zip(ps, gs):
                p.grad = place(g)[1]
            opt.step()
        for (big, v) in placed:
            assert bool((big[:shift] == 7.0).all()) and bool((big[shift + v.numel():] == 7.0).all())
        finals.append([p.data.clone() for p in ps] + [v.clone() for p in ps for _, v in sorted(opt.state[p].items()) if torch.is_tensor(v)])
    for other in finals[1:]:
        for a, b in zip(finals[0], other):
            assert torch.equal(a, b)


def test_more_param_groups_than_the_launch_carries():
    """Up to four groups travel as kernel arguments, more are read from the workspace: the same bytes."""
    import came_b200
    shapes = [(33, 77), (64, 48), (300,), (40, 24), (17, 16), (5,)]
    params0, grads = make_inputs(shapes, torch.bfloat16, 3, seed=9)
    finals = []
    for groups in (1, 4, 5, 6):
        ps = [torch.nn.Parameter(p.cuda()) for p in params0]
        opt = came_b200.CAME8bit([dict(params=ps[k:k + 1] if k < groups - 1 else ps[k:]) for k in range(groups)], **H)
        for gs in grads:
            for p, g in zip(ps, gs):
                p.grad = g.cuda()
            opt.step()
        finals.append([p.data for p in ps])
    for other in finals[1:]:
        for a, b in zip(finals[0], other):
            assert torch.equal(a, b)
