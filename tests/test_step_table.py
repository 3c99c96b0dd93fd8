"""The native step table on the CPU, with a stand-in for the plan: what makes it hand a step back instead of launching."""
import ctypes as C

import pytest
import torch

import came_b200
from came_b200 import _host


class _Plan:
    """The part of engine.DevicePlan the table uses."""

    def __init__(self):
        self.memory = C.create_string_buffer(1 << 16)
        self.handle = C.c_void_p(C.addressof(self.memory))
        self.addresses = ()


def _group(*shapes):
    ps = [torch.nn.Parameter(torch.zeros(s)) for s in shapes]
    for p in ps:
        p.grad = torch.zeros_like(p)
    return ps, [dict(params=ps, lr=1e-3, betas=(0.9, 0.99, 0.999), eps=(1e-30, 1e-16), clip_threshold=1.0, weight_decay=0.0)]


def _optimizer(cls=None):
    opt = (cls or came_b200.CAME8bit)([torch.nn.Parameter(torch.zeros(4, 4))], lr=1e-3)
    opt._collect = lambda: ([], [], [])      # (no GPU here: nothing to step)
    return opt


def test_a_closed_plan_is_not_stepped():
    ps, groups = _group((4, 4), (3,))
    plan, table = _Plan(), _host.StepTable()
    assert table.build(groups, [(plan, -1, 2)], [])
    plan.handle = None                       # what DevicePlan.close() leaves
    assert table.step(groups) == -1
    ps[0].grad = torch.ones(4, 4)            # gradients that moved: no pointer upload either
    assert table.step(groups) == -1


def test_priming_drops_the_table():
    """prime_for_cuda_graph() may replace or re-point the plans the table was built from."""
    opt = _optimizer()
    opt._table = object()
    opt.prime_for_cuda_graph()
    assert opt._table is None


def test_counts_go_up_for_all_or_none():
    ps, groups = _group((4, 4), (3,))
    states = [{"step": 3}, {}]               # the second has lost its count: the full path has to look at it
    plan, table = _Plan(), _host.StepTable()
    assert table.build(groups, [(plan, -1, 2)], states)
    assert table.step(groups) == -1
    assert states == [{"step": 3}, {}]
    states[1]["step"] = object()             # what the full path raises for, the table leaves to it
    assert table.step(groups) == -1
    assert states[0] == {"step": 3}


def test_an_exception_drops_the_table():
    class Raises:
        def step(self, groups):
            raise RuntimeError("no")

    opt = _optimizer()
    opt._table = Raises()
    with pytest.raises(RuntimeError):
        opt.step()
    assert opt._table is None


def test_the_table_holds_no_tensors():
    """torch.utils.swap_tensors() and the garbage collector count a parameter's references."""
    ps, groups = _group((4, 4), (4, 4))
    plan, table = _Plan(), _host.StepTable()
    assert table.build(groups, [(plan, -1, 2)], [])
    ps[0].grad = ps[1].grad = None
    torch.utils.swap_tensors(ps[0], torch.nn.Parameter(torch.ones(4, 4)))
    assert table.step(groups) == -1


def test_hooks_run_once_under_an_overridden_step():
    """torch wraps the subclass's step() with the hooks; the step it calls must not run them again."""
    class Mine(came_b200.CAME8bit):
        def step(self, closure=None):
            return super().step(closure)

    class Inherits(Mine):
        pass

    class Plain(came_b200.CAME8bit):
        pass

    for cls in (Mine, Inherits, Plain, came_b200.CAME8bit):
        opt, calls = _optimizer(cls), []
        opt.register_step_pre_hook(lambda *a: calls.append("pre"))
        opt.register_step_post_hook(lambda *a: calls.append("post"))
        opt.step()
        assert opt.step(lambda: 2.0) == 2.0
        assert calls == ["pre", "post"] * 2, cls


def test_entries_refuse_what_is_no_tensor():
    for call in (lambda: _host.quantize(object(), True, False), lambda: _host.dequantize(object(), torch.zeros(1), True, False),
                 lambda: _host.dequantize(torch.zeros(4, dtype=torch.int8), [1.0], True, False)):
        with pytest.raises(TypeError):
            call()


class _Raises(torch.Tensor):
    """A tensor whose layout is asked for in Python, which raises."""

    @staticmethod
    def __new__(cls, shape):
        return torch.Tensor._make_wrapper_subclass(cls, shape, dispatch_sizes_strides_policy="strides")

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise KeyError("asked")


def test_exceptions_out_of_tensors_reach_python():
    """A C++ or Python exception below the module's entries is raised as what it is; it does not end the process."""
    ps, groups = _group((4, 4))
    plan, table = _Plan(), _host.StepTable()
    assert table.build(groups, [(plan, -1, 1)], [])
    bad = torch.nn.Parameter(torch.zeros(4, 4))
    bad.grad = _Raises((4, 4))
    groups[0]["params"] = [bad]
    with pytest.raises(KeyError):
        _host.StepTable().build(groups, [(plan, -1, 1)], [])
    groups[0]["params"] = ps
    ps[0].grad = _Raises((4, 4))
    with pytest.raises(KeyError):
        table.step(groups)
