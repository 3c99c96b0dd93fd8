"""The native step table: which changes between two steps it takes by itself, which it hands back, and that either way
the result is the one of an optimizer that sees everything for the first time (bit for bit: same kernels)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(64, 48), (33, 770), (300,), (1024, 1024)]


def _make(seed=0):
    import came_b200
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ps = [torch.nn.Parameter((torch.randn(s, device="cuda", generator=gen) * 0.02).bfloat16()) for s in SHAPES]
    return ps, came_b200.CAME8bit([{"params": ps[:2]}, {"params": ps[2:], "lr": 3e-3}], lr=1e-3, weight_decay=0.1)


def _grads(step):
    gen = torch.Generator(device="cuda").manual_seed(100 + step)
    return [(torch.randn(s, device="cuda", generator=gen) * 1e-3).bfloat16() for s in SHAPES]


def _change(kind, step, ps, opt):
    """-> gradients that the parameters get for this step."""
    gs = _grads(step)
    if kind == "lr":
        opt.param_groups[0]["lr"] = 1e-3 * 0.5 ** step
        opt.param_groups[1]["betas"] = (0.8, 0.9, 0.95)
    elif kind == "scale":
        opt.param_groups[1]["grad_scale"] = 0.25
    elif kind == "none" and step == 2:
        gs[1] = None
    elif kind == "strided" and step == 2:
        gs[0] = gs[0].t().contiguous().t()
    elif kind == "unaligned" and step == 2:
        big = torch.zeros(gs[3].numel() + 1, device="cuda", dtype=torch.bfloat16)
        big[1:] = gs[3].reshape(-1)
        gs[3] = big[1:].view(SHAPES[3])
    return gs


@pytest.mark.parametrize("kind", ["same", "moved", "lr", "scale", "none", "strided", "unaligned"])
def test_table_equals_full_path(kind, route):
    (pa, oa), (pb, ob) = _make(), _make()
    keep = []
    for step in range(4):
        ga, gb = _change(kind, step, pa, oa), _change(kind, step, pb, ob)
        for ps, gs in ((pa, ga), (pb, gb)):
            for p, g in zip(ps, gs):
                if kind in ("moved", "strided", "unaligned") or g is None or p.grad is None:
                    keep.append(p.grad)      # the old buffers live on: addresses differ for certain
                    p.grad = g
                else:
                    p.grad.copy_(g)
        oa.step()
        ob._table = None                     # always the full path
        ob.step()
        assert oa.last_step_launches == ob.last_step_launches
    for p, q in zip(pa, pb):
        assert torch.equal(p.data, q.data)
        for k, v in oa.state[p].items():
            assert torch.equal(v, ob.state[q][k]) if torch.is_tensor(v) else v == ob.state[q][k], k


def test_hooks_closures_and_repeated_tables():
    ps, opt = _make()
    calls = []
    for p, g in zip(ps, _grads(0)):
        p.grad = g
    opt.step()
    h = opt.register_step_pre_hook(lambda *a: calls.append("pre"))
    opt.step()
    h.remove()
    opt.step()
    assert calls == ["pre"] and opt.step(lambda: 5.0) == 5.0
    assert opt.state[ps[2]]["step"] == 4
    opt.param_groups[0]["betas"] = (0.9, 0.99)
    with pytest.raises(Exception):
        opt.step()


@pytest.mark.parametrize("kind", ["alignment", "dropped", "and back"])
def test_plans_replaced_by_priming(kind):
    """prime_for_cuda_graph() between two steps closes or re-points the plan that the table was built from."""
    (pa, oa), (pb, ob) = _make(), _make()
    for ps, opt in ((pa, oa), (pb, ob)):
        sets = [_grads(0), _grads(1)]
        if kind == "alignment":
            big = torch.zeros(sets[1][3].numel() + 1, device="cuda", dtype=torch.bfloat16)
            big[1:] = sets[1][3].reshape(-1)
            sets[1][3] = big[1:].view(SHAPES[3])
        elif kind == "dropped":
            sets[1][2] = None
        for k, gs in enumerate((sets[0], sets[0], sets[1])):
            for p, g in zip(ps, gs):
                p.grad = g
            if k < 2:
                opt.step()
        if opt is ob:
            ob._table = None
        opt.prime_for_cuda_graph()
        if kind == "and back":
            for p, g in zip(ps, sets[0]):
                p.grad = g
        if opt is ob:
            ob._table = None
        opt.step()
        opt.step()
    assert oa.last_step_launches == ob.last_step_launches
    for p, q in zip(pa, pb):
        assert torch.equal(p.data, q.data)


def test_other_threads_run_while_launches_wait():
    """A launch that waits for room in the stream's queue must not hold the interpreter's lock."""
    import threading
    import time
    from came_b200 import quant
    ps, opt = _make()
    for p, g in zip(ps, _grads(0)):
        p.grad = g
    x = torch.ones(256, device="cuda")
    opt.step(); opt.step(); quant.dequantize_blockwise(*quant.quantize_blockwise(x, signed=True), signed=True)
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), []

    def ticks():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.005)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    for work in (opt.step, lambda: quant.quantize_blockwise(x, signed=True)):
        thread = threading.Thread(target=ticks)
        gaps.clear()
        stop.clear()
        thread.start()
        t0 = time.perf_counter()
        torch.cuda._sleep(3_000_000_000)      # about 1.5 s, in front of more launches than a queue holds
        for _ in range(3000):
            work()
        waited = time.perf_counter() - t0
        torch.cuda.synchronize()
        stop.set()
        thread.join()
        assert waited > 1.0 and max(gaps) < 0.5, (waited, max(gaps))


def test_out_of_memory_keeps_its_type():
    from came_b200 import quant
    x = torch.ones(1, device="cuda").expand(1 << 40)      # 4 TB once contiguous: refused at once
    with pytest.raises(torch.OutOfMemoryError):
        quant.quantize_blockwise(x, signed=True)
    assert quant.quantize_blockwise(x[:300], signed=True)[1].tolist() == [1.0, 1.0]
