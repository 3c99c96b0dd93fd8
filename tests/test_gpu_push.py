"""Push mode of the weight exchange on ONE GPU: the "peer" is a second buffer of the same device, so the stores the
apply kernel adds can be checked without a second process.  After a step the mirror must hold exactly the new values
of every tensor the plan reports as pushed, and nothing else; bad set-ups are refused on the host.  (Two ranks on two
GPUs: tests/test_gpu_peer_gather.py.)  No counterpart in the reference, which is single-GPU."""
import pytest
import torch

from tests.parity_util import kernels_of

pytestmark = pytest.mark.gpu

SHAPES = [(256, 1024), (4096,), (130, 2304), (64, 192), (300,), (129, 1088)]


def _setup(cls_name, dtype):
    import came_b200
    dev = torch.device("cuda", 0)
    sizes = [((torch.Size(s).numel() + 127) // 128) * 128 for s in SHAPES]
    flat = torch.zeros(sum(sizes), dtype=dtype, device=dev)
    gen = torch.Generator(device=dev).manual_seed(11)
    flat.copy_((torch.randn(flat.shape, generator=gen, device=dev) * 0.02).to(dtype))
    views, off = [], 0
    for s, n in zip(SHAPES, sizes):
        views.append(flat[off:off + torch.Size(s).numel()].view(s))
        off += n
    params = [torch.nn.Parameter(v) for v in views]
    for i, p in enumerate(params):
        p.grad = (torch.randn(p.shape, generator=gen, device=dev) * 10.0 ** (-2 - i % 3)).to(dtype)
    opt = getattr(came_b200, cls_name)(params, lr=1e-3, weight_decay=1e-2)
    opt.prime_for_cuda_graph()
    return flat, params, opt


@pytest.mark.parametrize("cls_name,dtype", [("CAME8bit", torch.bfloat16), ("CAME8bit", torch.float32),
                                            ("CAME8bitFull", torch.bfloat16)])
def test_mirror_receives_exactly_the_pushed_tensors(cls_name, dtype, route):
    flat, params, opt = _setup(cls_name, dtype)
    mirrors = [torch.zeros_like(flat) for _ in range(2)]
    nbytes = flat.numel() * flat.element_size()
    opt._engine.set_push(flat.data_ptr(), nbytes, [m.data_ptr() for m in mirrors])
    (plan,) = opt._engine.plans.values()
    pushed = plan.pushed()
    assert any(pushed) and not all(pushed)          # the matrices on the staged path, not the vectors / odd widths
    for _ in range(2):
        opt.step()
    torch.cuda.synchronize()
    assert plan.status() == 0
    base = flat.data_ptr()
    for p, flag in zip(params, pushed):
        lo = (p.data_ptr() - base) // flat.element_size()
        for m in mirrors:
            got = m[lo:lo + p.numel()].view(p.shape)
            if flag:
                assert torch.equal(got, p.data)
            else:
                assert not got.any()
    # switching the mode off stops the stores
    opt._engine.set_push(flat.data_ptr(), nbytes, [])
    before = [m.clone() for m in mirrors]
    opt.step()
    torch.cuda.synchronize()
    for m, b in zip(mirrors, before):
        assert torch.equal(m, b)
    assert ("moment_apply" in kernels_of(opt)) == (route == "staged")


def test_bad_push_setups_are_refused(route):
    flat, params, opt = _setup("CAME8bit", torch.bfloat16)
    (plan,) = opt._engine.plans.values()
    nbytes = flat.numel() * flat.element_size()
    other = torch.zeros_like(flat)
    with pytest.raises(Exception):      # more peers than the kernels serve
        plan.set_push(flat.data_ptr(), nbytes, [other.data_ptr()] * 8)
    with pytest.raises(Exception):      # a pushed tensor outside the local buffer
        plan.set_push(flat.data_ptr(), 1024, [other.data_ptr()])
    with pytest.raises(Exception):      # a peer buffer that overlaps the local one
        plan.set_push(flat.data_ptr(), nbytes, [flat.data_ptr() + 256])
    with pytest.raises(Exception):      # a misaligned peer buffer
        plan.set_push(flat.data_ptr(), nbytes, [other.data_ptr() + 2])
    opt.step()                          # none of the refused calls left the plan in push mode
    torch.cuda.synchronize()
    assert plan.status() == 0 and not other.any()


def test_odd_matrix_outside_the_local_buffer_is_left_out():
    """A matrix that no staged path takes may lie elsewhere: the set-up is accepted, and it is not delivered."""
    import came_b200
    flat = torch.zeros(64 * 192, dtype=torch.bfloat16, device="cuda")
    params = [torch.nn.Parameter(flat.view(64, 192)), torch.nn.Parameter(torch.zeros(33, 77, dtype=torch.bfloat16, device="cuda")),
              torch.nn.Parameter(torch.zeros(40, 3, dtype=torch.bfloat16, device="cuda"))]
    for p in params:
        p.grad = torch.ones_like(p)
    opt = came_b200.CAME8bit(params, lr=1e-3)
    opt.prime_for_cuda_graph()
    mirror = torch.zeros_like(flat)
    opt._engine.set_push(flat.data_ptr(), 2 * flat.numel(), [mirror.data_ptr()])
    (plan,) = opt._engine.plans.values()
    assert plan.pushed() == [True, False, False]
    params[1].grad = torch.ones_like(params[1])      # a new address: the plan is pointed at it
    opt.step()
    torch.cuda.synchronize()
    assert plan.status() == 0 and torch.equal(mirror, flat) and bool((params[1].data != 0).all())
    # inside the buffer it is delivered
    both = torch.zeros(64 * 192 + 33 * 77 + 7, dtype=torch.bfloat16, device="cuda")
    views = [both[:64 * 192].view(64, 192), both[64 * 192:64 * 192 + 33 * 77].view(33, 77)]
    ps = [torch.nn.Parameter(v) for v in views]
    for p in ps:
        p.grad = torch.ones_like(p)
    opt = came_b200.CAME8bit(ps, lr=1e-3)
    opt.prime_for_cuda_graph()
    mirror = torch.zeros(both.numel() + 7, dtype=torch.bfloat16, device="cuda")[:both.numel()]
    opt._engine.set_push(both.data_ptr(), 2 * both.numel(), [mirror.data_ptr()])
    opt.step()
    torch.cuda.synchronize()
    assert torch.equal(mirror, both) and bool((both[:64 * 192 + 33 * 77] != 0).all())
