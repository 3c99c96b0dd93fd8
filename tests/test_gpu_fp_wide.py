"""fp32-state layout (CAMECUDA): the shared-memory staged momentum / apply passes against the generic kernels and the
oracle, on shapes that exercise ragged last bands (rows not a multiple of 8), ragged tile widths (columns not a
multiple of 1024), several tiles per matrix and every weight-decay form.  Reference: kCameFactoredExpAvgRes,
kCameFactoredParamUpdate (came_kernels.cu:2307-2342, 2487-2511)."""
import os

import pytest
import torch

from oracle import came_oracle as orc
from tests.parity_util import kernels_of, relerr, run_pair
from tests.test_gpu_parity import H_DEFAULT, _check_fp, _dt

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("staged")]      # (as small sets they would take the whole-step kernel)

SHAPES = [(130, 1088), (257, 2304), (64, 64), (7, 192), (1000, 1024), (300, 4096), (129, 3072)]


def _run(dtype, disable_fast, wd, steps=3):
    import came_b200
    os.environ["CAME_B200_DISABLE_FAST"] = "1" if disable_fast else "0"
    try:
        gen = torch.Generator(device="cuda").manual_seed(5)
        params = [torch.nn.Parameter((torch.randn(s, device="cuda", generator=gen) * 0.02).to(dtype)) for s in SHAPES]
        opt = came_b200.CAMECUDA(params, **dict(H_DEFAULT, weight_decay=wd))
        for _ in range(steps):
            for i, p in enumerate(params):
                p.grad = (torch.randn(p.shape, device="cuda", generator=gen) * 10.0 ** (-2 - (i % 3))).to(dtype)
            opt.step()
        for plan in opt._engine.plans.values():
            assert plan.status() == 0
        names = kernels_of(opt)      # (a step more, on both sides)
        assert names == {"generic"} if disable_fast else {"moment", "apply"} <= names and "generic" not in names
        return params, opt
    finally:
        os.environ.pop("CAME_B200_DISABLE_FAST", None)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("wd", [0.0, 1e-2])
def test_staged_equals_generic(dtype, wd):
    pa, oa = _run(_dt(dtype), False, wd)
    pb, ob = _run(_dt(dtype), True, wd)
    for x, y in zip(pa, pb):
        if dtype == "float32":
            assert relerr(x.data, y.data) <= 1e-6
        else:
            # 16-bit parameters: the two orders of fp32 roundings may land on either side of a rounding boundary of the
            # stored value; such elements (rare) differ by one unit in the last place of the value they had at that
            # step, and keep that absolute difference afterwards (parameters here are N(0, 0.02^2))
            differ = (x.data != y.data)
            assert differ.float().mean().item() <= 2e-3
            ulp = 2.0 ** (-7 if dtype == "bfloat16" else -10)
            assert ((x.data.float() - y.data.float()).abs() <= 2 * ulp * (y.data.float().abs() + 0.05)).all()
        for k in ("exp_avg", "exp_avg_sq_row", "exp_avg_sq_col", "exp_avg_res_row", "exp_avg_res_col"):
            assert relerr(oa.state[x][k], ob.state[y][k]) <= 2e-5, k      # norm-wise: entries near zero are cancellations


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_staged_against_oracle(dtype):
    import came_b200
    out, opt, _ = run_pair(came_b200.CAMECUDA, lambda dim: orc.CUDAFP, SHAPES, _dt(dtype), 4, H_DEFAULT, seed=44,
                           per_tensor_scale=True)
    _check_fp(out, _dt(dtype))
    for plan in opt._engine.plans.values():
        assert plan.status() == 0
    assert {"moment", "apply"} <= kernels_of(opt)
