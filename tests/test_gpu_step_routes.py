"""Sizes at which the whole-step kernel and the 3 x 3 / 1 x 1 kernels change their inner route: enough flat blocks and chunks
that a warp or CTA goes through several with the next under way, whole bands next to ragged ones, rows on and off the
16-byte boundary, thin matrices.  Tolerances as in tests/test_gpu_parity.py."""
import pytest
import torch

from oracle import came_oracle as orc
from tests.parity_util import run_pair
from tests.test_gpu_parity import H_DEFAULT, H_LLAMA, _check_8bit, _check_fp, _dt

pytestmark = pytest.mark.gpu

# at most 3 CTAs of 8 warps on 148 SMs take 3552 blocks of 256 elements at a time: 5 rounds and a ragged last one
WIDE = [(3001, 1496), (2999, 1501)]
BANDS = [(272, 192), (273, 200), (271, 201), (400, 1032)]
THIN = [(640, 16), (1040, 24), (999, 17), (16, 640)]      # bands mostly empty


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("shapes,steps", [(WIDE, 2), (BANDS, 4), (THIN, 4)])
def test_flat_layout(dtype, shapes, steps):
    import came_b200
    out, opt, _ = run_pair(came_b200.CAME8bitFull, lambda dim: orc.FLAT8, shapes, _dt(dtype), steps, H_LLAMA, seed=71)
    _check_8bit(out, _dt(dtype))
    assert all(plan.status() == 0 for plan in opt._engine.plans.values())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("shapes", [BANDS, THIN])
def test_bands(dtype, shapes):
    import came_b200
    out, _, _ = run_pair(came_b200.CAME8bit, lambda dim: orc.TILE8, shapes, _dt(dtype), 4, H_LLAMA, seed=72)
    _check_8bit(out, _dt(dtype))
    out, _, _ = run_pair(came_b200.CAMECUDA, lambda dim: orc.CUDAFP, shapes, _dt(dtype), 4, H_DEFAULT, seed=73)
    _check_fp(out, _dt(dtype))


@pytest.mark.parametrize("cls_name,preset", [("CAME8bitFull", orc.FLAT8_CPU), ("CAMECUDA", orc.CUDAFP_GENERIC)])
def test_many_chunks(cls_name, preset):
    """More chunks of 256 matrices than 3 CTAs per SM: a CTA goes through several, the last one short."""
    import came_b200
    out, _, _ = run_pair(getattr(came_b200, cls_name), lambda dim: preset, [(1151, 101, 3, 3)], torch.float16, 2, H_LLAMA, seed=76)
    (_check_8bit if cls_name == "CAME8bitFull" else _check_fp)(out, torch.float16)
