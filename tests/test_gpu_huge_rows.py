"""Rows of more than 2^31 bytes: [2, 2^29 + 1] in fp32, a first step of CAME against the same formulas in torch
(CAME.py:117-172), whose sums are taken in fp64.  Tolerance: a row's 2^23 partial sums are added in eight fp32 chains of
2^20, whose roundings leave about sqrt(2^20) * 2^-24 = 6e-5 of the sum, and the row factors scale everything after them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_first_step_of_a_matrix_with_huge_rows():
    import came_b200
    rows, cols = 2, 2 ** 29 + 1
    lr, (b1, b2, b3), eps0, eps1 = 1e-2, (0.9, 0.999, 0.9999), 1e-30, 1e-16
    gen = torch.Generator(device="cuda").manual_seed(3)
    p = torch.nn.Parameter(torch.full((rows, cols), 0.5, device="cuda"))
    p.grad = torch.empty(rows, cols, device="cuda").normal_(generator=gen)
    p.grad[1] *= 10.0
    opt = came_b200.CAME([p], lr=lr, betas=(b1, b2, b3), eps=(eps0, eps1))
    opt.step()
    assert all(plan.status() == 0 for plan in opt._engine.plans.values())
    g, st = p.grad, opt.state[p]

    def near(got, want):
        assert ((got.double() - want.double()).norm() / want.double().norm()).item() <= 2e-4

    def vectors(x, beta, eps):
        row = torch.stack([x(i).sum(dtype=torch.float64) / cols + eps for i in range(rows)]).float() * (1 - beta)
        col = (sum(x(i) for i in range(rows)) / rows + eps) * (1 - beta)
        return row, col, (row / row.mean()).rsqrt(), col.rsqrt()

    v_row, v_col, r, c = vectors(lambda i: g[i] * g[i], b2, eps0)
    near(st["exp_avg_sq_row"], v_row)
    near(st["exp_avg_sq_col"], v_col)
    u = [g[i] * r[i] * c for i in range(rows)]
    rms = (sum((x * x).sum(dtype=torch.float64) for x in u) / (rows * cols)).sqrt()
    inv = (1.0 / rms.clamp(min=1.0)).float()
    for i in range(rows):
        u[i] *= inv
        near(st["exp_avg"][i], u[i] * (1 - b1))
    s_row, s_col, rr, rc = vectors(lambda i: (u[i] * b1) ** 2, b3, eps1)
    near(st["exp_avg_res_row"], s_row)
    near(st["exp_avg_res_col"], s_col)
    for i in range(rows):
        near(p.data[i] - 0.5, -lr * (u[i] * (1 - b1)) * rr[i] * rc)
