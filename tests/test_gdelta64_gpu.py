"""Gated delta rule, heads of 64, at the sizes where its chunks and sequences end: one step, one short of, at and one past
a chunk, several chunks with every barrier phase wrapping, resets everywhere, and more sequences than fit on the chip at
once.  Same oracle and tolerances as the heads of 128.  A first step's dalpha is <dS0, S0> / alpha, 64 x 64 products of
bf16-rounded factors that largely cancel: it has the rounding of that sum on top, four times its standard deviation of
0.8 x 2^-9 |dS0 o S0| / alpha (both factors off by up to 2^-9, evenly spread)."""
import pytest
import torch

from oracle import memoroid_oracle as mo
from test_gdelta_gpu import ATOL, GRAD_RTOL, make_case, max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,p_done", [((2, 1, 1), 0.0), ((1, 63, 2), 0.1), ((2, 64, 1), 1.0), ((1, 65, 3), 0.05), ((1, 450, 2), 0.004),
                                          ((60, 70, 8), 0.02)])
@pytest.mark.parametrize("carry", [False, True])
def test_against_the_oracle(shape, p_done, carry):
    from memorax_b200 import ops
    q, k, v, alpha, beta, s0, done = make_case(sum(shape), *shape, p_done, not carry, dim=64)
    gen = torch.Generator().manual_seed(8)
    d_o = torch.randn(*q.shape, generator=gen).bfloat16()
    ds_last = torch.randn(*s0.shape, generator=gen) * 0.2 if carry else torch.zeros_like(s0)
    leaves = [t.double().requires_grad_() for t in (q, k, v, alpha, beta, s0)]
    o_ref, s_ref = mo.gdelta_seq(*leaves, done.double())
    ((o_ref * d_o.double()).sum() + (s_ref * ds_last.double()).sum()).backward()
    x = [t.cuda() for t in (q, k, v, alpha, beta)]
    cu = lambda t: t.cuda() if carry else None
    o, s_last, states = ops.gdelta_fwd(*x, cu(s0), done.cuda(), save_states=True, check=True)
    plain, _, _ = ops.gdelta_fwd(*x, cu(s0), done.cuda(), check=True)
    assert torch.equal(plain, o)
    assert max_abs(o.float(), o_ref) <= ATOL
    assert max_abs(s_last, s_ref) <= 1e-2 * max(1.0, float(s_ref.detach().abs().max()))
    outs = ops.gdelta_bwd(*x, d_o.cuda(), states, done.cuda(), cu(ds_last), check=True)
    first = 4 * 0.8 * 2 ** -9 * float(((leaves[5].grad * leaves[5].detach()).flatten(2).norm(dim=2) / alpha[:, 0]).max())
    for got, leaf, name in zip(outs, leaves, ["dq", "dk", "dv", "dalpha", "dbeta", "ds0"]):
        err, tol = max_abs(got.float(), leaf.grad), GRAD_RTOL * max(1.0, float(leaf.grad.abs().max()))
        if name == "dalpha":
            tol = max(tol, first)
        assert err <= tol, f"{name}: {err:.4f} > {tol:.4f}"
