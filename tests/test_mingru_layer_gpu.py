"""The MinGRU layer (Dense layers, gate math, scan, read-out) and its gradients against the oracle."""
import pytest
import torch

from oracle import memoroid_oracle as mo

pytestmark = pytest.mark.gpu


# sixteen stretches of at most 8 steps per turn of 128: T on both sides of a step, a turn and a remainder; T = 1 is the
# fused acting step (without gradients); D on both sides of a block's 32 channels
@pytest.mark.parametrize("shape", [(9, 1, 5, 3), (2, 15, 8, 33), (2, 16, 8, 32), (3, 129, 20, 31), (1, 300, 64, 65)])
@pytest.mark.parametrize("with_carry", [False, True])
@pytest.mark.parametrize("scale", [2.0, 60.0])   # 60: pre-activations outside the linear form's range
def test_mingru_layer_matches_the_oracle(shape, with_carry, scale):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    bsz, steps, feat, dim = shape
    torch.manual_seed(0)
    cell = MinGRUCell(dim, in_features=feat).cuda()
    x = (scale * torch.randn(bsz, steps, feat, device="cuda")).requires_grad_()
    done = torch.rand(bsz, steps, device="cuda") < 0.05
    carry = (torch.randn(bsz, 1, dim, device="cuda").requires_grad_(), -torch.rand(bsz, 1, dim, device="cuda")) if with_carry else None
    gy, gl = torch.randn(bsz, steps, dim, device="cuda"), torch.randn(bsz, 1, dim, device="cuda")
    wrt = [x, cell.z.weight, cell.h.weight] + ([carry[0]] if with_carry else [])
    (h, a), y = Memoroid(cell)(x, done, carry)
    grads = torch.autograd.grad((y, h), wrt, (gy, gl))
    with torch.no_grad():
        (h_n, a_n), y_n = Memoroid(cell)(x, done, carry)

    d64 = lambda t: t.detach().cpu().double()
    xd, wz, wh = (d64(t).requires_grad_() for t in wrt[:3])
    x0 = d64(carry[0])[:, 0].requires_grad_() if with_carry else torch.full((bsz, dim), -float("inf"), dtype=torch.float64)
    z, ht, sp = xd @ wz.t(), xd @ wh.t(), torch.nn.functional.softplus
    ls = -sp(-z) + torch.where(ht >= 0, torch.log(torch.relu(ht) + 0.5), -sp(-ht))
    xs, a_ref = mo.mingru_seq(ls, -sp(z), x0, d64(done), d64(carry[1])[:, 0] if with_carry else None)
    want = torch.autograd.grad((xs.exp(), xs[:, -1:]), [xd, wz, wh] + ([x0] if with_carry else []), (d64(gy), d64(gl)))
    err = lambda got, ref: float((got.detach().cpu().reshape(ref.shape) - ref.detach()).abs().max()) / max(1e-30, float(ref.detach().abs().max()))
    for got, ref in ((h, xs[:, -1]), (h_n, xs[:, -1]), (a, a_ref), (a_n, a_ref), (y, xs.exp()), (y_n, xs.exp())):
        assert err(got, ref) <= 1e-5
    for got, ref in zip(grads, want):
        assert err(got, ref) <= 1e-4
