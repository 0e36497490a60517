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


# g's slope jumps at zero: an element whose product is rounding only takes the side of the plain float32 sum in the order
# of k, at every scale.  Weights orthogonal to the inputs up to rounding; every step starts afresh, so that the gradient of
# a channel's weights is sigmoid(z) g'(h~) x with g' = 1 or 1/4.
@pytest.mark.parametrize("scale", [1e-6, 1.0, 60.0, 1e4])
@pytest.mark.parametrize("w_scale", [1e-4, 1.0])
def test_the_side_of_the_kink_is_that_of_the_sum_in_order(scale, w_scale):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    torch.manual_seed(0)
    steps, feat, dim, t = 3, 512, 64, 1
    cell = MinGRUCell(dim, in_features=feat)
    x = scale * torch.randn(1, steps, feat)
    xt = x[0, t].double()
    with torch.no_grad():
        w = cell.h.weight.double()
        cell.h.weight.copy_(w_scale * (w - (w @ xt)[:, None] * xt / (xt @ xt)))
        cell.z.weight.zero_()
    terms = (cell.h.weight.double() * xt).detach()     # exact: 24 x 24 bits
    acc = torch.zeros(dim)
    for k in range(feat):
        acc = (acc.double() + terms[:, k]).float()
    assert bool(((acc >= 0) != (terms.sum(1) >= 0)).any())   # the order of the sum does decide
    cell, x = cell.cuda(), x.cuda()
    gy = torch.zeros(1, steps, dim, device="cuda")
    gy[:, t] = 1
    _, y = Memoroid(cell)(x, torch.ones(1, steps, device="cuda"), None)
    (gw,) = torch.autograd.grad(y, [cell.h.weight], gy)
    slope = (gw.cpu().double() @ xt) / (xt @ xt) / 0.5
    want = torch.where(acc >= 0, 1.0, 0.25).double()
    assert float((slope - want).abs().max()) <= 1e-3


# The same with few channels of a warp at the kink, which the warp sums one by one in chunks of 128 terms, and with one more
# than that; blocks of sixteen warps (one sequence) and of eight (a grid beyond two blocks an SM)
@pytest.mark.parametrize("feat", [65, 128, 130, 515])
@pytest.mark.parametrize("near", [(0,), (3, 17, 39), (1, 2, 30, 31), (4, 5, 6, 7, 8)])
@pytest.mark.parametrize("bsz", [1, 200])
def test_few_channels_at_the_kink(feat, near, bsz):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    torch.manual_seed(feat)
    steps, dim, b, t = 11, 40, bsz // 2, 9
    cell = MinGRUCell(dim, in_features=feat)
    x = torch.randn(bsz, steps, feat)
    xt, rows = x[b, t].double(), list(near)
    acc = torch.zeros(len(rows))
    with torch.no_grad():
        w = cell.h.weight[rows].double()
        cell.h.weight[rows] = (w - (w @ xt)[:, None] * xt / (xt @ xt)).float()
        cell.z.weight.zero_()
        terms = cell.h.weight[rows].double() * xt
        for k in range(feat):
            acc = (acc.double() + terms[:, k]).float()
    cell, x = cell.cuda(), x.cuda()
    gy = torch.zeros(bsz, steps, dim, device="cuda")
    gy[b, t] = 1
    _, y = Memoroid(cell)(x, torch.ones(bsz, steps, device="cuda"), None)
    (gw,) = torch.autograd.grad(y, [cell.h.weight], gy)
    slope = (gw.cpu().double() @ xt) / (xt @ xt) / 0.5
    # float32 logarithms of the states at magnitude 1/2: their errors are below 1e-5 of the slopes 1 and 1/4
    assert float((slope[rows] - torch.where(acc >= 0, 1.0, 0.25).double()).abs().max()) <= 1e-3


# Two large terms that nearly cancel, for many tokens and channels, in short and in long products.  A channel's own feature is zero in
# every input and its weight is 2^-10, so that the inputs' gradients there are those of the pre-activations, 1/2 g'.
@pytest.mark.parametrize("feat", [130, 256, 515])
def test_cancelling_terms_at_the_kink(feat):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    torch.manual_seed(feat)
    bsz, steps, dim = 64, 128, 64
    cell = MinGRUCell(dim, in_features=feat)
    x = torch.zeros(bsz, steps, feat)
    x[..., 2] = 1 + torch.rand(bsz, steps)
    x[..., feat - 1] = -x[..., 2] * (1 + 2.0 ** -20 * torch.randn(bsz, steps))
    with torch.no_grad():
        cell.z.weight.zero_()
        w = cell.h.weight.zero_()
        w[:, 2] = 1 + torch.rand(dim)
        w[:, feat - 1] = w[:, 2] * (1 + 2.0 ** -20 * torch.randn(dim))
        w[torch.arange(dim), 3 + torch.arange(dim)] = 2.0 ** -10
        first = (x[..., 2].double()[..., None] * w[:, 2].double()).float()              # the sum in order: one rounding,
        side = first.double() + x[..., feat - 1].double()[..., None] * w[:, feat - 1].double() >= 0   # then its sign
    cell, x = cell.cuda(), x.cuda().requires_grad_()
    _, y = Memoroid(cell)(x, torch.ones(bsz, steps, device="cuda"), None)
    slope = torch.autograd.grad(y, x, torch.ones_like(y))[0][..., 3:3 + dim].cpu() * 2 ** 11
    assert float((slope - torch.where(side, 1.0, 0.25)).abs().max()) <= 1e-3, int(((slope > 0.6) != side).sum())


# elements that are zero or tiny because the inputs or the weights are need no second look, which costs thousands of cycles
@pytest.mark.parametrize("case", ["zero inputs", "small inputs", "padding", "zero channels", "small channels", "one-hot inputs, pruned weights"])
def test_no_input_is_slow(case):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    torch.manual_seed(0)
    bsz, steps, dim = 32, 128, 256
    cell = MinGRUCell(dim).cuda()
    model, done = Memoroid(cell), torch.zeros(bsz, steps, device="cuda")
    x = torch.randn(bsz, steps, dim, device="cuda")

    def time(x):
        x, times = x.requires_grad_(), []
        for _ in range(8):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            model(x, done)
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)
    usual = time(x.clone())
    rows, w = torch.rand(dim, 1, device="cuda"), cell.h.weight.detach()
    if case == "zero inputs":
        x.zero_()
    elif case == "small inputs":
        x *= 1e-6
    elif case == "padding":
        x[:, 100:] = 0
    elif case == "zero channels":
        w *= rows > 0.1
    elif case == "small channels":
        w *= torch.where(rows > 0.1, 1.0, 1e-6)
    else:
        x = torch.zeros_like(x).scatter_(2, torch.randint(0, dim, (bsz, steps, 1), device="cuda"), 1.0)
        w *= torch.rand_like(w) > 0.5
    assert time(x) <= 3 * usual


# three turns of 100 steps, in linear or in log form by the size of their pre-activations: the state between two turns is in
# the form of the one it was left by
@pytest.mark.parametrize("large", [(0,), (1,), (2,), (0, 1), (1, 2), (0, 2)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_turns_in_different_forms(large, with_carry):
    from memorax_b200.memoroid import MinGRUCell, Memoroid
    bsz, steps, feat, dim = 2, 300, 16, 40
    torch.manual_seed(0)
    cell = MinGRUCell(dim, in_features=feat).cuda()
    x = torch.randn(bsz, steps, feat, device="cuda")
    for turn in large:
        x[:, turn * 100:turn * 100 + 100] *= 40
    x.requires_grad_()
    done = torch.rand(bsz, steps, device="cuda") < 0.01
    carry = (3 * torch.randn(bsz, 1, dim, device="cuda").requires_grad_(), torch.zeros(bsz, 1, dim, device="cuda")) if with_carry else None
    gy, gl = torch.randn(bsz, steps, dim, device="cuda"), torch.randn(bsz, 1, dim, device="cuda")
    wrt = [x, cell.z.weight, cell.h.weight] + ([carry[0]] if with_carry else [])
    (h, _), y = Memoroid(cell)(x, done, carry)
    grads = torch.autograd.grad((y, h), wrt, (gy, gl))
    with torch.no_grad():
        (h_n, _), y_n = Memoroid(cell)(x, done, carry)
    assert torch.equal(h_n, h) and torch.equal(y_n, y)
    d64 = lambda t: t.detach().cpu().double()
    xd, wz, wh = (d64(t).requires_grad_() for t in wrt[:3])
    x0 = d64(carry[0])[:, 0].requires_grad_() if with_carry else torch.full((bsz, dim), -float("inf"), dtype=torch.float64)
    z, ht, sp = xd @ wz.t(), xd @ wh.t(), torch.nn.functional.softplus
    xs, _ = mo.mingru_seq(-sp(-z) + torch.where(ht >= 0, torch.log(torch.relu(ht) + 0.5), -sp(-ht)), -sp(z), x0, d64(done), None)
    want = torch.autograd.grad((xs.exp(), xs[:, -1:]), [xd, wz, wh] + ([x0] if with_carry else []), (d64(gy), d64(gl)))
    err = lambda got, ref: float((got.detach().cpu().reshape(ref.shape) - ref.detach()).abs().max()) / max(1e-30, float(ref.detach().abs().max()))
    assert err(h, xs[:, -1]) <= 1e-5 and err(y, xs.exp()) <= 1e-5
    for got, ref in zip(grads, want):
        assert err(got, ref) <= 1e-4


# a step that is not finite spoils its episode, and ends with it: in the same stretch of steps, turn, and in a later one
@pytest.mark.parametrize("steps,bad,reset", [(20, 3, 9), (100, 10, 12), (100, 3, 70), (300, 50, 60), (300, 50, 250)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("with_carry", [False, True])
def test_a_broken_episode_ends_at_its_reset(steps, bad, reset, value, raw, with_carry):
    from memorax_b200.memoroid import MinGRUCell, Memoroid, MemoroidCellBase
    torch.manual_seed(0)
    bsz, dim = 2, 40
    cell = MinGRUCell(dim).cuda()
    layer = (lambda *a: MemoroidCellBase.layer(cell, *a)) if raw else Memoroid(cell)
    x = torch.randn(bsz, steps, dim, device="cuda")
    x[:, bad] = value
    x.requires_grad_()
    done = torch.zeros(bsz, steps, device="cuda")
    done[:, reset] = 1
    gy = torch.zeros(bsz, steps, dim, device="cuda")
    gy[:, reset:] = torch.randn(bsz, steps - reset, dim, device="cuda")
    carry = (torch.full((bsz, 1, dim), value, device="cuda"), torch.zeros(bsz, 1, dim, device="cuda")) if with_carry else None
    (h, a), y = layer(x, done, carry)
    (gx,) = torch.autograd.grad(y, x, gy)
    rest = x.detach()[:, reset:].requires_grad_()
    (h2, a2), y2 = layer(rest, done[:, reset:], None)
    (gx2,) = torch.autograd.grad(y2, rest, gy[:, reset:])
    for got, want in ((h, h2), (a, a2), (y[:, reset:], y2), (gx[:, reset:], gx2)):
        assert float((got - want).detach().abs().max()) <= 1e-5 * max(1.0, float(want.detach().abs().max()))
