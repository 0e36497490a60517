"""float32 products of long contractions: with a weight, and of two activations (the gradient of a weight)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Elementwise, relative to sum |a||b|: the operands are exact sums of their planes, the products that are left out are 2^-25 of a term; eight
# truncating additions of at most 2^-23 to the accumulator of the large products, those to the one of the small products 2^-8 as large, and
# the float32 sums of the accumulators, 2^-24 each for K / 64 of them.
BOUND = 2.0 ** -20 + 2.0 ** -21


def product(x, w, b=None):
    from memorax_b200 import _C, ops
    got = _C.linear_f32(x, w, b)
    ops.check_status()
    return got


# tiles of 256 and 128 columns on pairs and of 64 on one SM, their edges, stages of 64 k and runs of two, split contractions,
# rows that start anywhere
@pytest.mark.parametrize("m,n,k", [(1, 1, 256), (127, 64, 257), (129, 130, 320), (300, 776, 513), (9000, 256, 264), (20000, 128, 384),
                                   (20001, 520, 300), (4097, 300, 1100)])
@pytest.mark.parametrize("kind", ["plain", "grows", "leaps", "wide range", "zeros first"])
def test_products_stay_within_the_bound_of_their_terms(m, n, k, kind):
    g = torch.Generator("cuda").manual_seed(m + n + k)
    x, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((m, k), (n, k), (n,)))
    at = torch.arange(k, device="cuda")
    if kind == "grows":         # from stage to stage in steps of 2^9, over the range of float32
        x *= 2.0 ** (9.0 * (at // 64) * (torch.arange(m, device="cuda")[:, None] % 3) - 60).clamp(max=40)
    elif kind == "leaps":       # one element far above its row, at any place
        x[torch.arange(m, device="cuda"), torch.randint(k, (m,), generator=g, device="cuda")] *= 2.0 ** 40
    elif kind == "wide range":  # rows and columns of very different sizes
        x *= 2.0 ** torch.randint(-60, 61, (m, 1), generator=g, device="cuda")
        w *= 2.0 ** torch.randint(-60, 61, (n, 1), generator=g, device="cuda")
    elif kind == "zeros first":
        x[:, :130] = 0
        x[::3] = 0
    got = product(x, w, b).double()
    want, scale = x.double() @ w.double().t() + b.double(), x.abs().double() @ w.abs().double().t() + b.abs().double()
    bound = BOUND * scale
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound.clamp(min=1e-300)).max())


# rows that begin anywhere: activations cut out of a larger buffer, widths that are no multiple of four
@pytest.mark.parametrize("m,n,k", [(300, 70, 257), (9000, 256, 320), (20000, 260, 514)])
def test_rows_at_any_address(m, n, k):
    torch.manual_seed(m)
    x, w = torch.empty(m * k + 1, device="cuda")[1:].view(m, k).normal_(), torch.randn(n, k, device="cuda")
    got, want, scale = product(x, w).double(), x.double() @ w.double().t(), x.abs().double() @ w.abs().double().t()
    assert bool(((got - want).abs() <= BOUND * scale).all())


# the gradient of a weight contracts the tokens of two activations: tiles of 256 x 128 on pairs and 128 x 64
# alone, their edges, runs of two stages, splits, columns that grow from stage to stage, leap, differ, begin with zeros, or start anywhere
@pytest.mark.parametrize("tokens,m,n", [(256, 1, 1), (257, 64, 127), (1000, 130, 70), (4097, 256, 300), (24000, 520, 260), (300, 2000, 1100)])
@pytest.mark.parametrize("kind", ["plain", "grows", "leaps", "wide range", "zeros first", "any address"])
def test_gradients_of_weights_stay_within_the_bound_of_their_terms(tokens, m, n, kind):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(tokens + m + n)
    a, b = (torch.randn(tokens, s, generator=g, device="cuda") for s in (m, n))
    at = torch.arange(tokens, device="cuda")[:, None]
    if kind == "grows":
        for t in (a, b):
            t *= 2.0 ** (9.0 * (at // 64) * (torch.arange(t.shape[1], device="cuda") % 3) - 60).clamp(max=0)
    elif kind == "leaps":
        for t in (a, b):
            t[torch.randint(tokens, (t.shape[1],), generator=g, device="cuda"), torch.arange(t.shape[1], device="cuda")] *= 2.0 ** 30
    elif kind == "wide range":
        for t in (a, b):
            t *= 2.0 ** torch.randint(-60, 56, (1, t.shape[1]), generator=g, device="cuda")   # (sums of 24000 terms stay below 2^128)
    elif kind == "zeros first":
        a[:130], b[:70], a[:, ::3] = 0, 0, 0
    elif kind == "any address":
        a = torch.empty(tokens * m + 1, device="cuda")[1:].view(tokens, m).copy_(a)
    w = torch.zeros(m, n, device="cuda", requires_grad=True)
    y = _C.linear_f32(b, w, None)
    got = torch.autograd.grad(y, w, a)[0].double()
    ops.check_status()
    ad, bd = a.double(), b.double()
    bound = BOUND * (ad.abs().t() @ bd.abs())
    bad = (got - ad.t() @ bd).abs() > bound
    assert not bool(bad.any()), (int(bad.sum()), float(((got - ad.t() @ bd).abs() / bound.clamp(min=1e-300)).max()))


def test_a_broken_row_stays_alone():
    torch.manual_seed(0)
    x, w = torch.randn(300, 512, device="cuda"), torch.randn(260, 512, device="cuda") / 512
    want = product(x, w)
    x[7, 300], x[9, 3], w[11, 5] = float("nan"), float("inf"), float("nan")
    got = product(x, w)
    assert bool(got[7].isnan().all()) and bool(got[:, 11].isnan().all())
    keep_r, keep_c = [i for i in range(300) if i not in (7, 9)], [i for i in range(260) if i != 11]
    assert torch.equal(got[keep_r][:, keep_c], want[keep_r][:, keep_c])
    assert not got[9][keep_c].isnan().any() and bool((got[9].sign() == w[:, 3].sign())[keep_c].all()) and float(got[9][keep_c].abs().min()) > 1e30


# the weights of the layers: complex pairs along rows and along columns, stacked ones whose pieces end inside a vector, each also
# transposed (the gradients of the inputs); against the same layers in float64
@pytest.mark.parametrize("cell", ["lru", "mingru"])
@pytest.mark.parametrize("feat,width", [(256, 128), (261, 131), (520, 300)])
def test_layers_with_long_contractions(cell, feat, width):
    from memorax_b200.memoroid import LRUCell, Memoroid, MinGRUCell
    torch.manual_seed(feat)
    bsz, steps = 3, 50
    made = (LRUCell(feat, width, r_min=0.5, r_max=0.9, max_phase=0.6) if cell == "lru" else MinGRUCell(width, in_features=feat)).cuda()
    x = torch.randn(bsz, steps, feat, device="cuda", requires_grad=True)
    gy = torch.randn(bsz, steps, feat if cell == "lru" else width, device="cuda")
    _, y = Memoroid(made)(x, torch.zeros(bsz, steps, device="cuda"), None)
    wrt = [x, *made.parameters()]
    grads = torch.autograd.grad(y, wrt, gy)
    xd, p = x.detach().double().requires_grad_(), {n: v.detach().double().requires_grad_() for n, v in made.named_parameters()}
    if cell == "lru":
        lam = torch.exp(torch.complex(-torch.exp(p["nu_log"]), torch.exp(p["theta_log"])))
        bu = xd.to(torch.complex128) @ (torch.complex(p["B_real"], p["B_imag"]) * torch.exp(p["gamma_log"])[:, None]).t()
        h, out = torch.zeros_like(bu[:, 0]), []
        for t in range(steps):
            h = lam * h + bu[:, t]
            out.append(h)
        want_y = (torch.stack(out, 1) @ torch.complex(p["C_real"], p["C_imag"]).t()).real + p["D"] * xd
    else:
        z, ht = xd @ p["z.weight"].t(), xd @ p["h.weight"].t()
        g = torch.where(ht >= 0, torch.relu(ht) + 0.5, torch.sigmoid(ht))
        h, out = torch.zeros_like(z[:, 0]), []
        for t in range(steps):
            h = torch.sigmoid(-z[:, t]) * h + torch.sigmoid(z[:, t]) * g[:, t]
            out.append(h)
        want_y = torch.stack(out, 1)
    want = torch.autograd.grad(want_y, [xd, *p.values()], gy.double())
    for name, a, b in zip(["y", "x", *p], [y, *grads], [want_y, *want]):
        assert float((a.detach().double() - b).norm() / b.norm()) <= 2e-6, name


# the skip weight's gradient: vectors and single columns, more columns than threads, remainders of the rows a block takes
@pytest.mark.parametrize("tokens,feat", [(1, 4), (700, 3), (3000, 264), (5000, 256), (2500, 1028), (600, 1300)])
def test_column_sums_of_products(tokens, feat):
    from memorax_b200.memoroid import LRUCell, Memoroid
    torch.manual_seed(tokens)
    cell = LRUCell(feat, 8).cuda()
    x, gy = torch.randn(1, tokens, feat, device="cuda"), torch.randn(1, tokens, feat, device="cuda")
    _, y = Memoroid(cell)(x, torch.zeros(1, tokens, device="cuda"), None)
    got, want = torch.autograd.grad(y, cell.D, gy)[0], (x.double() * gy.double()).sum((0, 1))
    # (float32 sums in some order: at most 24 additions in a row at these sizes, each to 2^-24 of the terms' sum)
    assert bool(((got.double() - want).abs() <= 24 * 2.0 ** -24 * (x.double() * gy.double()).abs().sum((0, 1))).all())


# Padding that holds a sentinel and meets a cotangent of exactly zero, a feature without a weight, one-hot rows, elements of all sizes: what is far
# below the largest of its row or column loses nothing, since a float32 number is the exact sum of its planes.
FAINT = ["sentinel 1e6", "sentinel 1e9", "sentinel 1e12", "sentinel 1e15", "sentinel 1e30", "one-hot", "all sizes", "left behind"]


def faint_pair(kind, g, k, m, n):
    """Operands (k, m) and (k, n) of a contraction over k."""
    a, b = (torch.randn(k, s, generator=g, device="cuda") for s in (m, n))
    at = torch.arange(k, device="cuda")
    if kind.startswith("sentinel"):
        pad = at % 32 >= 28
        a[pad, ::2], b[pad] = float(kind.split()[1]), 0
    elif kind == "one-hot":
        b = torch.zeros(k, n, device="cuda")
        b[torch.randint(k, (n,), generator=g, device="cuda"), torch.arange(n, device="cuda")] = 1
        a *= 2.0 ** -torch.randint(0, 60, (k, m), generator=g, device="cuda")
    elif kind == "all sizes":
        a *= 2.0 ** -torch.randint(0, 60, (k, m), generator=g, device="cuda")
        b *= 2.0 ** -torch.randint(0, 60, (k, n), generator=g, device="cuda")
    else:   # large numbers at the end meet zeros there
        a *= torch.where(at < k - 40, 2.0 ** -40, 2.0 ** 60)[:, None]
        b[k - 40:] = 0
    return a, b


def within(got, a, b):
    want, scale = a.double().t() @ b.double(), a.double().abs().t() @ b.double().abs()
    bad = (got.double() - want).abs() > BOUND * scale
    assert not bool(bad.any()), (int(bad.sum()), float(((got.double() - want).abs() / (BOUND * scale).clamp(min=1e-300)).max()))


@pytest.mark.parametrize("kind", FAINT)
@pytest.mark.parametrize("m,n,k", [(1, 1, 256), (300, 776, 513), (1500, 300, 1100), (9000, 256, 264), (20001, 130, 300)])
@pytest.mark.parametrize("large", ["activations", "weight"])
def test_faint_terms_of_products_with_a_weight(kind, m, n, k, large):
    g = torch.Generator("cuda").manual_seed(m + n + k)
    if large == "activations":
        x, w = (t.t().contiguous() for t in faint_pair(kind, g, k, m, n))
    else:
        w, x = (t.t().contiguous() for t in faint_pair(kind, g, k, n, m))
    within(product(x, w), x.t(), w.t())


@pytest.mark.parametrize("kind", FAINT)
@pytest.mark.parametrize("tokens,m,n", [(256, 1, 1), (1000, 130, 70), (4097, 256, 300), (24000, 300, 40), (300, 1500, 500)])
@pytest.mark.parametrize("large", ["cotangents", "activations"])
def test_faint_terms_of_gradients_of_weights(kind, tokens, m, n, large):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(tokens + m + n)
    a, b = faint_pair(kind, g, tokens, m, n)
    if large == "activations":
        a, b = b, a
    w = torch.zeros(a.shape[1], b.shape[1], device="cuda", requires_grad=True)
    got = torch.autograd.grad(_C.linear_f32(b, w, None), w, a)[0]
    ops.check_status()
    within(got, a, b)
