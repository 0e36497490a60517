"""The bf16 linear-attention and delta-rule layers: the native call (one product for the inputs, strided chunk kernels,
one-step forms) against the same layer composed from its parts, and both directions of carry and resets."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(model, x, done, carry, gy, gc, wrt, native):
    from memorax_b200.memoroid import MemoroidCellBase
    cell = model.cell
    out, y = model(x, done, carry) if native else MemoroidCellBase.layer(cell, x, done, carry)
    grads = torch.autograd.grad([y, *out], wrt, [gy, *gc])
    return [y, *out, *grads]


def _close(got, want, tol):
    got, want = got.detach().float(), want.detach().float()
    assert got.shape == want.shape
    assert float((got - want).norm()) <= tol * max(1e-3 * want.numel() ** 0.5, float(want.norm())), float((got - want).norm() / want.norm())


# head dims and head counts that pad the joint projection; T = 1 with gradients stays on the chunk kernels
@pytest.mark.parametrize("kind,heads,dim", [("linattn", 4, 64), ("linattn", 2, 32), ("linattn", 3, 24), ("deltanet", 2, 64), ("deltanet", 3, 128)])
@pytest.mark.parametrize("bsz,steps", [(3, 1), (2, 70)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_native_layer_equals_the_composed_one(kind, heads, dim, bsz, steps, with_carry):
    from memorax_b200.memoroid import DeltaNetCell, LinearAttentionCell, Memoroid
    torch.manual_seed(0)
    feat = 96
    cell = (LinearAttentionCell if kind == "linattn" else DeltaNetCell)(feat, dim, heads)
    model = Memoroid(cell).cuda().bfloat16()
    x = torch.randn(bsz, steps, feat, device="cuda").bfloat16().requires_grad_()
    done = torch.rand(bsz, steps, device="cuda") < 0.1
    leaves = [(0.3 * torch.randn(bsz, 1, heads, dim, dim, device="cuda")).requires_grad_()]
    if kind == "linattn":
        leaves.append(torch.rand(bsz, 1, heads, dim, device="cuda").requires_grad_())
    carry = tuple(leaves) if with_carry else None
    gy, gc = torch.randn_like(x), [torch.randn_like(t) for t in leaves]
    wrt = [x, *model.parameters()] + (leaves if with_carry else [])
    want = _run(model, x, done, carry, gy, gc, wrt, native=False)
    got = _run(model, x, done, carry, gy, gc, wrt, native=True)
    for g, w in zip(got, want):
        _close(g, w, 2e-2)
    with torch.no_grad():
        out, y = model(x, done, carry)
    for g, w in zip([y, *out], want):
        _close(g, w, 2e-2)


# one step: few rows (fragments of 16 x 32, K split over four warps) and many (library product); no carry = zero state
@pytest.mark.parametrize("kind,heads,dim", [("linattn", 4, 64), ("linattn", 2, 32), ("deltanet", 2, 64), ("deltanet", 8, 128)])
@pytest.mark.parametrize("bsz", [1, 17, 300])
@pytest.mark.parametrize("with_carry", [False, True])
def test_one_step_equals_a_segment_of_one(kind, heads, dim, bsz, with_carry):
    from memorax_b200.memoroid import DeltaNetCell, LinearAttentionCell, Memoroid, MemoroidCellBase
    torch.manual_seed(1)
    feat = 128
    model = Memoroid((LinearAttentionCell if kind == "linattn" else DeltaNetCell)(feat, dim, heads)).cuda().bfloat16()
    x = torch.randn(bsz, 1, feat, device="cuda").bfloat16()
    done = torch.rand(bsz, 1, device="cuda") < 0.2
    leaves = [0.3 * torch.randn(bsz, 1, heads, dim, dim, device="cuda")]
    if kind == "linattn":
        leaves.append(torch.rand(bsz, 1, heads, dim, device="cuda"))
    carry = tuple(leaves) if with_carry else None
    with torch.no_grad():
        got_c, got = model(x, done, carry)
        want_c, want = MemoroidCellBase.layer(model.cell, x, done, carry)
    for g, w in zip([got, *got_c], [want, *want_c]):
        _close(g, w, 1e-2)


# a carry cut out of a flat buffer starts at any float: linear attention takes it, the delta rule's kernels refuse it
@pytest.mark.parametrize("kind,heads,dim", [("linattn", 4, 64), ("linattn", 2, 32), ("deltanet", 2, 64), ("deltanet", 8, 128)])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_one_step_from_a_carry_at_any_address(kind, heads, dim, offset):
    from memorax_b200._lib import MxkError
    from memorax_b200.memoroid import DeltaNetCell, LinearAttentionCell, Memoroid
    torch.manual_seed(2)
    bsz, feat = 5, 128
    model = Memoroid((LinearAttentionCell if kind == "linattn" else DeltaNetCell)(feat, dim, heads)).cuda().bfloat16()
    x, done = torch.randn(bsz, 1, feat, device="cuda").bfloat16(), torch.zeros(bsz, 1, dtype=torch.bool, device="cuda")
    s0 = 0.3 * torch.randn(bsz, 1, heads, dim, dim, device="cuda")
    flat = torch.zeros(s0.numel() + 4, device="cuda")
    cut = flat[offset:offset + s0.numel()].view_as(s0).copy_(s0)
    rest = (torch.rand(bsz, 1, heads, dim, device="cuda"),) if kind == "linattn" else ()
    with torch.no_grad():
        if kind == "deltanet":
            with pytest.raises(MxkError):
                model(x, done, (cut,))
            return
        want_c, want = model(x, done, (s0, *rest))
        got_c, got = model(x, done, (cut, *rest))
    for g, w in zip([got, *got_c], [want, *want_c]):
        _close(g, w, 1e-2)


# inputs cut out of a larger buffer start at any bf16: not for the 16-byte loads of the small products
@pytest.mark.parametrize("kind,heads,dim", [("linattn", 4, 64), ("deltanet", 2, 64)])
@pytest.mark.parametrize("bsz,steps", [(7, 1), (2, 70)])
@pytest.mark.parametrize("offset", [1, 4])
def test_inputs_at_any_address(kind, heads, dim, bsz, steps, offset):
    from memorax_b200.memoroid import DeltaNetCell, LinearAttentionCell, Memoroid
    torch.manual_seed(3)
    feat = 128
    model = Memoroid((LinearAttentionCell if kind == "linattn" else DeltaNetCell)(feat, dim, heads)).cuda().bfloat16()
    x, done = torch.randn(bsz, steps, feat, device="cuda").bfloat16(), torch.rand(bsz, steps, device="cuda") < 0.1
    flat = torch.zeros(x.numel() + 8, device="cuda", dtype=torch.bfloat16)
    cut = flat[offset:offset + x.numel()].view_as(x).copy_(x)
    with torch.no_grad():
        want_c, want = model(x, done)
        got_c, got = model(cut, done)
    for g, w in zip([got, *got_c], [want, *want_c]):
        _close(g, w, 1e-2)


# The native delta-rule layer adds in other orders than the composed one before it rounds to bf16.  Neither is the exact one:
# both are as far from float64 as bf16 makes them, and no further from each other than two such errors are.
@pytest.mark.parametrize("heads,dim", [(4, 64), (2, 128)])
def test_native_gradients_are_as_close_to_float64_as_the_composed_ones(heads, dim):
    import torch.nn.functional as F
    from memorax_b200.memoroid import DeltaNetCell, Memoroid
    from oracle import memoroid_oracle as mo
    torch.manual_seed(4)
    bsz, steps, feat = 17, 132, 256
    model = Memoroid(DeltaNetCell(feat, dim, heads)).cuda().bfloat16()
    x = torch.randn(bsz, steps, feat, device="cuda").bfloat16().requires_grad_()
    done = torch.rand(bsz, steps, device="cuda") < 0.02
    gy = torch.randn_like(x)
    wrt = [x, *model.parameters()]
    runs = [_run(model, x, done, None, gy, [torch.zeros(bsz, 1, heads, dim, dim, device="cuda")], wrt, native=n)[2:] for n in (True, False)]
    p = {k: v.detach().double().cpu().requires_grad_() for k, v in model.cell.named_parameters()}
    xd = x.detach().double().cpu().requires_grad_()
    head = lambda name: F.linear(xd, p[name + ".weight"]).view(bsz, steps, heads, dim)
    b_logit, a_logit = F.linear(xd, p["gate.weight"], p["gate.bias"]).chunk(2, dim=-1)
    o, _ = mo.gdelta_seq(F.normalize(head("query"), dim=-1), F.normalize(head("key"), dim=-1), head("value"), torch.exp(-F.softplus(a_logit)),
                         torch.sigmoid(b_logit), torch.zeros(bsz, heads, dim, dim, dtype=torch.float64), done.cpu().double())
    o = F.rms_norm(o.reshape(bsz, steps, -1), (heads * dim,), p["norm.weight"], 1e-6)
    y = F.linear(o, p["output_projection.weight"], p["output_projection.bias"])
    want = torch.autograd.grad(y, [xd, *(p[k] for k, _ in model.cell.named_parameters())], gy.double().cpu())
    for (name, _), native, composed, ref in zip([("x", None), *model.cell.named_parameters()], *runs, want):
        native, composed = native.double().cpu(), composed.double().cpu()
        off = [float((t - ref).norm() / ref.norm()) for t in (native, composed)]
        apart = float((native - composed).norm() / ref.norm())
        assert off[0] <= 1.1 * off[1] + 2 ** -10 and apart <= off[0] + off[1], (name, off, apart)
