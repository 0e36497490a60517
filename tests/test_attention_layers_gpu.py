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
