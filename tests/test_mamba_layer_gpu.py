"""The fused Mamba layer against the same layer composed in float64 (the scan as the oracle's sequential recurrence)."""
import pytest
import torch

from oracle import memoroid_oracle as mo

pytestmark = pytest.mark.gpu


# stretches of 64 steps in quarters of 16, with the convolution's three-step halo across them
@pytest.mark.parametrize("shape", [(2, 1, 24, 1), (3, 16, 40, 2), (2, 65, 33, 2), (1, 150, 64, 4)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_mamba_layer_and_its_gradients(shape, with_carry):
    from memorax_b200.memoroid import MambaCell, Memoroid
    bsz, steps, feat, heads = shape
    torch.manual_seed(0)
    cell = MambaCell(feat, num_heads=heads).cuda()
    with torch.no_grad():
        cell.norm.weight.add_(0.1 * torch.randn_like(cell.norm.weight))
    x = torch.randn(bsz, steps, feat, device="cuda", requires_grad=True)
    done = torch.rand(bsz, steps, device="cuda") < 0.05
    carry = None
    if with_carry:
        carry = ((0.3 * torch.randn(bsz, 1, heads, 16, 16, device="cuda")).requires_grad_(), torch.rand(bsz, 1, heads, 1, 1, device="cuda"))
    gy, gl = torch.randn_like(x), torch.randn(bsz, 1, heads, 16, 16, device="cuda")
    wrt = [x, *cell.parameters()] + ([carry[0]] if with_carry else [])
    (h, a), y = Memoroid(cell)(x, done, carry)
    grads = torch.autograd.grad((y, h), wrt, (gy, gl))
    with torch.no_grad():
        (h_n, a_n), y_n = Memoroid(cell)(x, done, carry)

    import copy
    ref = copy.deepcopy(cell).cpu().double()
    xd = x.detach().cpu().double().requires_grad_()
    h_el, decay, projected = ref(xd)
    width = heads * 256
    h0 = carry[0].detach().cpu().double().requires_grad_() if with_carry else torch.zeros(bsz, 1, heads, 16, 16, dtype=torch.float64)
    a0 = carry[1].cpu().double().expand(bsz, 1, heads, 16, 16).reshape(bsz, width) if with_carry else None
    states, a_ref = mo.linrec_seq(decay.expand(bsz, steps, heads, 16, 16).reshape(bsz, steps, width), h_el.reshape(bsz, steps, width),
                                  h0.reshape(bsz, width), done.cpu().double(), a0)
    states = states.reshape(bsz, steps, heads, 16, 16)
    y_ref = ref.read((states, None), xd, projected=projected)
    want = torch.autograd.grad((y_ref, states[:, -1:]), [xd, *ref.parameters()] + ([h0] if with_carry else []),
                               (gy.cpu().double(), gl.cpu().double()))
    err = lambda got, r: float((got.detach().cpu().reshape(r.shape) - r.detach()).abs().max()) / max(0.05, float(r.detach().abs().max()))
    a_ref = a_ref.reshape(bsz, 1, heads, 256)[..., :1, None]
    for got, r in ((h, states[:, -1:]), (h_n, states[:, -1:]), (a, a_ref), (a_n, a_ref), (y, y_ref), (y_n, y_ref)):
        assert err(got, r) <= 1e-5
    for name, got, r in zip(["x", *(n for n, _ in cell.named_parameters()), "h0"], grads, want):
        assert err(got, r) <= 1e-4, (name, err(got, r))


# one, two and four parts of 16 steps, on both sides of each; the last two have more blocks than fit at a time
@pytest.mark.parametrize("shape", [(3, 15, 8, 3), (2, 17, 8, 2), (2, 31, 8, 3), (2, 32, 8, 2), (2, 33, 8, 4), (2, 64, 8, 3), (150, 16, 8, 8), (70, 97, 8, 8)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_parts_of_a_stretch(shape, with_carry):
    test_mamba_layer_and_its_gradients(shape, with_carry)


# rows of the gate in four and in eight registers a lane, cut and whole, and longer ones; several tokens to a warp
@pytest.mark.parametrize("heads", [1, 3, 8, 9, 16, 17])
@pytest.mark.parametrize("bsz", [2, 290])
def test_rows_of_the_gate(heads, bsz):
    test_mamba_layer_and_its_gradients((bsz, 17, 8, heads), False)


# the gate's backward pass keeps 512 bytes of shared memory a head: more of it in a later call than in an earlier one, and
# on both sides of what an SM has
def test_head_counts_one_after_another():
    from memorax_b200.memoroid import MambaCell, Memoroid, MemoroidCellBase
    bsz, steps, feat = 2, 9, 8
    for heads in (97, 100, 200, 454, 455):
        torch.manual_seed(heads)
        cell = MambaCell(feat, num_heads=heads).cuda()
        x, done = torch.randn(bsz, steps, feat, device="cuda", requires_grad=True), torch.rand(bsz, steps, device="cuda") < 0.1
        gy, wrt = torch.randn(bsz, steps, feat, device="cuda"), [x, *cell.parameters()]
        runs = []
        for layer in (Memoroid(cell), lambda *a: MemoroidCellBase.layer(cell, *a)):
            _, y = layer(x, done, None)
            runs.append([y, *torch.autograd.grad(y, wrt, gy)])
        for got, want in zip(*runs):
            assert float((got - want).detach().abs().max()) <= 1e-4 * max(0.05, float(want.detach().abs().max())), heads
