"""The native bf16 mLSTM layer against the same layer composed from its parts (torch products and elementwise calls around
the same chunk kernels), in value and in every gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# the convolution's runs of 4 (and, in the last case, 16) tokens and its three-token halo; channel groups that share a block; head dims 16 / 32 / 64
@pytest.mark.parametrize("bsz,steps,feat,heads,dim", [(3, 1, 64, 2, 32), (2, 16, 96, 4, 16), (2, 35, 64, 1, 64), (1, 130, 128, 4, 64), (500, 67, 64, 8, 64)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_native_mlstm_layer_equals_the_composed_one(bsz, steps, feat, heads, dim, with_carry):
    from memorax_b200.memoroid import Memoroid, MemoroidCellBase, mLSTMCell
    torch.manual_seed(0)
    cell = mLSTMCell(feat, heads * dim, num_heads=heads, tensor_cores=True)
    with torch.no_grad():
        cell.i_gate.weight.normal_(std=0.05)
        cell.f_gate.weight.normal_(std=0.05)
        cell.norm_weight.normal_(std=0.1)
    model = Memoroid(cell).cuda().bfloat16()
    x = torch.randn(bsz, steps, feat, device="cuda").bfloat16().requires_grad_()
    done = torch.rand(bsz, steps, device="cuda") < 0.05
    rn = lambda *s: torch.randn(*s, device="cuda")
    carry = None
    if with_carry:
        carry = ((0.1 * rn(bsz, 1, heads, dim, dim)).requires_grad_(), -rn(bsz, 1, heads, 1, 1).abs(),
                 (0.1 * rn(bsz, 1, heads, dim, 1)).requires_grad_(), (0.1 * rn(bsz, 1, heads, 1, 1)).requires_grad_())
    gy, gc, gn = torch.randn_like(x), rn(bsz, 1, heads, dim, dim), rn(bsz, 1, heads, dim, 1)
    wrt = [x, *model.parameters()] + ([carry[0], carry[2]] if with_carry else [])

    def run(layer):
        (c, f, n, m), y = layer()
        return [y, c, f, n, m, *torch.autograd.grad([y, c, n], wrt, [gy, gc, gn])]

    got, want = run(lambda: model(x, done, carry)), run(lambda: MemoroidCellBase.layer(cell, x, done, carry))
    with torch.no_grad():
        (c, f, n, m), y = model(x, done, carry)
    for g, w in list(zip(got, want)) + list(zip([y, c, f, n, m], want)):
        g, w = g.detach().float(), w.detach().float()
        assert g.shape == w.shape
        assert float((g - w).norm()) <= 2e-2 * max(5e-2 * w.numel() ** 0.5, float(w.norm())), float((g - w).norm() / w.norm())
