"""The gated pre-norm block's joint backward passes (norm with its input's two other readers, bias gradients added up as the
cotangents are written) against the same block taken apart, which a hook on its parts forces, at the smallest widths, widths
past a warp's vectors, and row counts around a block's share."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features", [8, 264, 1024])
@pytest.mark.parametrize("rows", [(1, 1), (1, 7), (3, 111), (2, 2500)])
def test_joint_passes_equal_the_parts(features, rows):
    from memorax_b200 import blocks
    torch.manual_seed(features + rows[1])
    joint = blocks.GatedResidual(blocks.PreNorm(blocks.FFN(features), features), features).cuda()
    with torch.no_grad():
        for p in joint.parameters():
            p.add_(0.1 * torch.randn_like(p))
    joint = joint.to(torch.bfloat16)
    parts = copy.deepcopy(joint)
    for m in (parts.module, parts.gate, parts.module.module.up):
        m.register_forward_hook(lambda *a: None)
    x = torch.randn(*rows, features, device="cuda").bfloat16()
    w = torch.randn(*rows, features, device="cuda").bfloat16()
    got = []
    for model in (joint, parts):
        leaf = x.clone().requires_grad_()
        _, y = model(leaf * 1)
        names = ["x"] + [n for n, _ in model.named_parameters()]
        got.append([y, *torch.autograd.grad(y, [leaf, *model.parameters()], w)])
    assert torch.equal(got[0][0], got[1][0])
    for name, a, b in zip(names, got[0][1:], got[1][1:]):
        scale = float(b.float().abs().max())
        assert float((a.float() - b.float()).abs().max()) <= 1.5e-2 * scale + 1e-6, name


def test_products_of_another_type_under_autocast():
    """Autocast gives a Dense layer's product its own type: the fused passes, which read bf16, leave it to the general ones."""
    from memorax_b200 import ops
    from memorax_b200.blocks import Dense
    torch.manual_seed(0)
    layer = Dense(32, 64).cuda().bfloat16()
    x, o = torch.randn(5, 32, device="cuda").bfloat16(), torch.randn(5, 64, device="cuda").bfloat16()
    with torch.autocast("cuda", dtype=torch.float16):
        up, gated = ops.dense_gelu(x, layer), ops.gated_dense(o, x, layer, o)
    a = x.double() @ layer.weight.double().t() + layer.bias.double()
    near = lambda got, want: float((got.double() - want).detach().abs().max()) <= 2e-2 * float(want.detach().abs().max())
    assert near(up, torch.nn.functional.gelu(a, approximate="tanh")) and near(gated, o.double() * (1 + torch.sigmoid(a)))
