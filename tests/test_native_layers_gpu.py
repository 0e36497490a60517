"""Calls that the native layers leave to the composed ones."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


# a parameter of another shape: composed, it raises (or broadcasts), and no kernel reads past its end
@pytest.mark.parametrize("kind", ["linattn key", "deltanet value", "deltanet gate", "mlstm gate bias", "mlstm value", "mamba conv bias", "mamba dt", "lru C"])
@pytest.mark.parametrize("grad", [False, True])
def test_parameters_of_another_shape_are_refused(kind, grad):
    from memorax_b200.memoroid import DeltaNetCell, LinearAttentionCell, LRUCell, MambaCell, Memoroid, mLSTMCell
    torch.manual_seed(0)
    name, dtype = kind.split()[0], torch.float32
    par = lambda *s: nn.Parameter(torch.randn(*s))
    if name == "linattn":
        cell, dtype = LinearAttentionCell(32, 64, 2), torch.bfloat16
        cell.key = nn.Linear(32, 64, bias=False)
    elif name == "deltanet":
        cell, dtype = DeltaNetCell(32, 64, 2), torch.bfloat16
        if kind.endswith("value"):
            cell.value = nn.Linear(32, 64, bias=False)
        else:
            cell.gate.bias = par(2)
    elif name == "mlstm":
        cell, dtype = mLSTMCell(32, 64, num_heads=2, tensor_cores=True), torch.bfloat16
        if kind.endswith("bias"):
            cell.i_gate.bias = par(3)
        else:
            cell.value = par(2, 32, 16)
    elif name == "mamba":
        cell = MambaCell(32, num_heads=2)
        if kind.endswith("bias"):
            cell.conv.bias = par(48)
        else:
            cell.dt_bias = par(3)
    else:
        cell = LRUCell(32, 16)
        cell.C_real = par(32, 8)
    model = Memoroid(cell).cuda().to(dtype)
    x = torch.randn(2, 5, 32, device="cuda", dtype=dtype, requires_grad=grad)
    with torch.set_grad_enabled(grad), pytest.raises(RuntimeError):
        model(x, torch.zeros(2, 5, device="cuda"))


def test_a_skip_weight_for_all_features():
    from memorax_b200.memoroid import LRUCell, Memoroid
    torch.manual_seed(0)
    model = Memoroid(LRUCell(32, 16)).cuda()
    x, done = torch.randn(2, 5, 32, device="cuda"), torch.zeros(2, 5, device="cuda")
    model.cell.D = nn.Parameter(torch.full((32,), 0.7, device="cuda"))
    _, want = model(x, done)
    model.cell.D = nn.Parameter(torch.full((1,), 0.7, device="cuda"))
    _, got = model(x, done)
    assert float((got - want).detach().abs().max()) <= 1e-5 * float(want.detach().abs().max())
