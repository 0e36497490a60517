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


CELLS = {"lru": lambda m: m.LRUCell(32, 16), "s5": lambda m: m.S5Cell(32, 16), "mingru": lambda m: m.MinGRUCell(32), "mamba": lambda m: m.MambaCell(32, num_heads=2),
         "linattn": lambda m: m.LinearAttentionCell(32, 64, 2).bfloat16(), "deltanet": lambda m: m.DeltaNetCell(32, 64, 2).bfloat16(),
         "mlstm": lambda m: m.mLSTMCell(32, 64, num_heads=2, tensor_cores=True).bfloat16()}


# the kernels have neither tangents nor a graph form: both are refused, not dropped
@pytest.mark.parametrize("kind", CELLS)
@pytest.mark.parametrize("what", ["inputs", "carry", "parameter"])
def test_forward_mode_is_refused(kind, what):
    import torch.autograd.forward_ad as fwd
    from memorax_b200 import memoroid
    torch.manual_seed(0)
    model = memoroid.Memoroid(CELLS[kind](memoroid)).cuda().requires_grad_(False)
    x, done = torch.randn(2, 5, 32, device="cuda", dtype=torch.float32 if kind in ("lru", "s5", "mingru", "mamba") else torch.bfloat16), torch.zeros(2, 5, device="cuda")
    carry = [c.cuda() for c in model.initialize_carry(None, (2, 32))]
    with fwd.dual_level():
        dual = lambda t: fwd.make_dual(t, torch.ones_like(t))
        if what == "inputs":
            x = dual(x)
        elif what == "carry":
            carry[0] = dual(carry[0])
        else:   # the cell's own parameter, or a Dense layer's
            holder = model.cell if model.cell._parameters else next(m for m in model.cell.children() if isinstance(m, nn.Linear))
            name = next(iter(holder._parameters))
            holder._parameters[name] = dual(holder._parameters[name])
        with pytest.raises(NotImplementedError):
            model(x, done, tuple(carry))


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("kind", CELLS)
def test_a_trace_is_refused_or_follows_its_inputs(kind):
    from memorax_b200 import memoroid
    torch.manual_seed(0)
    model = memoroid.Memoroid(CELLS[kind](memoroid)).cuda().requires_grad_(False)
    dtype = torch.float32 if kind in ("lru", "s5", "mingru", "mamba") else torch.bfloat16
    x, other = (torch.randn(2, 5, 32, device="cuda", dtype=dtype) for _ in range(2))
    done = torch.zeros(2, 5, device="cuda")
    try:
        traced = torch.jit.trace(lambda x, done: model(x, done)[1], (x, done), check_trace=False)
    except RuntimeError:
        return
    want = model(other, done)[1].float()
    assert float((traced(other, done).float() - want).norm()) <= 1e-5 * float(want.norm())


# products in TF32 are the library's, whichever of torch's two settings asked for them
@pytest.mark.parametrize("setting", ["older", "newer"])
@pytest.mark.parametrize("kind", ["lru", "s5", "mingru", "mamba"])
def test_tf32_products_are_composed(kind, setting):
    from memorax_b200 import memoroid
    torch.manual_seed(0)
    model = memoroid.Memoroid(CELLS[kind](memoroid)).cuda().requires_grad_(False)
    x, done = torch.randn(2, 5, 32, device="cuda"), torch.zeros(2, 5, device="cuda")
    exact = model(x, done)[1]
    matmul = torch.backends.cuda.matmul
    name, value = ("allow_tf32", True) if setting == "older" else ("fp32_precision", "tf32")
    before = getattr(matmul, name)
    try:
        setattr(matmul, name, value)
        got, want = model(x, done)[1], memoroid.MemoroidCellBase.layer(model.cell, x, done, None)[1]
    finally:
        setattr(matmul, name, before)
    assert torch.equal(got, want) and not torch.equal(got, exact)


# conj() only sets a bit: the memory that a kernel would read is the unconjugated tensor's
@pytest.mark.parametrize("kind", ["lru", "s5"])
def test_conjugated_views_are_what_they_show(kind):
    from memorax_b200 import memoroid, ops
    torch.manual_seed(0)
    model = memoroid.Memoroid(CELLS[kind](memoroid)).cuda()
    x, done = torch.randn(2, 5, 32, device="cuda"), torch.zeros(2, 5, device="cuda")
    c64 = lambda: torch.view_as_complex(torch.randn(2, 1, 16, 2, device="cuda")).conj()
    state, one, cotangent = c64(), torch.ones(2, 1, 16, dtype=torch.complex64, device="cuda"), c64()
    params = list(model.parameters())
    runs = []
    for view in (lambda t: t, lambda t: t.resolve_conj()):
        (h, _), y = model(x, done, (view(state), one))
        runs.append([h, y, *torch.autograd.grad(h, params, view(cotangent), allow_unused=True)])
    for got, want in zip(*runs):
        assert (got is None and want is None) or torch.equal(got, want)
    a, b = state[0, 0], c64().expand(2, 3, 16).resolve_conj().conj()
    assert torch.equal(ops.linrec_fwd(a, b)[0], ops.linrec_fwd(a.resolve_conj(), b.resolve_conj())[0])


# nothing that a layer returns to be read is needed by its backward pass: it may be changed in place
@pytest.mark.parametrize("kind", CELLS)
def test_the_read_out_may_be_changed_in_place(kind):
    from memorax_b200 import memoroid
    torch.manual_seed(0)
    model = memoroid.Memoroid(CELLS[kind](memoroid)).cuda()
    dtype = next(model.parameters()).dtype
    x, done = torch.randn(2, 5, 32, device="cuda").to(dtype).requires_grad_(), torch.zeros(2, 5, device="cuda")
    wrt = [x, *model.parameters()]
    _, y = model(x, done)
    want = torch.autograd.grad(2 * y, wrt, torch.ones_like(y))
    _, y = model(x, done)
    got = torch.autograd.grad(y.mul_(2), wrt, torch.ones_like(y))
    for g, w in zip(got, want):
        assert torch.equal(g, w)
