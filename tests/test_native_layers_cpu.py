"""When a layer goes to its native call, and when it has to be composed from its parts: anything that PyTorch lets a user
hang onto a module (hooks, weight norm, pruning, parametrisations, another forward) must keep its effect."""
import copy

import pytest
import torch
from torch import nn
from torch.nn.utils import parametrize, prune, weight_norm


@pytest.fixture(scope="module")
def memoroid():
    from memorax_b200.build import build_library
    build_library()
    from memorax_b200 import memoroid
    return memoroid


# cell, a Dense layer in it (None: it has parameters of its own only)
CELLS = {"lru": (lambda m: m.LRUCell(8, 16), None), "mingru": (lambda m: m.MinGRUCell(8), "h"),
         "linattn": (lambda m: m.LinearAttentionCell(8, 64, 1), "key"), "deltanet": (lambda m: m.DeltaNetCell(8, 64, 1), "gate"),
         "mlstm": (lambda m: m.mLSTMCell(8, 64, num_heads=2, tensor_cores=True), "up_projection"),
         "mamba": (lambda m: m.MambaCell(8, num_heads=2), "input_projection")}
NATIVE = ("lru_layer", "mingru_layer", "linattn_layer", "deltanet_layer", "mlstm_layer", "mamba_layer", "lru_rtrl")


class Adapter(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


def _replace(cell, name, kind, **kw):
    old = getattr(cell, name)
    setattr(cell, name, kind(old.in_features, old.out_features, **{"bias": old.bias is not None, **kw}))


def _own_forward(module):
    module.forward = type(module).forward.__get__(module)


CHANGES = {
    "weight_norm": lambda cell, name: weight_norm(getattr(cell, name)),
    "pruned": lambda cell, name: prune.l1_unstructured(getattr(cell, name), "weight", 0.5),
    "parametrised": lambda cell, name: parametrize.register_parametrization(getattr(cell, name), "weight", nn.Identity()),
    "adapter": lambda cell, name: _replace(cell, name, Adapter),
    "forward of its own": lambda cell, name: _own_forward(getattr(cell, name)),
    "forward hook": lambda cell, name: getattr(cell, name).register_forward_hook(lambda *a: None),
    "forward pre-hook": lambda cell, name: getattr(cell, name).register_forward_pre_hook(lambda *a: None),
    "backward hook": lambda cell, name: getattr(cell, name).register_full_backward_hook(lambda *a: None),
    "backward pre-hook": lambda cell, name: getattr(cell, name).register_full_backward_pre_hook(lambda *a: None),
}


def _calls(monkeypatch, memoroid, cell):
    """Names of the native calls one forward pass of the layer makes (each answers that it has no such form)."""
    called = []

    class Recorder:
        def __getattr__(self, name):
            return lambda *a, **kw: called.append(name)
    assert all(hasattr(memoroid._C, name) for name in NATIVE)
    with monkeypatch.context() as m:
        m.setattr(memoroid, "_C", Recorder())
        m.setattr(memoroid.MemoroidCellBase, "layer", lambda *a, **kw: (None, None))
        memoroid.Memoroid(cell)(torch.zeros(2, 3, 8), torch.zeros(2, 3))
    return called


@pytest.mark.parametrize("kind", CELLS)
def test_a_plain_cell_goes_to_its_native_layer(monkeypatch, memoroid, kind):
    assert _calls(monkeypatch, memoroid, CELLS[kind][0](memoroid)) == [f"{kind}_layer"]
    assert _calls(monkeypatch, memoroid, copy.deepcopy(CELLS[kind][0](memoroid))) == [f"{kind}_layer"]


@pytest.mark.parametrize("change", CHANGES)
@pytest.mark.parametrize("kind", [k for k in CELLS if CELLS[k][1]])
def test_a_changed_submodule_is_composed(monkeypatch, memoroid, kind, change):
    make, name = CELLS[kind]
    cell = make(memoroid)
    CHANGES[change](cell, name)
    assert _calls(monkeypatch, memoroid, cell) == []


@pytest.mark.parametrize("kind", CELLS)
@pytest.mark.parametrize("change", [k for k in CHANGES if "hook" in k or "own" in k])
def test_a_changed_cell_is_composed(monkeypatch, memoroid, kind, change):
    cell = CELLS[kind][0](memoroid)
    holder = nn.Module()
    holder.cell = cell
    CHANGES[change](holder, "cell")
    assert _calls(monkeypatch, memoroid, cell) == []


@pytest.mark.parametrize("kind", CELLS)
def test_hooks_on_every_module_are_seen(monkeypatch, memoroid, kind):
    handle = nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert _calls(monkeypatch, memoroid, CELLS[kind][0](memoroid)) == []
    finally:
        handle.remove()
    assert _calls(monkeypatch, memoroid, CELLS[kind][0](memoroid)) == [f"{kind}_layer"]


@pytest.mark.parametrize("change", ["bias", "eps", "dilation", "missing parameter"])
def test_other_settings_than_the_cells_own(monkeypatch, memoroid, change):
    if change == "bias":
        cell = memoroid.LinearAttentionCell(8, 64, 1)
        _replace(cell, "query", nn.Linear, bias=True)
    elif change == "eps":
        cell = memoroid.DeltaNetCell(8, 64, 1)
        cell.norm.eps = None
    elif change == "dilation":
        cell = memoroid.MambaCell(8, num_heads=2)
        cell.conv.dilation, cell.conv.padding = (2,), (6,)
    else:   # the replicas of nn.DataParallel hold their parameters as plain attributes
        cell = memoroid.LRUCell(8, 16)
        weight = cell._parameters.pop("B_real")
        cell.__dict__["B_real"] = weight.detach()
    assert _calls(monkeypatch, memoroid, cell) == []


def test_the_fused_rtrl_segment_sees_the_cells_hooks(monkeypatch, memoroid):
    cell = memoroid.LRUCell(8, 16)
    sens = cell.initialize_sensitivity(None, (2, 8))
    carry = cell.initialize_carry(None, (2, 8))
    called = []
    monkeypatch.setattr(memoroid, "_C", type("Recorder", (), {"lru_rtrl": staticmethod(lambda *a: called.append("lru_rtrl"))}))
    x, done = torch.zeros(2, 3, 8), torch.zeros(2, 3)
    assert cell.jacobian_segment(x, done, carry, sens) is None and called == ["lru_rtrl"]
    cell.register_forward_hook(lambda *a: None)
    assert cell.jacobian_segment(x, done, carry, sens) is None and called == ["lru_rtrl"]


def test_the_composed_layers_norm_is_called_where_it_was_changed(memoroid):
    norm, x = nn.RMSNorm(8), torch.randn(3, 8)
    norm.register_forward_hook(lambda module, args, out: out + 1)
    assert torch.equal(memoroid._normed(norm, x), nn.functional.rms_norm(x, (8,), norm.weight, None) + 1)
