"""float32 products on the tensor cores (three bf16 terms per operand) and the LRU layer built on them."""
import pytest
import torch

from oracle import memoroid_oracle as mo

pytestmark = pytest.mark.gpu


# edges of the 128 x {64,128} and the paired 256 x 256 tiles and of the 32-deep stages, split contractions, accumulators
# drained in between, unaligned rows
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (127, 64, 31), (129, 65, 33), (257, 257, 100), (300, 776, 513), (128, 256, 4000),
                                   (20000, 512, 96), (20001, 520, 300), (20000, 300, 1100)])
def test_linear_f32_and_its_gradients_match_float64(m, n, k):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(m + n + k)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, b, gy = mk(m, k).requires_grad_(), mk(n, k).requires_grad_(), mk(n).requires_grad_(), mk(m, n)
    y = _C.linear_f32(x, w, b)
    gx, gw, gb = torch.autograd.grad(y, (x, w, b), gy)
    xd, wd, gd = x.detach().double(), w.detach().double(), gy.double()
    for got, want in ((y, xd @ wd.t() + b.detach().double()), (gx, gd @ wd), (gw, gd.t() @ xd), (gb, gd.sum(0))):
        assert float((got.detach().double() - want).norm() / want.norm()) <= 2e-6
    ops.check_status()


# T = 1 is the fused acting step; odd sizes leave remainders in every tile
@pytest.mark.parametrize("shape", [(3, 1, 5, 3), (9, 1, 33, 65), (2, 17, 8, 16), (33, 40, 96, 72)])
@pytest.mark.parametrize("with_carry", [False, True])
def test_lru_layer_matches_the_oracle(shape, with_carry):
    from memorax_b200.memoroid import LRUCell, Memoroid
    bsz, steps, feat, hid = shape
    torch.manual_seed(0)
    cell = LRUCell(feat, hid, r_min=0.5, r_max=0.99, max_phase=0.6).cuda()
    x = torch.randn(bsz, steps, feat, device="cuda", requires_grad=True)
    done = torch.rand(bsz, steps, device="cuda") < 0.1
    cplx = lambda *s: torch.view_as_complex(torch.randn(*s, 2, device="cuda"))
    carry = (cplx(bsz, 1, hid).requires_grad_(), cplx(bsz, 1, hid)) if with_carry else None
    gy, gl = torch.randn_like(x), cplx(bsz, 1, hid)
    wrt = [x, *cell.parameters()] + ([carry[0]] if with_carry else [])
    (h, a), y = Memoroid(cell)(x, done, carry)
    grads = torch.autograd.grad((y, h), wrt, (gy, gl))
    with torch.no_grad():
        (h_n, a_n), y_n = Memoroid(cell)(x, done, carry)

    p = {n: v.detach().cpu().double().requires_grad_() for n, v in cell.named_parameters()}
    xd = x.detach().cpu().double().requires_grad_()
    h0 = carry[0].detach().cpu()[:, 0].to(torch.complex128).requires_grad_() if with_carry else None
    lam = torch.exp(torch.complex(-torch.exp(p["nu_log"]), torch.exp(p["theta_log"])))
    b_norm = torch.complex(p["B_real"], p["B_imag"]) * torch.exp(p["gamma_log"])[:, None]
    bu = xd.to(torch.complex128) @ b_norm.t()
    a0 = carry[1].cpu()[:, 0].to(torch.complex128) if with_carry else None
    hs, a_ref = mo.linrec_seq(lam, bu, h0 if with_carry else torch.zeros(bsz, hid, dtype=torch.complex128), done.cpu().double(),
                              *([a0] if with_carry else []))
    y_ref = (hs @ torch.complex(p["C_real"], p["C_imag"]).t()).real + p["D"] * xd
    wrt_ref = [xd, *p.values()] + ([h0] if with_carry else [])
    want = torch.autograd.grad((y_ref, hs[:, -1:]), wrt_ref, (gy.cpu().double(), gl.cpu().to(torch.complex128)))
    err = lambda got, ref: float((got.detach().cpu().reshape(ref.shape) - ref.detach()).abs().max()) / max(1e-30, float(ref.detach().abs().max()))
    for got, ref in ((h[:, 0], hs[:, -1]), (h_n[:, 0], hs[:, -1]), (a[:, 0], a_ref), (a_n[:, 0], a_ref), (y, y_ref), (y_n, y_ref)):
        assert err(got, ref) <= 1e-5
    for got, ref in zip(grads, want):
        assert err(got, ref) <= 1e-4


# stretches of 64 steps, eight pieces of time for the leaves per unit, 8 / 16 / 32 units by 128 / 64 / 32 features; with and without a reset in a sequence
@pytest.mark.parametrize("shape", [(2, 1, 4, 3), (3, 64, 33, 9), (2, 65, 130, 16), (4, 150, 8, 130), (2, 9, 48, 33)])
@pytest.mark.parametrize("p_done", [0.0, 0.03])
def test_fused_rtrl_segment_matches_the_oracle(shape, p_done):
    from memorax_b200.memoroid import LRUCell, Memoroid
    bsz, steps, feat, hid = shape
    torch.manual_seed(0)
    cell = LRUCell(feat, hid, r_min=0.5, r_max=0.999, max_phase=0.6).cuda()
    model = Memoroid(cell)
    x, done = torch.randn(bsz, steps, feat, device="cuda"), torch.rand(bsz, steps, device="cuda") < p_done
    cplx = lambda s: torch.view_as_complex(torch.randn(*s, 2, device="cuda"))
    carry = (cplx((bsz, 1, hid)), torch.ones(bsz, 1, hid, dtype=torch.complex64, device="cuda"))
    sens = {k: cplx(v.shape) for k, v in model.initialize_sensitivity(None, (bsz, feat)).items()}
    with torch.no_grad():
        (h, _), y, out = model.local_jacobian(x, done, carry, sens)
    p = {n: v.detach().cpu().double() for n, v in cell.named_parameters()}
    h_ref, y_ref, s_ref = mo.lru_rtrl_seq(
        x.cpu().double(), done.cpu().double(), carry[0][:, 0].cpu().to(torch.complex128), p["nu_log"], p["theta_log"], p["gamma_log"],
        torch.complex(p["B_real"], p["B_imag"]), torch.complex(p["C_real"], p["C_imag"]), p["D"],
        {k: v.cpu().to(torch.complex128) for k, v in sens.items()})
    err = lambda got, ref: float((got.cpu().reshape(ref.shape) - ref).abs().max()) / float(ref.abs().max())
    assert err(h, h_ref) <= 1e-5 and err(y, y_ref) <= 1e-5
    for name in s_ref:
        assert err(out[name], s_ref[name]) <= 1e-5, name


# sensitivities cut out of a flat buffer start at any complex number; the wide accesses are for 16-byte boundaries
@pytest.mark.parametrize("feat", [8, 6])
def test_fused_rtrl_segment_from_sensitivities_at_any_address(feat):
    from memorax_b200.memoroid import LRUCell, Memoroid
    torch.manual_seed(4)
    bsz, steps, hidden = 3, 20, 40
    model = Memoroid(LRUCell(feat, hidden).cuda())
    c64 = lambda *s: torch.view_as_complex(torch.randn(*s, 2, device="cuda"))
    x, done = torch.randn(bsz, steps, feat, device="cuda"), torch.rand(bsz, steps, device="cuda") < 0.1
    carry = (c64(bsz, 1, hidden), torch.ones(bsz, 1, hidden, dtype=torch.complex64, device="cuda"))
    sens = {k: c64(*v.shape) for k, v in model.initialize_sensitivity(None, (bsz, feat)).items()}
    cut = {k: torch.zeros(v.numel() + 1, dtype=torch.complex64, device="cuda")[1:].view_as(v).copy_(v) for k, v in sens.items()}
    with torch.no_grad():
        *_, want = model.local_jacobian(x, done, carry, sens)
        *_, got = model.local_jacobian(x, done, carry, cut)
    for k in want:
        assert torch.equal(got[k], want[k]), k


# the largest floats lie beyond bf16's largest number, and masks are made of them
@pytest.mark.parametrize("m,n,k", [(3, 5, 32), (130, 70, 100), (300, 256, 512)])
def test_products_of_the_largest_floats(m, n, k):
    from memorax_b200 import _C
    torch.manual_seed(0)
    x, w = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda") / k
    x[0, :3], x[-1, k // 2] = torch.finfo(torch.float32).min, torch.finfo(torch.float32).max
    got, want = _C.linear_f32(x, w), x.double() @ w.double().t()
    assert float(((got - want).abs() / want.abs().amax(1, keepdim=True)).max()) <= 1e-6
    x[1, 0] = float("inf")
    got = _C.linear_f32(x, w)
    assert not got.isnan().any() and bool((got[1].sign() == w[:, 0].sign()).all()) and float(got[1].abs().min()) > 1e30


# an episode that has gone wrong ends at its reset
@pytest.mark.parametrize("feat", [8, 6])
def test_fused_rtrl_segment_forgets_at_a_reset(feat):
    from memorax_b200.memoroid import LRUCell, Memoroid
    torch.manual_seed(5)
    bsz, steps, hidden = 2, 20, 40
    model = Memoroid(LRUCell(feat, hidden).cuda())
    x, done = torch.randn(bsz, steps, feat, device="cuda"), torch.zeros(bsz, steps, device="cuda")
    done[:, 7] = 1
    x[:, 3] = float("nan")
    bad = lambda *s: torch.full(s, float("nan"), dtype=torch.complex64, device="cuda")
    sens = {k: bad(*v.shape) for k, v in model.initialize_sensitivity(None, (bsz, feat)).items()}
    ones = torch.ones(bsz, 1, hidden, dtype=torch.complex64, device="cuda")
    with torch.no_grad():
        (h, _), _, got = model.local_jacobian(x, done, (bad(bsz, 1, hidden), ones), sens)
        zero = {k: torch.zeros_like(v) for k, v in sens.items()}
        (h2, _), _, want = model.local_jacobian(x[:, 7:], done[:, 7:], (torch.zeros_like(ones), ones), zero)
    for k in want:
        assert float((got[k] - want[k]).abs().max()) <= 1e-5 * float(want[k].abs().max()), k
