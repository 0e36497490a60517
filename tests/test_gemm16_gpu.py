"""bf16 products on the tensor cores against float64: tile edges, both contraction indices of either operand, batches in
strided views, split contractions, bias and accumulation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (127, 65, 64), (129, 136, 72), (260, 16, 200), (16, 768, 1000), (3000, 256, 96), (512, 256, 6000)])
@pytest.mark.parametrize("a_t", [False, True])
@pytest.mark.parametrize("b_t", [False, True])
def test_product_matches_float64(m, n, k, a_t, b_t):
    from memorax_b200 import _C, ops
    pad = lambda v: -(-v // 8) * 8
    g = torch.Generator("cuda").manual_seed(m + n + k)
    mk = lambda r, c: torch.randn(r, pad(c), generator=g, device="cuda").bfloat16()[:, :c]
    a, b = (mk(k, m).t() if a_t else mk(m, k)), (mk(n, k).t() if b_t else mk(k, n))
    bias, c0 = mk(1, n)[0].contiguous(), mk(m, n).contiguous()
    ref = a.double() @ b.double()
    for got, want in ((_C.product_bf16(a, b), ref), (_C.product_bf16(a, b, bias), ref + bias.double()),
                      (_C.product_bf16(a, b, None, c0.clone()), ref + c0.double())):
        assert float((got.double() - want).norm() / want.norm()) <= 4e-3
    ops.check_status()


@pytest.mark.parametrize("tokens,heads,dim", [(5, 1, 16), (200, 4, 64), (130, 2, 32)])
def test_batched_product_on_strided_heads(tokens, heads, dim):
    from memorax_b200 import _C
    g = torch.Generator("cuda").manual_seed(1)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    u, w, out = mk(tokens, heads, dim).permute(1, 0, 2), mk(heads, 2 * dim, dim), mk(tokens, heads, 3 * dim)
    part = out[..., : 2 * dim].permute(1, 0, 2)
    want = u.double() @ w.double().transpose(1, 2) + part.double()
    rest = out[..., 2 * dim:].clone()
    _C.product_bf16(u, w.transpose(1, 2), None, part)
    assert float((part.double() - want).norm() / want.norm()) <= 4e-3 and torch.equal(out[..., 2 * dim:], rest)
    gw = _C.product_bf16(part.transpose(1, 2), u)
    want = part.double().transpose(1, 2) @ u.double()
    assert float((gw.double() - want).norm() / want.norm()) <= 4e-3


# sums into rows on 32, 16 and 2 bytes, and the sum of few and of many splits into them, four elements at a time and one
@pytest.mark.parametrize("n,ld,at", [(96, 96, 0), (96, 104, 8), (96, 99, 1), (100, 104, 4), (41, 41, 0)])
@pytest.mark.parametrize("k", [40, 640, 6000])
def test_sums_into_rows_at_any_address(n, ld, at, k):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(n + k)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    a, b, held = mk(130, k), mk(k, -(-n // 8) * 8)[:, :n], mk(130 * ld + at)
    c, before = held[at:].view(130, ld)[:, :n], held.clone()
    want = a.double() @ b.double() + c.double()
    _C.product_bf16(a, b, None, c)
    assert float((c.double() - want).norm() / want.norm()) <= 4e-3
    rest = torch.ones_like(held, dtype=torch.bool)
    rest[at:].view(130, ld)[:, :n] = False
    assert torch.equal(held[rest], before[rest])
    ops.check_status()


# sums into whole tiles, whose rows are fetched ahead, beside cut ones; rows on 32 and on 16 bytes, in batches
@pytest.mark.parametrize("m", [1, 127, 300])
@pytest.mark.parametrize("n", [56, 64, 128, 200, 320])
@pytest.mark.parametrize("k", [8, 72])
@pytest.mark.parametrize("pad", [0, 8])
def test_sums_into_whole_tiles(m, n, k, pad):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(m + n + k)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    a, b, held = mk(2, m, k), mk(2, k, n), mk(2, m + 3, n + pad)
    c, before = held[:, :m, :n], held.clone()
    want = a.double() @ b.double() + c.double()
    _C.product_bf16(a, b, None, c)
    # one rounding to bf16 of a float32 sum
    assert float(((c.double() - want).abs() / (want.abs() + 1e-3)).max()) <= 2.0 ** -8 + 1e-4
    held[:, :m, :n] = before[:, :m, :n]
    assert torch.equal(held, before)
    ops.check_status()


# several products in one launch: of one size and of very different ones, batched and not, split and whole; in launches of their own (the
# last size, where they are no gradients)
@pytest.mark.parametrize("tokens", [5, 700, 6000, 20000])
@pytest.mark.parametrize("by_rows", [False, True])
def test_products_that_share_a_launch(tokens, by_rows):
    from memorax_b200 import _C, ops
    g = torch.Generator("cuda").manual_seed(tokens)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    if by_rows:   # gradients of weights: both contracted over their rows
        a, b = [mk(tokens, 264).t(), mk(3, tokens, 72).transpose(1, 2), mk(tokens, 8).t(), mk(tokens, 128).t()], [mk(tokens, 136), mk(3, tokens, 40), mk(tokens, 768), mk(tokens, 64)]
    else:
        a, b = [mk(4, tokens, 64), mk(4, tokens, 64), mk(tokens, 520)], [mk(4, 128, 64).transpose(1, 2), mk(4, 64, 64).transpose(1, 2), mk(96, 520).t()]
    c = [torch.empty(*x.shape[:-1], y.shape[-1], device="cuda", dtype=torch.bfloat16) for x, y in zip(a, b)]
    _C.products_bf16(a, b, c)
    for x, y, got in zip(a, b, c):
        want = x.double() @ y.double()
        assert float((got.double() - want).norm() / want.norm()) <= 4e-3
    ops.check_status()
