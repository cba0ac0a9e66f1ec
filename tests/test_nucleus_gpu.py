"""The nucleus search of the sampler around the sizes where it changes hands: fewer and more open entries than one warp's list
holds, rows of one entry and of equal entries, limits next to 0 and 1, with and without top-k.  Against the draw in fp64.
Rows without mass (NaN, infinities) and tails that are far below the rounding of the row's sum: the search ends on them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [256, 1024, 1280, 16384])
@pytest.mark.parametrize("top_p,top_k", [(1e-6, 0), (0.5, 0), (0.95, 0), (0.95, 40), (0.9995, 0), (0.9999999, 0)])
def test_nucleus_draw(V, top_p, top_k):
    from tests.test_kernels_gpu import _sample
    g = torch.Generator(device="cuda").manual_seed(V)
    T, (a, b, c) = 0.8, (23.0, 5.0, 7.5)
    x = torch.randn(6, V, device="cuda", generator=g) * torch.tensor([0.01, 0.3, 3.0, 8.0, 0.0, 0.2], device="cuda")[:, None]
    x[5] -= 12
    x[5, V // 3] = 40.0                                     # a sharp row
    x = x.repeat_interleave(8, 0).bfloat16()
    u = torch.rand(len(x), device="cuda", generator=g)
    tok, logp = (torch.from_numpy(v).cuda() for v in _sample(x, u=u, T=T, top_k=top_k, top_p=top_p))
    z = a * torch.sigmoid((x.double() + b) / c) / T
    e = torch.exp(z - z.max(1, keepdim=True).values)
    assert torch.allclose(logp.double(), torch.log_softmax(z, 1).gather(1, tok[:, None])[:, 0], atol=2e-3, rtol=1e-4)
    if top_k:
        e = e * (e >= e.topk(top_k, 1).values[:, -1:])
    s, order = e.sort(1, descending=True)
    S = e.sum(1, keepdim=True)
    before = s.cumsum(1) - s
    cut = torch.where(before < top_p * S, s, torch.inf).min(1, keepdim=True).values
    kept = e * (e >= cut * (1 - 1e-5))
    assert (kept.gather(1, tok[:, None]) > 0).all() or top_p > 0.999
    cdf, edge = kept.cumsum(1), 1e-5 * S[:, 0] + 2 * cut[:, 0] * (1 if top_p < 0.999 else 20)
    target = (1 - u.double()) * kept.sum(1)
    at = cdf.gather(1, tok[:, None])[:, 0]
    assert (at >= target - edge).all() and (at - e.gather(1, tok[:, None])[:, 0] <= target + edge).all()


@pytest.mark.parametrize("V", [256, 16384])
@pytest.mark.parametrize("top_p,top_k", [(1e-38, 0), (0.5, 0), (0.95, 40), (0.9999999, 0)])
@pytest.mark.parametrize("precapped", [False, True])
def test_rows_without_mass(V, top_p, top_k, precapped):
    from tests.test_kernels_gpu import _sample
    g = torch.Generator(device="cuda").manual_seed(V)
    good = torch.randn(4, V, device="cuda", generator=g) * 3
    bad = good[:1].repeat(6, 1)
    bad[0], bad[1] = torch.nan, -torch.inf
    bad[2, V // 2] = torch.inf
    bad[3, ::3] = torch.nan
    bad[4, 1:] = -torch.inf
    bad[5] = torch.inf
    x = torch.cat([good, bad, good])
    u = torch.rand(len(x), device="cuda", generator=g)
    draw = lambda a, b: _sample(x[a:b].contiguous(), u=u[a:b].contiguous(), T=0.8, top_k=top_k, top_p=top_p, precapped=precapped)
    tok, logp = draw(0, len(x))
    assert (tok >= 0).all() and (tok < V).all()
    assert tok[7] % 3 != 0                                  # an entry that is a number, where there are some
    if precapped:
        assert tok[8] == 0                                  # the one entry with mass
    for a in (0, 10):                                       # the rows beside them
        t, p = draw(a, a + 4)
        assert (t == tok[a:a + 4]).all() and (p == logp[a:a + 4]).all()
    if top_p == 1e-38:
        assert (tok[:4] == good.argmax(1).cpu().numpy()).all()


def test_tail_below_the_rounding_of_the_sum():
    from tests.test_kernels_gpu import _sample
    V, n = 16384, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    x = -20.7 - 0.3 * torch.rand(n, V, device="cuda", generator=g)
    x[:, 77] = 0.0
    u = torch.rand(n, device="cuda", generator=g)
    u[::2] = 1e-6 * u[::2]
    tok, _ = _sample(x, u=u, T=1.0, top_p=0.9999999, precapped=True)
    e = x.double().exp()
    cdf, tok = e.cumsum(1), torch.from_numpy(tok).cuda()
    at, target = cdf.gather(1, tok[:, None])[:, 0], (1 - u.double()) * e.sum(1)
    # off by the share left out (1.2e-7) and the rounding of fp32 sums near 1 (256 chunk sums: 256 * 6e-8)
    assert (at >= target - 2e-5).all() and (at - e.gather(1, tok[:, None])[:, 0] <= target + 2e-5).all()
