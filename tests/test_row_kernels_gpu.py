"""The row kernels that launches of many rows take (a warp a row) against the ones that launches of few rows take, on the
same rows handed over in one call and in pieces: around the row count where the choice changes, on the last rows of a
block, on every head width, with and without gates, value embedding, rotation and cache append."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pieces(n, cut):
    return [(a, min(a + cut, n)) for a in range(0, n, cut)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,d,f", [(768, 640, 1664), (769, 64, 128), (1003, 1032, 4096),
                                   (800, 320, 8), (771, 2056, 1800)])
def test_swiglu_of_many_rows(dtype, n, d, f):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels._util import DTYPE_CODE, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(n)
    gu = torch.randn(n, 2 * f, device="cuda", generator=g).to(dtype) * 4
    h = (torch.randn(n, d, device="cuda", generator=g) * 3).to(dtype)
    got, want = (torch.zeros(n, f, device="cuda", dtype=dtype) for _ in range(2))
    for out, cut in ((got, n), (want, 256)):
        for a, b in _pieces(n, cut):
            _lib.check(_lib.lib().uv_swiglu_rs(gu[a:b].data_ptr(), h[a:b].data_ptr(), DTYPE_CODE[dtype], d, f,
                                               out[a:b].data_ptr(), b - a, stream_ptr(gu.device)), "uv_swiglu_rs")
    rs = torch.rsqrt(h.float().pow(2).mean(1, keepdim=True) + 2.0 ** -23)
    x = gu.float() * rs
    ref = torch.nn.functional.silu(x[:, :f]) * x[:, f:]
    tol = 2e-2 if dtype == torch.bfloat16 else 3e-3
    assert torch.allclose(got.float(), ref, rtol=tol, atol=tol * ref.abs().max().item() * 1e-2)
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_swiglu_of_every_value(dtype):
    """silu of all 65,536 bit patterns: the quotient that many rows take rounds as the one that few rows take."""
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels._util import DTYPE_CODE, stream_ptr
    n, d, f = 1024, 64, 1024
    g = torch.arange(n * f, device="cuda").remainder(1 << 16).to(torch.int16).view(dtype).view(n, f)
    gu, h = torch.cat([g, torch.ones_like(g)], 1), torch.ones(n, d, device="cuda", dtype=dtype)
    out = [torch.zeros(n, f, device="cuda", dtype=dtype) for _ in range(2)]
    for o, cut in zip(out, (n, 256)):
        for a, b in _pieces(n, cut):
            _lib.check(_lib.lib().uv_swiglu_rs(gu[a:b].data_ptr(), h[a:b].data_ptr(), DTYPE_CODE[dtype], d, f,
                                               o[a:b].data_ptr(), b - a, stream_ptr(gu.device)), "uv_swiglu_rs")
    assert torch.equal(out[0].view(torch.int16), out[1].view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,H,K,hd,d,pairs,gate,ve,ring", [
    (768, 8, 1, 64, 640, 16, 128, 12, True), (1001, 8, 1, 64, 640, 0, 128, 0, False), (770, 4, 2, 64, 64, 16, 16, 4, True),
    (800, 3, 1, 128, 1040, 32, 0, 5, False), (900, 6, 2, 32, 192, 8, 24, 12, True),
    (800, 3, 1, 128, 1000, 64, 0, 128, False), (777, 5, 1, 16, 96, 8, 18, 3, True), (780, 11, 3, 64, 1024, 32, 100, 37, True),
    (769, 9, 1, 128, 520, 32, 127, 0, True), (768, 1, 1, 32, 8, 16, 8, 1, False),
    (768, 192, 12, 16, 64, 8, 16, 4, True)])     # (more gate weights than shared memory takes)
def test_qkv_post_of_many_rows(dtype, n, H, K, hd, d, pairs, gate, ve, ring):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels._util import DTYPE_CODE, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    S, rows, vocab = 40, 64, 50
    x, qkv0 = (rnd(n, d) * 2).to(dtype), rnd(n, (H + 2 * K) * hd).to(dtype)
    tok = torch.randint(-2, vocab + 2, (n,), device="cuda", generator=g)
    perm = torch.randperm(rows * (30 if ring else S), device="cuda", generator=g)[:n]     # no two entries share a slot
    row, pos = perm % rows, perm // rows
    pos = pos + (S * 3 if ring else 0)
    if not ring:
        pos[5] = S + 2                                                                    # past the cache: counted
    last = torch.where(torch.rand(n, device="cuda", generator=g) < 0.1, pos + S, pos)     # overwritten within the launch
    gw, vw, emb = rnd(H, max(gate, 1)).to(dtype), rnd(K, max(ve, 1)).to(dtype), rnd(vocab, K * hd).to(dtype)
    inv = torch.rand(max(pairs, 1), device="cuda", generator=g)
    cs = torch.cat([torch.cos(pos[:, None] * inv), torch.sin(pos[:, None] * inv)], 1).to(dtype).float().contiguous()
    res = []
    for cut in (n, 250):
        qkv = qkv0.clone()
        gates = torch.zeros(n, H, device="cuda")
        kc, vc = (torch.zeros(rows, K, S, hd, dtype=torch.int8, device="cuda") for _ in range(2))
        ks, vs = (torch.zeros(rows, K, S, dtype=torch.float16, device="cuda") for _ in range(2))
        oob = torch.zeros(1, dtype=torch.int32, device="cuda")
        for a, b in _pieces(n, cut):
            q = _lib.QkvArgs()
            q.qkv, q.xn, q.tok, q.pos = (t[a:b].data_ptr() for t in (qkv, x, tok, pos))
            q.row_map, q.last_pos = row[a:b].data_ptr(), last[a:b].data_ptr()
            q.k_cache, q.v_cache, q.k_scale, q.v_scale = kc.data_ptr(), vc.data_ptr(), ks.data_ptr(), vs.data_ptr()
            q.oob_count, q.dtype, q.vocab, q.xn_raw, q.ring = oob.data_ptr(), DTYPE_CODE[dtype], vocab, 1, int(ring)
            q.B, q.H, q.K, q.hd, q.d, q.S, q.S_alloc, q.n_pairs = b - a, H, K, hd, d, S, S, pairs
            if pairs:
                q.inv_freq, q.rope_cs = inv.data_ptr(), cs[a:b].data_ptr()
            if ve:
                q.ve_gate, q.value_embed, q.ve_ch = vw.data_ptr(), emb.data_ptr(), ve
            if gate:
                q.gate_w, q.gate_out, q.gate_ch = gw.data_ptr(), gates[a:b].data_ptr(), gate
            _lib.check(_lib.lib().uv_qkv_post_args(C.byref(q), stream_ptr(x.device)), "uv_qkv_post")
        res.append((qkv, gates, kc, vc, ks, vs, oob))
    (q1, g1, *c1, o1), (q2, g2, *c2, o2) = res
    assert int(o1) == int(o2) == (0 if ring else 2 * K)
    for a, b in zip((q1, g1, *c1), (q2, g2, *c2)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_qkv_post_takes_its_table_at_any_float(offset):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels._util import stream_ptr
    n, H, K, hd, d, pairs = 770, 2, 1, 64, 64, 16
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, qkv0, pos = rnd(n, d).bfloat16(), rnd(n, (H + 2 * K) * hd).bfloat16(), torch.arange(n, device="cuda")
    inv, table = rnd(pairs), rnd(n * 2 * pairs + offset)[offset:].view(n, 2 * pairs)
    res = []
    for cut in (n, 250):
        qkv = qkv0.clone()
        for a, b in _pieces(n, cut):
            q = _lib.QkvArgs()
            q.qkv, q.xn, q.pos = (t[a:b].data_ptr() for t in (qkv, x, pos))
            q.inv_freq, q.rope_cs, q.dtype, q.xn_raw = inv.data_ptr(), table[a:b].data_ptr(), 2, 1
            q.B, q.H, q.K, q.hd, q.d, q.n_pairs = b - a, H, K, hd, d, pairs
            _lib.check(_lib.lib().uv_qkv_post_args(C.byref(q), stream_ptr(x.device)), "uv_qkv_post")
        res.append(qkv)
    assert torch.equal(*res) and not torch.equal(res[0], qkv0)
