"""All layers of a decode step in one launch (uv_decode_step) against one launch per operation: hidden states, appended
cache entries and the count of skipped writes after several steps.  Batches around the row tiles, mixed contexts (a single
key, ends inside a chunk, ring caches before and after they wrap, a position past the cache), remapped cache rows, models
with fewer heads, odd gate widths, other rotation widths and features left out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(dtype, **over):
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(3)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", **over))
    g = torch.Generator(device="cuda").manual_seed(4)
    with torch.no_grad():
        for b in m.blocks:
            for w in (b.attn.wo, b.mlp.w_down):
                w.normal_(std=0.02, generator=g)
            if m.cfg.gate_channels:
                b.attn.attn_gate.normal_(std=0.05, generator=g)
    return m.to(dtype).fuse_for_inference(dtype)


def _state(cfg, rows, max_len, dtype, g):
    from ultraviolet_b200.fast_decode import KernelDecodeState
    st = KernelDecodeState(cfg, rows, max_len, dtype, "cuda")
    for l in range(cfg.n_layers):
        for kv, sc in ((st.k[l], st.k_scale[l]), (st.v[l], st.v_scale[l])):
            kv.copy_(torch.randint(-127, 128, kv.shape, device="cuda", generator=g, dtype=torch.int8))
            sc.copy_(torch.rand(sc.shape, device="cuda", generator=g).to(sc.dtype) * 0.02)
    return st


SMALL = dict(vocab_size=300, d_model=128, n_layers=3, d_ff=192, global_every=2, window=40)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,max_len,over", [
    (1, 300, {}), (8, 700, {}), (9, 130, {}), (16, 300, {}), (17, 530, {}), (32, 400, {}), (48, 400, {}),
    (3, 90, SMALL), (33, 200, dict(SMALL, n_heads=3, xsa=False)), (2, 60, dict(SMALL, d_model=64, d_ff=64, n_heads=1)),
    (5, 100, dict(SMALL, attn_gate_channels=18, ve_gate_channels=5, window=33)),
    (7, 100, dict(SMALL, d_model=1024, d_ff=2048, n_layers=2))])
def test_one_launch_against_single_kernels(dtype, B, max_len, over):
    import ctypes as C
    from ultraviolet_b200 import _lib
    m = _model(dtype, **over)
    eng = m.engine
    cfg, rows = eng.cfg, B + 3
    gc = torch.Generator().manual_seed(B)
    res = []
    for one in (True, False):
        g = torch.Generator(device="cuda").manual_seed(B)
        st = _state(cfg, rows, max_len, dtype, g)
        gc.manual_seed(B)
        pos = torch.randint(0, max_len - 3, (B,), generator=gc)
        pos[0] = max_len - 4
        starts = (pos * torch.rand(B, generator=gc)).long()
        if B > 2:
            pos[1], starts[1] = 0, 0
            pos[2] = starts[2] = max_len - 2                    # its third step lies past the cache
        rm = torch.randperm(rows, generator=gc)[:B].cuda()
        pos, starts = pos.cuda(), starts.cuda()
        eng.one_launch = one
        out = []
        for step in range(3):
            tok = torch.randint(0, cfg.vocab_size, (B,), device="cuda", generator=g)
            out.append(eng.trunk(tok, st, pos, starts, g_len=max_len, row_map=rm).float().clone())
            pos = pos + 1
        if one:
            a = eng._step_args(tok, st, pos, starts, rm.data_ptr(), eng.scratch(B))
            assert _lib.lib().uv_decode_step_supported(C.byref(a)) == 1
        res.append((out, st, eng.device_status(B)))
        eng.scratch(B)["flags"].zero_()
    (xs, sa, fa), (ys, sb, fb) = res
    tol = 3e-2 if dtype == torch.bfloat16 else 5e-3
    for x, y in zip(xs, ys):
        assert (x - y).norm() <= tol * y.norm() and (x - y).abs().max() <= 4 * tol * y.abs().max()
    assert fa["attn_status"] == fb["attn_status"] == 0 and fa["kv_oob"] == fb["kv_oob"]
    for l in range(cfg.n_layers):
        for p, q in ((sa.k[l], sb.k[l]), (sa.v[l], sb.v[l])):
            d = (p.int() - q.int()).abs()
            assert d.max() <= (2 if l == 0 else 12) and (d > 1).float().mean() < 1e-3
        for p, q in ((sa.k_scale[l], sb.k_scale[l]), (sa.v_scale[l], sb.v_scale[l])):
            assert torch.allclose(p.float(), q.float(), rtol=4 * tol, atol=0)


def test_launch_count():
    m = _model(torch.bfloat16, vocab_size=300, n_layers=2)
    eng, st = m.engine, m.new_state(300, 40)
    assert eng.launches_per_step(st, 1) == eng.launches_per_step(st, 48) == 2
    assert eng.launches_per_step(st) == eng.launches_per_step(st, 256) == eng.launches_per_step() == 1 + 7 * 2 + 2
    eng.one_launch = False
    assert eng.launches_per_step(st, 1) == 17
