"""The native host paths against the Python ones they stand in for: same launches, so the same bits; and the launches
around a packed prompt pass (offsets, packing, last-token norm, softcap) at the sizes where they can go wrong."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,window,dtype,splits", [(1, 40, 0, torch.float16, None), (37, 900, 0, torch.bfloat16, None),
                                                     (5, 256, 256, torch.bfloat16, None), (3, 4096, 0, torch.float16, 12)])
def test_decode_attention_host_path(B, S, window, dtype, splits):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels import decode_attention
    from ultraviolet_b200.kernels.decode_attn import _decode_attn_op, default_splits
    g = torch.Generator(device="cuda").manual_seed(S)
    q = torch.randn(B, 8, 64, device="cuda", generator=g).to(dtype)
    k, v = (torch.randint(-127, 128, (B, 1, S, 64), device="cuda", generator=g, dtype=torch.int8) for _ in range(2))
    ks, vs = (torch.rand(B, 1, S, device="cuda", generator=g).half() * 0.02 for _ in range(2))
    pos = torch.randint(0, S, (B,), device="cuda", generator=g)
    st = torch.zeros(B, dtype=torch.long, device="cuda")
    args = (q, k, v, pos, st, 0.14)
    native = _lib.host().decode_attention(*args, window, -1, ks, vs, 0, splits or -2 ** 31)
    assert native is not None
    n = splits or default_splits(B, min(S, window) if window else S, q.device)
    want = _decode_attn_op(*args, window, window > 0, ks, vs, n)
    assert torch.equal(native, want)
    assert torch.equal(decode_attention(*args, window=window, k_scale=ks, v_scale=vs, num_splits=splits), want)
    # numbers of any kind
    assert torch.equal(decode_attention(*args[:5], torch.tensor(0.14, dtype=torch.float64), window=float(window), k_scale=ks,
                                        v_scale=vs, num_splits=float(n), ctx_hint=float(S)), want)
    # what it does not take goes to the op: gradients wanted, other index types, a dispatch mode
    assert _lib.host().decode_attention(q.clone().requires_grad_(), k, v, pos, st, 0.14, window, -1, ks, vs, 0, 1) is None
    assert torch.equal(decode_attention(q, k, v, pos.int(), st, 0.14, window=window, k_scale=ks, v_scale=vs,
                                        num_splits=n), want)
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode() as mode:
        fake = [mode.from_tensor(t) for t in (q, k, v, pos, st, ks, vs)]
        out = decode_attention(*fake[:5], 0.14, window=window, k_scale=fake[5], v_scale=fake[6], num_splits=n)
        assert out.shape == q.shape
    with pytest.raises(RuntimeError):
        decode_attention(*args, window=window, k_scale=ks, v_scale=vs, num_splits=-1)


@pytest.mark.parametrize("lens,T", [([1], 1), ([0, 5, 16, 17, 0], 17), (list(range(1500)), 1500)])
def test_prompt_packing(lens, T):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.fast_decode import pack_prompts
    from ultraviolet_b200.kernels._util import stream_ptr
    n, dev = len(lens), "cuda"
    lens = np.minimum(np.array(lens), T)
    g = torch.Generator(device=dev).manual_seed(n)
    idx = torch.randint(0, 99, (n, T + 3), device=dev, generator=g)[:, 1:T + 1]
    starts, rows = torch.from_numpy(T - lens).to(dev), torch.randperm(n, device=dev, generator=g)
    M = int(lens.sum())
    out = torch.full((4, max(M, 1)), -1, dtype=torch.int64, device=dev)
    cu = torch.full((2, n + 1), -1, dtype=torch.int32, device=dev)
    _lib.check(_lib.lib().uv_pack_prompts(idx.data_ptr(), idx.stride(0), T, starts.data_ptr(), rows.data_ptr(), n, M,
                                          cu[0].data_ptr(), cu[1].data_ptr(), *(o.data_ptr() for o in out),
                                          stream_ptr(out.device)), "uv_pack_prompts")
    want = pack_prompts(idx, starts, rows, lens)
    assert torch.equal(cu[0], want["cu"]) and torch.equal(cu[1], want["tile_cu"])
    for got, name in zip(out, ("tok", "pos", "rows", "last_pos")):
        assert torch.equal(got[:M], want[name])
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.randn(max(M, 1), 72, device=dev, generator=g).to(dtype)
        y = torch.empty(n, 72, dtype=dtype, device=dev)
        _lib.check(_lib.lib().uv_gather_norm(x.data_ptr(), 1 if dtype == torch.float16 else 2, 72, cu[0].data_ptr(), n,
                                             y.data_ptr(), stream_ptr(x.device)), "uv_gather_norm")
        ref = torch.nn.functional.rms_norm(x.float(), (72,))[want["last_row"]].masked_fill(want["empty"][:, None], 0)
        assert torch.allclose(y.float(), ref, rtol=1e-2, atol=1e-3)


@pytest.mark.parametrize("shape", [(1, 3), (7, 16384), (3, 1003)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_softcap(shape, dtype):
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.kernels._util import DTYPE_CODE, stream_ptr
    x = (torch.randn(shape, device="cuda") * 20).to(dtype)
    out = torch.empty(shape, device="cuda")
    _lib.check(_lib.lib().uv_softcap(x.data_ptr(), DTYPE_CODE[dtype], x.numel(), 23.0, 5.0, 7.5, out.data_ptr(),
                                     stream_ptr(x.device)), "uv_softcap")
    assert torch.allclose(out, 23.0 * torch.sigmoid((x.float() + 5.0) / 7.5), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("switch", [None, "allow_fp16_reduced_precision_reduction", "allow_bf16_reduced_precision_reduction",
                                    "allow_fp16_accumulation", "library"])
def test_prefill_follows_the_switches_of_matmul(dtype, switch, monkeypatch):
    """The native prompt pass gives the bits of the one that calls torch.mm, whatever torch's matrix products are set to."""
    from ultraviolet_b200.engine import DecodeEngine
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(5)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", vocab_size=500, n_layers=3, global_every=2))
    with torch.no_grad():
        for b in m.blocks:
            b.attn.wo.normal_(std=0.02), b.mlp.w_down.normal_(std=0.02)
    m = m.to(dtype).fuse_for_inference(dtype)
    lens, T = torch.tensor([300, 1, 17, 290, 260]), 300
    idx = torch.randint(1, 500, (5, T), device="cuda")
    starts = (T - lens).cuda()
    mm = torch.backends.cuda.matmul
    before = mm.allow_fp16_accumulation if switch == "allow_fp16_accumulation" else True
    lib = torch.backends.cuda.preferred_blas_library()
    try:
        if switch == "library":
            torch.backends.cuda.preferred_blas_library("cublaslt")
        elif switch:
            setattr(mm, switch, not before)
        assert (m.engine.prefill_trunk() is None) == bool(switch)
        res = []
        for native in (True, False):
            if not native:
                monkeypatch.setattr(DecodeEngine, "prefill_trunk", lambda self: None)
            st = m.new_state(5, T + 8)
            res.append((m.prefill(idx, starts, st), *st.k, *st.v, *st.k_scale, *st.v_scale))
        for a, b in zip(*res):
            assert torch.equal(a, b)
    finally:
        torch.backends.cuda.preferred_blas_library(lib)
        if switch and switch != "library":
            setattr(mm, switch, before)


@pytest.mark.parametrize("native", [True, False])
def test_prefill_keeps_no_buffers_per_length(native, monkeypatch):
    """Prompts of many lengths one after the other: what a pass allocated is given back (native pass) or shared by the lengths of a
    bucket (the pass through ``trunk``), and its count of skipped cache writes is read with the other failure words."""
    from ultraviolet_b200 import _lib
    from ultraviolet_b200.engine import DecodeEngine
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(6)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", vocab_size=500, n_layers=2)).bfloat16().fuse_for_inference()
    if not native:
        monkeypatch.setattr(DecodeEngine, "prefill_trunk", lambda self: None)
    eng, st = m.engine, m.new_state(1, 2200)
    used = []
    for T in (2150, 2049, *range(1, 130, 3), 1000, 2048):
        m.prefill(torch.ones(1, T, dtype=torch.long, device="cuda"), torch.zeros(1, dtype=torch.long, device="cuda"), st)
        used.append(torch.cuda.memory_allocated())
    if native:
        assert not eng._scratch and max(used[1:]) == min(used[1:])
        eng.prefill_oob()[0] = 2
        with pytest.raises(_lib.UvError):
            eng.check_status(1)
        assert eng.device_status() == {"attn_status": 0, "kv_oob": 0}
    else:
        assert sorted(k[0] for k in eng._scratch) == [64, 128, 1024, 2048, 4096]        # (1 ... 127, 1000, 2048, 2049, 2150)


def test_prefill_into_strided_rows_and_what_it_refuses():
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(7)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", vocab_size=500, n_layers=2)).bfloat16().fuse_for_inference()
    idx, starts = torch.randint(1, 500, (3, 20), device="cuda"), torch.tensor([0, 5, 19], device="cuda")
    rows = torch.tensor([[6, 0], [1, 0], [4, 0]], device="cuda")
    res = []
    for r, s in ((rows[:, 0], starts), (torch.tensor([6, 1, 4], device="cuda"), starts),
                 (rows[:, 0].int(), torch.stack([starts, starts], 1)[:, 1].int())):
        st = m.new_state(8, 24)
        res.append((m.prefill(idx, s, st, rows=r), st.pos, st.starts, *st.k, *st.v))
    for other in res[1:]:
        for a, b in zip(res[0], other):
            assert torch.equal(a, b)
    st, good = m.new_state(8, 24), torch.tensor([6, 1, 4], device="cuda")
    for bad in (dict(rows=good[:2]), dict(rows=good[:, None]), dict(starts=starts[:1]), dict(starts=torch.zeros(4).cuda().long())):
        with pytest.raises(ValueError):
            m.prefill(idx, bad.get("starts", starts), st, rows=bad.get("rows", good))
    for bad in (dict(rows=good.cpu()), dict(starts=starts.cpu()), dict(idx=idx.cpu())):
        with pytest.raises(RuntimeError):
            m.prefill(bad.get("idx", idx), bad.get("starts", starts), st, rows=bad.get("rows", good))
    assert not any(k.any() for k in st.k)
    for field in ("k", "v", "k_scale", "v_scale"):          # a state of a model with fewer layers
        few = m.new_state(8, 24)
        getattr(few, field).pop()
        with pytest.raises(IndexError):
            m.prefill(idx, starts, few, rows=good)


def test_watched_attention_calls_go_through_the_op():
    """Tracers, transforms and subclasses see the custom op, not a result computed behind their back."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from ultraviolet_b200.kernels import decode_attention
    g = torch.Generator(device="cuda").manual_seed(0)

    def inputs():
        q = torch.randn(4, 8, 64, device="cuda", generator=g).half()
        k, v = (torch.randint(-127, 128, (4, 1, 64, 64), device="cuda", generator=g, dtype=torch.int8) for _ in range(2))
        ks, vs = (torch.rand(4, 1, 64, device="cuda", generator=g).half() * 0.02 for _ in range(2))
        return q, k, v, torch.full((4,), 50, device="cuda"), torch.zeros(4, dtype=torch.long, device="cuda"), ks, vs

    def f(q, k, v, pos, starts, ks, vs):
        return decode_attention(q, k, v, pos, starts, 0.1, k_scale=ks, v_scale=vs, num_splits=1)
    a, b = inputs(), inputs()
    want = f(*b)
    assert torch.equal(torch.jit.trace(f, a, check_trace=False)(*b), want)
    for pre in (False, True):
        assert torch.equal(make_fx(f, pre_dispatch=pre)(*a)(*b), want)
    assert torch.equal(torch.func.vmap(f)(*(torch.stack(t) for t in zip(a, b)))[1], want)
    seen = []

    class Watch(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return super().__torch_function__(func, types, args, kwargs or {})
    f(b[0].as_subclass(Watch), *b[1:])
    assert any("decode_attn" in n for n in seen)
    # a view that stands for other values than those in memory
    assert torch.equal(f(torch._neg_view(b[0]), *b[1:]), f(-b[0], *b[1:]))


def test_logits_keep_gradients_and_transforms():
    """MathLM.logits of hidden states that want gradients, or under a transform or tracer, is the tensor expression."""
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(8)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", vocab_size=500, n_layers=1)).bfloat16().fuse_for_inference()
    w, (a, b, c) = m.engine.w["embed"], m.cfg.softcap
    h, t = torch.randn(2, 5, w.size(1), device="cuda").bfloat16()
    ref = lambda x: a * torch.sigmoid((torch.mm(x, w.t()).float() + b) / c)
    assert torch.allclose(m.logits(h), ref(h), rtol=1e-5, atol=1e-6)
    x, y = h.clone().requires_grad_(), h.clone().requires_grad_()
    got, want = m.logits(x), ref(y)
    got.square().sum().backward(), want.square().sum().backward()
    assert torch.equal(got, want) and torch.equal(x.grad, y.grad) and x.grad.any()
    for p, q in zip(torch.func.jvp(m.logits, (h,), (t,)), torch.func.jvp(ref, (h,), (t,))):
        assert torch.equal(p, q)
    assert torch.equal(torch.func.vmap(m.logits)(torch.stack([h, t])), torch.func.vmap(ref)(torch.stack([h, t])))
    assert torch.equal(torch.jit.trace(lambda x: m.logits(x), (h,), check_trace=False)(t), ref(t))


def test_watched_prefill_shows_its_products():
    from torch.utils.flop_counter import FlopCounterMode
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(9)
    with torch.device("cuda"):
        m = MathLM(make_config("uv-50m-alpha", vocab_size=500, n_layers=2)).bfloat16().fuse_for_inference()
    idx, starts = torch.randint(1, 500, (3, 20), device="cuda"), torch.tensor([0, 5, 19], device="cuda")
    M, c = 20 + 15 + 1, m.cfg
    d, q, kv, f = c.d_model, c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim, c.d_ff
    a, b = m.new_state(3, 24), m.new_state(3, 24)
    want = m.prefill(idx, starts, a)
    with FlopCounterMode(display=False) as count:
        got = m.prefill(idx, starts, b)
    # (QKV, gate | up and the head; the counter does not know the in-place addmm_ of the other two)
    assert count.get_total_flops() == 2 * (c.n_layers * M * d * (q + 2 * kv + 2 * f) + 3 * d * 500)
    assert torch.allclose(got, want, rtol=1e-5, atol=1e-6)
    for x, y in zip(a.k + a.v + a.k_scale, b.k + b.v + b.k_scale):
        assert torch.equal(x, y)
