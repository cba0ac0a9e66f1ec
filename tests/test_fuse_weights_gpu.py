"""uv_fuse_weights (the one-launch load_from) against the tensor operations it replaces: same bits, for every pair of
parameter and engine dtypes, on matrices smaller than a block, not a multiple of it, and whose rows break 16-byte
alignment, and for a folded and a literal residual stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(over, dtype, seed=0):
    from ultraviolet_b200.model import MathLM, make_config
    torch.manual_seed(seed)
    m = MathLM(make_config("tiny", xsa=True, **over)).cuda()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn_like(p) * 0.2 if p.dim() else 1.0 + 0.2 * torch.randn_like(p))
    return m.to(dtype)


@pytest.mark.parametrize("over", [{}, dict(d_model=72, d_ff=136, head_dim=64, n_kv_heads=1),
                                  dict(d_model=200, d_ff=328, vocab_size=1000, n_layers=3, attn_gate_channels=13)])
@pytest.mark.parametrize("src", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dst", [torch.float16, torch.bfloat16])
def test_one_launch_gives_the_bits_of_the_tensor_ops(over, src, dst):
    from ultraviolet_b200.engine import DecodeEngine
    m = _model(over, src)
    eng = DecodeEngine.from_model(m, dst)
    n32 = eng.cfg.n_layers * eng.n32_layer
    for fold in (True, False):
        eng.fold = fold
        with torch.no_grad():
            eng._fuse_by_tensor_ops(m)
        want, want32 = eng.arena.clone(), eng.arena32.clone()
        eng.arena.fill_(7)
        eng.arena32[:n32].fill_(7)
        eng.load_from(m)
        assert eng._fuse_plan["args"] is not None
        for name, (off, shp) in eng.layout.items():
            n = torch.Size(shp).numel()
            assert torch.equal(eng.arena[off:off + n], want[off:off + n]), (name, fold)
        assert torch.equal(eng.arena32, want32)


def test_parameters_it_cannot_take_and_lambdas_it_cannot_fold():
    from ultraviolet_b200.engine import DecodeEngine
    m = _model({}, torch.float32)
    eng = DecodeEngine.from_model(m, torch.bfloat16)
    want = eng.arena.clone()
    m.blocks[1].attn.wo.data = m.blocks[1].attn.wo.data.t().contiguous().t()      # not contiguous: tensor operations
    eng.arena.zero_()
    eng.load_from(m)
    assert eng._fuse_plan["args"] is None and torch.equal(eng.arena, want)
    m.blocks[1].attn.wo.data = m.blocks[1].attn.wo.data.contiguous()
    m.blocks[2].resid_mlp.data.fill_(1e-3)
    with pytest.raises(ValueError, match="layer 2"):
        eng.load_from(m)


@pytest.mark.parametrize("name,shape", [("wq", (40, 64)), ("wk", (64, 32)), ("attn_gate", (4, 8)), ("xsa_alpha", (2,)),
                                        ("o_scale", (1,)), ("embed", (500, 64)), ("value_embed", (512, 16))])
def test_shapes_that_are_not_the_configs(name, shape):
    """Parameters of other shapes are not for the launch, which reads them by the config's: they go to the tensor operations, which
    take or refuse them."""
    from ultraviolet_b200.engine import DecodeEngine
    m = _model({}, torch.float32)
    eng = DecodeEngine.from_model(m, torch.bfloat16)
    at = m.blocks[1].attn
    p = getattr(m, name).weight if "embed" in name else getattr(at, name)
    assert p.shape != shape
    p.data = torch.ones(shape, device="cuda")
    if name == "o_scale":
        eng.load_from(m)
    else:
        with pytest.raises(RuntimeError):
            eng.load_from(m)
    assert eng._fuse_plan["args"] is None


def test_same_memory_other_form():
    """Parameters that come back in the same memory with another shape, order or type are looked at again."""
    from ultraviolet_b200.engine import DecodeEngine
    m = _model(dict(d_model=64, n_heads=4, head_dim=16), torch.float32)         # wq and wo are square
    eng = DecodeEngine.from_model(m, torch.bfloat16)
    eng.load_from(m)
    plan = eng._fuse_plan
    eng.load_from(m)
    assert eng._fuse_plan is plan and plan["args"] is not None
    at = m.blocks[2].attn
    at.wq.data = at.wq.data.t()
    eng.load_from(m)
    got = eng.arena.clone()
    with torch.no_grad():
        eng._fuse_by_tensor_ops(m)
    assert torch.equal(got, eng.arena) and eng._fuse_plan["args"] is None
    at.wq.data = at.wq.data.t()
    eng.load_from(m)
    assert eng._fuse_plan["args"] is not None
    at.wk.data = at.wk.data.reshape(-1)
    with pytest.raises((RuntimeError, ValueError)):
        eng.load_from(m)


def test_parametrised_weight():
    from ultraviolet_b200.engine import DecodeEngine
    m = _model({}, torch.float32)
    eng = DecodeEngine.from_model(m, torch.bfloat16)

    class Double(torch.nn.Module):
        def forward(self, w):
            return 2 * w
    torch.nn.utils.parametrize.register_parametrization(m.blocks[0].attn, "wv", Double())
    eng.load_from(m)
    got = eng.arena.clone()
    with torch.no_grad():
        eng._fuse_by_tensor_ops(m)
    assert torch.equal(got, eng.arena) and eng._fuse_plan["args"] is None
