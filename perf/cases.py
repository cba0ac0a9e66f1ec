"""The calls a user of this framework makes, over the sizes they make them at.

Every case is UV-50M (the ``uv-50m-alpha`` preset with a 16384-token vocabulary) driven through the public entry points:

* ``step``     ``DecodeRunner.step``: a few consecutive decode steps of a running batch (prompts left-padded to one
               position, tokens fed back), with the logits of the last step
* ``prefill``  ``model.prefill`` of a left-padded batch of prompts
* ``rollout``  ``GpuScheduler``: a job of requests through continuous batching, enqueue to last harvest
* ``attn``     ``kernels.decode_attention`` called directly, as a host with its own step does
* ``sample``   ``kernels.fused_sample`` on raw head output
* ``publish``  ``publish_weights``: the trainer's fp32 parameters into the decode engine, once per RL step
"""
import math

import numpy as np
import torch

from ultraviolet_b200.fast_decode import KernelDecodeState
from ultraviolet_b200.generate import DecodeRunner
from ultraviolet_b200.kernels import decode_attention, fused_sample, quantize_kv
from ultraviolet_b200.model import MathLM, make_config
from ultraviolet_b200.rl_stream import publish_weights
from ultraviolet_b200.scheduler import GpuScheduler

DEV = "cuda:0"
VOCAB = 16384
CFG = make_config("uv-50m-alpha", vocab_size=VOCAB)
DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16}
GLOBAL = sum(CFG.is_global(l) for l in range(CFG.n_layers))
LOCAL = CFG.n_layers - GLOBAL
KEY_BYTES = 2 * CFG.n_kv_heads * (CFG.head_dim + 2)     # one cached position of one layer: int8 K and V, two scales
CHECK_EVERY = 32                                        # decode steps between two harvests of a rollout job


def listed():
    return [
        # one sequence, greedy: interactive use, nothing but latency
        dict(name="step_1", kind="step", batch=1, lo=200, hi=200, steps=4, temperature=0.0, top_p=1.0, dtype="bf16"),
        # an evaluation batch of odd size, nucleus sampling, fp16 weights
        dict(name="step_37_fp16_top_p", kind="step", batch=37, lo=300, hi=900, steps=4, temperature=0.8, top_p=0.95,
             dtype="fp16"),
        # the benchmark's batch: 256 sequences, short contexts, greedy
        dict(name="step_256", kind="step", batch=256, lo=32, hi=384, steps=8, temperature=0.0, top_p=1.0,
             dtype="bf16"),
        # a rollout generator's full set of slots, T = 1, contexts up to prompt + max_new
        dict(name="step_512", kind="step", batch=512, lo=64, hi=2304, steps=8, temperature=1.0, top_p=1.0,
             dtype="bf16"),
        # long contexts: the step is mostly KV-cache traffic
        dict(name="step_64_long", kind="step", batch=64, lo=8192, hi=8192, steps=4, temperature=1.0, top_p=1.0,
             dtype="bf16"),
        # one short prompt (latency) and the benchmark's prompt batch
        dict(name="prefill_1", kind="prefill", prompts=1, lo=48, hi=48, dtype="bf16"),
        dict(name="prefill_256", kind="prefill", prompts=256, lo=32, hi=128, dtype="bf16"),
        # a few long prompts, fp16: attention over long ranges, windowed and global
        dict(name="prefill_7_long_fp16", kind="prefill", prompts=7, lo=700, hi=2000, dtype="fp16"),
        # a GRPO-shaped round: more requests than slots, ragged stop lengths
        dict(name="rollout_256", kind="rollout", slots=256, requests=384, lo=64, hi=256, mean_new=80, max_new=256,
             temperature=0.8, dtype="bf16"),
        # the attention call alone: the ragged 16-row batch of the reference's tests, and long contexts
        dict(name="attn_16", kind="attn", batch=16, lo=32, hi=512, window=0, dtype="fp16"),
        # the sampler alone on a full batch of raw head output
        dict(name="sample_512", kind="sample", batch=512, temperature=1.0, top_p=1.0, dtype="bf16"),
        # weight refresh after a trainer step
        dict(name="publish", kind="publish", dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 4 + ["prefill"] * 2 + ["rollout", "attn", "attn", "sample"])
    dt = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "step":
        batch = _log_int(rng, 1, 512)
        hi = _log_int(rng, 40, min(8192, 2304 * 512 // batch))
        t, p = rng.choice([(0.0, 1.0), (1.0, 1.0), (0.8, 0.95)])
        return dict(kind=kind, batch=batch, lo=max(1, int(hi * rng.uniform(0.1, 1.0))), hi=hi, steps=rng.randint(2, 8),
                    temperature=t, top_p=p, dtype=dt)
    if kind == "prefill":
        hi = _log_int(rng, 16, 2000)
        return dict(kind=kind, prompts=_log_int(rng, 1, min(256, max(1, 32768 // hi))),
                    lo=max(2, int(hi * rng.uniform(0.2, 1.0))), hi=hi, dtype=dt)
    if kind == "rollout":
        slots, hi = rng.choice([32, 48, 96, 128, 200, 256]), rng.randint(16, 256)
        return dict(kind=kind, slots=slots, requests=int(slots * rng.uniform(0.6, 1.5)), lo=max(2, hi // 4), hi=hi,
                    mean_new=rng.randint(24, 80), max_new=rng.choice([96, 128, 200, 256]), temperature=0.8, dtype=dt)
    if kind == "attn":
        batch, window = _log_int(rng, 1, 512), rng.choice([0, 0, 256])
        hi = _log_int(rng, 32, min(8192, 2304 * 512 // batch))
        return dict(kind=kind, batch=batch, lo=max(1, int(hi * rng.uniform(0.1, 1.0))), hi=hi, window=window, dtype=dt)
    return dict(kind=kind, batch=_log_int(rng, 1, 512), temperature=rng.choice([0.7, 1.0]),
                top_p=rng.choice([1.0, 1.0, 0.95]), dtype=dt)


# ------------------------------------------------------------------------------------------------ the model
_models = {}


def _parameters(seed):
    """UV-50M with weights that act as a trained policy's do.  The random init leaves wo and w_down at zero, so nothing
    but the embedding would reach the head: they get small random values.  A trained head keeps unlikely tokens far
    below the softcap's knee: here 64 channels shared by every embedding row are turned around by one feature of the
    last MLP, which puts almost all probability on one token per position (as in RL rollouts, and a draw then does not
    hang on the last bit of a logit)."""
    torch.manual_seed(seed)
    with torch.device(DEV):
        m = MathLM(CFG)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    with torch.no_grad():
        m.embed.weight.normal_(std=0.08, generator=g)
        m.embed.weight[:, :64] = 0.1
        for b in m.blocks:
            b.attn.wo.normal_(std=0.02, generator=g)
            b.mlp.w_down.normal_(std=0.02, generator=g)
            b.attn.attn_gate.normal_(std=0.05, generator=g)
            b.attn.xsa_alpha.normal_(std=0.3, generator=g)
            if b.attn.has_ve:
                b.attn.ve_gate.normal_(std=0.1, generator=g)
            for lam in (b.resid_attn, b.post_attn, b.resid_mlp, b.post_mlp):
                lam.copy_(1.0 + 0.02 * torch.randn((), device=DEV, generator=g))
            b.mlp.w_down[:64] = 0.0
            b.attn.wo[:64] = 0.0
        last = m.blocks[-1].mlp
        last.w_gate[0], last.w_up[0] = 0.0, 0.0
        last.w_gate[0, :64], last.w_up[0, :64] = 0.03, 0.03
        last.w_down[:, 0] = 0.0
        last.w_down[:64, 0] = -1.2
    return m


def _model(dtype):
    """The checkpoint a program keeps in hand, one per dtype."""
    if dtype not in _models:
        _models[dtype] = _parameters(0).to(DTYPE[dtype]).fuse_for_inference(DTYPE[dtype])
    return _models[dtype]


def _lengths(case, n, g):
    """n lengths in [lo, hi], the longest present (it sets the padded frame)."""
    x = torch.randint(case["lo"], case["hi"] + 1, (n,), generator=g)
    x[int(torch.randint(0, n, (1,), generator=g))] = case["hi"]
    return x


def _fill(cache, scale, g):
    """Quantised N(0, 1) keys / values in every slot (in pieces: a long cache as fp32 is four times its int8 bytes)."""
    for b in range(0, cache.size(0), 64):
        q, s = quantize_kv(torch.randn(cache[b:b + 64].shape, device=DEV, generator=g, dtype=torch.float32))
        cache[b:b + 64].copy_(q)
        scale[b:b + 64].copy_(s)


def _state(batch, max_len, dtype, g):
    st = KernelDecodeState(CFG, batch, max_len, DTYPE[dtype], DEV)
    for l in range(CFG.n_layers):
        _fill(st.k[l], st.k_scale[l], g)
        _fill(st.v[l], st.v_scale[l], g)
    return st


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    gc = torch.Generator().manual_seed(seed)
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind, dt = case["kind"], case["dtype"]
    s = dict(case=case)
    if kind == "step":
        B, P = case["batch"], case["hi"]
        s["st"] = st = _state(B, P + case["steps"] + 1, dt, g)
        st.starts.copy_(P - _lengths(case, B, gc))
        st.set_pos(P)
        s["pos"], s["host_pos"] = st.pos.clone(), st.host_pos.copy()
        s["tok"] = torch.randint(1, VOCAB, (B,), device=DEV, generator=g)
        s["runner"] = DecodeRunner(_model(dt), st, temperature=case["temperature"], top_p=case["top_p"], seed=seed)
        s["runner"].step(s["tok"])                      # captures the step's graph
    elif kind == "prefill":
        n, T = case["prompts"], case["hi"]
        s["starts"] = (T - _lengths(case, n, gc)).to(DEV)
        s["idx"] = torch.randint(1, VOCAB, (n, T), device=DEV, generator=g)
        s["idx"].masked_fill_(torch.arange(T, device=DEV)[None] < s["starts"][:, None], 0)
        s["model"] = _model(dt)
        s["st"] = s["model"].new_state(n, T + 64)
    elif kind == "rollout":
        r, n = np.random.default_rng(seed), case["requests"]
        s["prompts"] = [r.integers(1, VOCAB, int(k)).tolist() for k in r.integers(case["lo"], case["hi"] + 1, n)]
        # geometric stop lengths, one from each of n equal slices of the distribution: a job's total is always the same
        q = (np.arange(n) + 0.5) / n
        s["limits"] = np.minimum(np.ceil(np.log1p(-q) / math.log1p(-1.0 / case["mean_new"])).astype(int),
                                 case["max_new"])[r.permutation(n)]
        m = _model(dt)
        st = m.new_state(GpuScheduler.state_rows(case["slots"], packed_prefill=True),
                         case["hi"] + case["max_new"] + CHECK_EVERY)
        s["sched"] = GpuScheduler(m.engine, st, max_new=case["max_new"], temperature=case["temperature"], eos_id=0,
                                  seed=seed, q_cap=2 * n, max_prompt=case["hi"], packed_prefill=True)
    elif kind == "attn":
        B, S = case["batch"], case["window"] or (case["hi"] + 7) // 8 * 8
        H, K, hd = CFG.n_heads, CFG.n_kv_heads, CFG.head_dim
        s["q"] = torch.randn(B, H, hd, device=DEV, generator=g).to(DTYPE[dt])
        s["k"], s["v"] = (torch.empty(B, K, S, hd, dtype=torch.int8, device=DEV) for _ in range(2))
        s["ks"], s["vs"] = (torch.empty(B, K, S, dtype=torch.float16, device=DEV) for _ in range(2))
        _fill(s["k"], s["ks"], g)
        _fill(s["v"], s["vs"], g)
        s["pos"] = (_lengths(case, B, gc) - 1).to(DEV)
        s["starts"] = torch.zeros(B, dtype=torch.long, device=DEV)
    elif kind == "sample":
        B = case["batch"]
        x = torch.randn(B, VOCAB, device=DEV, generator=g) * 2.0 - 14.0
        top = torch.randint(0, VOCAB, (B, 4), device=DEV, generator=g)      # a handful of plausible tokens per row
        x.scatter_(1, top, torch.rand(B, 4, device=DEV, generator=g) * 12.0 + 4.0)
        s["x"] = x.to(DTYPE[dt])
        s["u"] = torch.rand(B, device=DEV, generator=g)
    else:
        s["raw"] = _parameters(seed)
        with torch.device(DEV):
            s["gen"] = MathLM(CFG).to(DTYPE[dt]).fuse_for_inference(DTYPE[dt])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        st, runner, tok = s["st"], s["runner"], s["tok"]
        st.pos.copy_(s["pos"])
        st.host_pos[:] = s["host_pos"]
        runner.steps.zero_()
        toks, logps = [], []
        for _ in range(case["steps"]):
            tok = runner.step(tok).clone()
            toks.append(tok)
            logps.append(runner.out_logp.clone())
        return dict(tok=torch.stack(toks), logp=torch.stack(logps), logits=runner.out_logits)
    if kind == "prefill":
        st = s["st"]
        logits = s["model"].prefill(s["idx"], s["starts"], st)
        # (the int8 bytes are not compared: where a bf16 rounding differs they move by one step)
        return dict(logits=logits, k_scale=st.k_scale, v_scale=st.v_scale, pos=st.pos)
    if kind == "rollout":
        sched, n = s["sched"], case["requests"]
        sched.enqueue(s["prompts"], limits=s["limits"], keys=np.arange(n), metas=list(range(n)))
        done = []
        while len(done) < n:
            done += sched.unpack(sched.window(CHECK_EVERY))
            if len(done) < n and sched.live_bound() == 0:
                done += sched.harvest()
        done.sort(key=lambda d: d[0])
        return dict(tok=np.concatenate([np.asarray(t) for _, t, _, _ in done]),
                    logp=np.concatenate([lp for _, _, lp, _ in done]))
    if kind == "attn":
        return decode_attention(s["q"], s["k"], s["v"], s["pos"], s["starts"], CFG.attn_scale, window=case["window"],
                                k_scale=s["ks"], v_scale=s["vs"])
    if kind == "sample":
        tok, logp = fused_sample(s["x"], s["u"], CFG.softcap, case["temperature"], top_p=case["top_p"])
        return dict(tok=tok, logp=logp)
    publish_weights(s["gen"], s["raw"])
    eng = s["gen"].engine
    return dict(arena=eng.arena, arena32=eng.arena32)


_LAYER_W = CFG.param_counts()["non_embedding"]
_HEAD_W = VOCAB * CFG.d_model


def _keys(case, extra=0.0):
    """Mean cached positions read per row, summed over the layers."""
    n = 0.5 * (case["lo"] + case["hi"]) + extra
    return GLOBAL * n + LOCAL * min(n, CFG.window)


def work(case):
    kind, d, hd, H = case["kind"], CFG.d_model, CFG.head_dim, CFG.n_heads
    if kind == "step":
        B, k = case["batch"], case["steps"]
        keys = _keys(case, 0.5 * k)
        return dict(bytes=k * (2 * (_LAYER_W + _HEAD_W) + B * (keys + CFG.n_layers) * KEY_BYTES + 20 * B)
                    + 4 * B * VOCAB, flops=k * B * (2 * (_LAYER_W + _HEAD_W) + 4 * H * hd * keys))
    if kind == "prefill":
        n, t = case["prompts"], 0.5 * (case["lo"] + case["hi"])
        w = min(t, CFG.window)
        pairs = GLOBAL * t * t / 2 + LOCAL * (t * w - w * w / 2)
        cached = GLOBAL * t + LOCAL * w
        return dict(bytes=2 * (_LAYER_W + _HEAD_W) + n * (cached * KEY_BYTES + 8 * t + 4 * VOCAB),
                    flops=n * (2 * _LAYER_W * t + 2 * _HEAD_W + 4 * H * hd * pairs))
    if kind == "rollout":
        n, p = case["requests"], 0.5 * (case["lo"] + case["hi"])
        new = case["mean_new"] * (1 - math.exp(-case["max_new"] / case["mean_new"]))
        passes = max(case["max_new"], n * new / case["slots"])      # dependent steps: the weights are read in each
        return dict(bytes=passes * 2 * (_LAYER_W + _HEAD_W) + n * new * _keys(dict(lo=p, hi=p), new / 2) * KEY_BYTES,
                    flops=n * (2 * _LAYER_W * (p + new) + 2 * _HEAD_W * new))
    if kind == "attn":
        B, n = case["batch"], 0.5 * (case["lo"] + case["hi"])
        n = min(n, case["window"]) if case["window"] else n
        return dict(bytes=B * (n * KEY_BYTES + 2 * H * hd * 2 + 16), flops=4 * B * H * hd * n)
    if kind == "sample":
        return dict(bytes=case["batch"] * (2 * VOCAB + 16), flops=10 * case["batch"] * VOCAB)
    values = _LAYER_W + _HEAD_W + VOCAB * hd
    return dict(bytes=6 * values, flops=values)


def tolerance(case):
    """Half-precision weights and activations through ten layers; log-probs of near-certain tokens are small
    differences, hence 3e-2 there.  Attention alone: one rounding of the output.  Sampling alone: 32-bit sums, ties
    where a draw falls on the edge of a token.  Weights: one rounding, the products before it in either order."""
    kind = case["kind"]
    if kind in ("step", "rollout"):
        return {"rel": 3e-2, "max": 0.9, "differ": 0.01}
    if kind == "prefill":
        return {"rel": 2e-2, "max": 0.5}
    if kind == "attn":
        return {"rel": 5e-3 if case["dtype"] == "bf16" else 2e-3, "max": 0.05}
    if kind == "sample":
        return {"rel": 1e-3, "max": 0.5, "differ": 0.005}
    return {"rel": 2e-3, "max": 0.02}
