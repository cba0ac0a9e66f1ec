"""The prompt a tile of uv_prefill_attn belongs to, found 32 prefix sums at a time: prompt counts around the steps of that
search, prompts without tokens among them; every prompt's rows against the same prompt handed over in a small batch."""
import numpy as np
import pytest

from tests.test_prefill_gpu import _run_attn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 1023, 1025])
def test_many_prompts(n):
    import torch
    r = np.random.default_rng(n)
    lens = r.integers(0, 40, n).tolist()
    lens[0], lens[-1] = 5, 17
    H, K, hd, cu = 4, 1, 64, np.concatenate([[0], np.cumsum(lens)])
    qkv = r.standard_normal((cu[-1], (H + 2 * K) * hd)).astype(np.float32)
    xsa, gates = r.uniform(0, 1, H).astype(np.float32), r.uniform(0, 2, (cu[-1], H)).astype(np.float32)
    out, _ = _run_attn(qkv, lens, H, K, hd, 24, 0.2, torch.bfloat16, xsa=xsa, gates=gates)
    for a in range(0, n, 7):
        b = min(a + 7, n)
        if cu[b] > cu[a]:
            want, _ = _run_attn(qkv[cu[a]:cu[b]], lens[a:b], H, K, hd, 24, 0.2, torch.bfloat16, xsa=xsa, gates=gates[cu[a]:cu[b]])
            assert (out[cu[a]:cu[b]] == want).all()
