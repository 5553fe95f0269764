"""Prompt attention (``cobalt_attn_prompt``, tcgen05) against the spec's arithmetic in fp64 (needs a B200).

Reference: scores rounded to bf16, scaled and rounded again, fp32 softmax, probabilities rounded to bf16
(src/cobaltkernel/ref_llama.py:117-137), every contraction in fp64.  Tolerance: the result is a bf16 rounding (at most 2^-9
relative per element) of a sum whose bf16 scores and probabilities may fall on the other side of a rounding boundary (at most
2^-8 relative each, for a small share of them): 2^-8 on the 2-norm, and 2^-6 of the largest value on a single element.
"""
import pytest
import torch

from cobalt_b200 import _lib

pytestmark = pytest.mark.gpu


def spec(q, k, v, pos, n_slots, window, scale, nh, nkv, D):
    T, rep = q.shape[0], nh // nkv
    slots = torch.arange(n_slots, device=q.device)
    allowed = slots[None] <= pos[:, None]
    if window > 0:
        allowed &= slots[None] > pos[:, None] - window
    out = torch.empty(T, nh, D, dtype=torch.float64, device=q.device)
    for h in range(nh):
        s = (q.view(T, nh, D)[:, h].double() @ k[h // rep, :n_slots].double().t()).to(torch.bfloat16) * scale
        p = torch.softmax(s.float().masked_fill(~allowed, float("-inf")), -1).to(torch.bfloat16)
        out[:, h] = p.double() @ v[h // rep, :n_slots].double()
    return out.view(T, nh * D)


def call(q, k, v, pos, n_slots, window, scale, nh, nkv, D):
    out, status = torch.full_like(q, float("nan")), torch.zeros(1, dtype=torch.int32, device=q.device)
    rc = _lib.load().cobalt_attn_prompt(q.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), out.data_ptr(), q.shape[0], nh, nkv,
                                        D, n_slots, k.shape[1], window, scale, 1, 0, status.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
    return rc, out, status


# one token, tiles of 128 rows minus / plus one, head groups that do not divide 128 rows, windows that end inside a
# tile, a prompt that continues a filled cache, scores far from zero (the maximum is what keeps exp in range)
@pytest.mark.parametrize("T,nh,nkv,D,ctx,window,start,gain", [
    (1, 4, 2, 64, 40, 0, 0, 1.0), (2, 8, 2, 128, 40, 0, 0, 1.0), (31, 8, 2, 128, 40, 0, 0, 1.0), (33, 8, 2, 64, 64, 0, 0, 1.0),
    (127, 1, 1, 128, 128, 0, 0, 1.0), (129, 1, 1, 64, 200, 0, 0, 1.0), (200, 6, 2, 128, 256, 0, 0, 1.0), (150, 7, 1, 64, 160, 64, 0, 1.0),
    (300, 5, 1, 128, 300, 100, 0, 1.0), (100, 8, 2, 128, 700, 128, 500, 1.0), (77, 16, 1, 128, 500, 0, 333, 1.0), (640, 4, 2, 128, 640, 0, 0, 12.0)])
def test_prompt_attention_matches_spec(T, nh, nkv, D, ctx, window, start, gain):
    g = torch.Generator(device="cuda").manual_seed(T + nh)
    n_slots = start + T
    q = (torch.randn(T, nh * D, generator=g, device="cuda") * gain).bfloat16()
    k, v = (torch.randn(nkv, ctx, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.arange(start, n_slots, device="cuda")
    rc, out, status = call(q, k, v, pos, n_slots, window, D ** -0.5, nh, nkv, D)
    ref = spec(q, k, v, pos, n_slots, window, D ** -0.5, nh, nkv, D)
    assert rc == 0 and int(status) == 0
    d = out.double() - ref
    assert float(d.norm() / ref.norm()) <= 2.0 ** -8
    assert float(d.abs().max()) <= 2.0 ** -6 * float(ref.abs().max())


@pytest.mark.parametrize("gain", [1.0, 4.0, 12.0])
def test_probabilities_are_those_of_an_fp32_softmax(gain):
    """Unit vectors as keys and values: the scores are exact and the result is the probabilities themselves.  An fp32 softmax is off by
    about 6e-8 (relative, on average) before the rounding to bf16, whose values lie 2^-8 to 2^-7 apart: about 2e-5 of them round
    to the other side.  torch's own fp32 softmax: 1.1e-5 at most; a softmax of twice that error exceeds the bound."""
    T, nh, D = 512, 16, 128
    g = torch.Generator(device="cuda").manual_seed(2)
    q = (torch.randn(T, nh * D, generator=g, device="cuda") * gain * D ** 0.5).bfloat16()
    eye = torch.eye(128, device="cuda").bfloat16().view(1, 128, 128).contiguous()
    pos = torch.full((T,), 127, device="cuda")
    rc, out, status = call(q, eye, eye, pos, 128, 0, D ** -0.5, nh, 1, D)
    scores = (q.float() * D ** -0.5).bfloat16().view(T, nh, 128)
    want = torch.softmax(scores.double(), -1).bfloat16().view(T, nh * 128)
    assert rc == 0 and int(status) == 0
    assert float((out != want).float().mean()) <= 5e-5


def test_slots_beyond_the_prompt_are_not_read():
    """What an earlier, longer prompt left in the cache (here: NaN) does not reach the result."""
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(50, 4 * 64, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(2, 300, 64, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.arange(50, device="cuda")
    _, want, _ = call(q, k, v, pos, 50, 0, 0.125, 4, 2, 64)
    k[:, 50:] = float("nan")
    v[:, 50:] = float("nan")
    _, got, _ = call(q, k, v, pos, 50, 0, 0.125, 4, 2, 64)
    assert torch.equal(got, want)


def test_unsupported_shapes_are_refused():
    q = torch.zeros(4, 4 * 96, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(2, 8, 96, dtype=torch.bfloat16, device="cuda")
    pos = torch.arange(4, device="cuda")
    assert call(q, k, k, pos, 4, 0, 0.1, 4, 2, 96)[0] == _lib.EUNSUPPORTED
    assert call(q, k, k, pos, 9, 0, 0.1, 4, 2, 96)[0] != 0                       # more slots than the cache has


@pytest.mark.parametrize("family,batch,T", [("llama", 3, 17), ("gemma", 8, 40), ("llama", 5, 150)])
def test_prompts_together_equal_prompts_alone(family, batch, T):
    """Prompts of several sequences through the layers at once: the logits and caches of each are those of its prompt alone."""
    from cobalt_b200 import SparseQuantConfig
    from cobalt_b200.decoder import build_random_decoder
    from oracle import model_oracle as MO
    if family == "gemma":
        cfg = MO.gemma3_config(hidden=512, layers=2, heads=8, kv_heads=2, head_dim=64, inter=1024, vocab=1008, sliding_window=16, pattern=2,
                               query_pre_attn_scalar=96, rope_scaling={"rope_type": "linear", "factor": 8.0})
    else:
        cfg = MO.llama_config(hidden=512, layers=2, heads=8, kv_heads=2, head_dim=64, inter=1024, vocab=1008)
    dec = build_random_decoder(cfg, SparseQuantConfig(4, 0.5, 0.5), T + 8, torch.device("cuda"), batch=batch, head_bits=4)
    ids = torch.randint(0, 1000, (batch, T), generator=torch.Generator().manual_seed(T))
    assert dec._prompts_at_once(T) == batch
    together = dec.prefill(ids)
    kc, vc = dec.k_cache.clone(), dec.v_cache.clone()
    pos = torch.arange(T, device="cuda")
    for b in range(batch):
        assert torch.equal(dec._forward(ids[b].cuda(), pos, T, seq=b)[0], together[b]), b
    assert torch.equal(dec.k_cache, kc) and torch.equal(dec.v_cache, vc)
    assert int(dec.prompt_status) == 0


def test_prompts_of_watched_modules_run_one_by_one():
    """A hook on o or down sees every prompt by itself, in the order of the sequences, also where prompts could run together."""
    from cobalt_b200 import SparseQuantConfig
    from cobalt_b200.decoder import build_random_decoder
    from oracle import model_oracle as MO
    cfg = MO.llama_config(hidden=512, layers=2, heads=8, kv_heads=2, head_dim=64, inter=1024, vocab=1008)
    dec = build_random_decoder(cfg, SparseQuantConfig(4, 0.5, 0.5), 48, torch.device("cuda"), batch=3, head_bits=4)
    ids = torch.randint(0, 1000, (3, 40), generator=torch.Generator().manual_seed(1))
    want, seen = dec.prefill(ids), []
    handle = dec.lin[(1, "mlp.down_proj")].register_forward_hook(lambda m, args, out: seen.append(tuple(args[0].shape)))
    assert torch.equal(dec.prefill(ids), want) and seen == [(40, 1024)] * 3
    handle.remove()
    assert torch.equal(dec.prefill(ids), want) and len(seen) == 3


def test_prompts_together_give_way_to_memory(monkeypatch):
    """Where the activations of all prompts at once do not fit, or the caller wants less, the prompts run in smaller parts: same bits."""
    from cobalt_b200 import SparseQuantConfig
    from cobalt_b200.decoder import build_random_decoder
    from oracle import model_oracle as MO
    cfg = MO.llama_config(hidden=512, layers=2, heads=8, kv_heads=2, head_dim=64, inter=1024, vocab=1008)
    dec = build_random_decoder(cfg, SparseQuantConfig(4, 0.5, 0.5), 48, torch.device("cuda"), batch=5, head_bits=4)
    ids = torch.randint(0, 1000, (5, 40), generator=torch.Generator().manual_seed(1))
    want = dec.prefill(ids)
    caches = dec.k_cache.clone(), dec.v_cache.clone()
    parts, inner = [], dec._forward_prompts

    def forward_prompts(ids, positions, first):
        parts.append(ids.shape[0])
        if dec.prompt_rows == 199:                            # no allocation is made to fail: the error alone matters
            raise torch.cuda.OutOfMemoryError("no room")
        return inner(ids, positions, first)

    monkeypatch.setattr(dec, "_forward_prompts", forward_prompts)
    for rows, expect in ((8192, [5]), (100, [2, 2, 1]), (0, []), (199, [4])):
        dec.prompt_rows = rows
        dec.k_cache.zero_()
        dec.v_cache.zero_()
        del parts[:]
        assert torch.equal(dec.prefill(ids), want) and parts == expect
        assert torch.equal(dec.k_cache, caches[0]) and torch.equal(dec.v_cache, caches[1])
