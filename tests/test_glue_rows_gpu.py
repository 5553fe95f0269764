"""Element-wise kernels of a prompt and the greedy token against their plain forms (needs a B200)."""
import pytest
import torch

from cobalt_b200 import _lib

pytestmark = pytest.mark.gpu


def stream():
    return torch.cuda.current_stream().cuda_stream


def rand(*shape, seed=0, gain=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed + sum(shape)), device="cuda") * gain).bfloat16()


# one block per token (2^18 values on; with the norm 288 tokens and heads of 128 on) against the same tokens in calls of 16, which
# take the kernels that spread every head: same bits.  The first four stay below the line, the others lie on or beyond it.
@pytest.mark.parametrize("T,nh,nkv,D", [(32, 8, 2, 128), (77, 6, 2, 64), (48, 4, 1, 256), (33, 3, 3, 16), (288, 8, 2, 128), (300, 4, 1, 256),
                                        (331, 5, 1, 144), (2731, 3, 3, 16), (700, 6, 2, 64)])
@pytest.mark.parametrize("norm", [False, True])
def test_rope_of_many_tokens_equals_few(T, nh, nkv, D, norm):
    lib, ctx = _lib.load(), T + 7
    k, v, pos = rand(T, nkv * D, seed=1), rand(T, nkv * D, seed=2), torch.arange(3, 3 + T, device="cuda")
    pos[5], pos[6] = -1, ctx                                     # outside the cache: not stored
    inv = 1.0 / (1e4 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    keep = [rand(D, seed=s, gain=0.1) for s in (3, 4)]           # owns the norm weights
    w = [t.data_ptr() if norm else None for t in keep]
    res = []
    for step in (T, 16):
        q = rand(T, nh * D, seed=5)
        kc, vc = (torch.zeros(nkv, ctx, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        for t in range(0, T, step):
            n = min(step, T - t)
            rc = lib.cobalt_rope_kv(q[t:].data_ptr(), k[t:].data_ptr(), v[t:].data_ptr(), pos[t:].data_ptr(), inv.data_ptr(), kc.data_ptr(),
                                    vc.data_ptr(), n, nh, nkv, D, ctx, w[0], w[1], 1e-6, 0, stream())
            assert rc == 0
        res.append((q, kc, vc))
    for a, b in zip(*res):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("n", [8, 4096, 100003 * 8, 1000])
@pytest.mark.parametrize("act", [0, 1])
def test_gated_activation_in_chunks_equals_value_by_value(n, act):
    lib = _lib.load()
    g, u = rand(n + 8, seed=1, gain=3.0), rand(n + 8, seed=2)
    outs = []
    for shift in (0, 1):                                         # an odd start takes the value-by-value kernel
        a, b = torch.empty(n + 8, dtype=torch.bfloat16, device="cuda"), torch.empty(n + 8, dtype=torch.bfloat16, device="cuda")
        out = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")
        a[shift:shift + n], b[shift:shift + n] = g[:n], u[:n]
        assert lib.cobalt_swiglu(a[shift:].data_ptr(), b[shift:].data_ptr(), out[shift:].data_ptr(), n, act, stream()) == 0
        outs.append(out[shift:shift + n].clone())
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))


@pytest.mark.parametrize("n", [8000, 8001])
@pytest.mark.parametrize("target", [0, 1])
def test_gated_activation_in_place(n, target):
    """The result may take the place of either input, whichever kernel runs."""
    lib = _lib.load()
    g, u, out = rand(n, seed=1, gain=3.0), rand(n, seed=2), torch.empty(n, dtype=torch.bfloat16, device="cuda")
    assert lib.cobalt_swiglu(g.data_ptr(), u.data_ptr(), out.data_ptr(), n, 0, stream()) == 0
    assert lib.cobalt_swiglu(g.data_ptr(), u.data_ptr(), (g, u)[target].data_ptr(), n, 0, stream()) == 0
    assert torch.equal((g, u)[target], out)


@pytest.mark.parametrize("rows,V", [(1, 1), (1, 7), (3, 8), (2, 4095), (1, 32000), (16, 32000), (2, 262144), (5, 1001)])
def test_argmax_matches_torch(rows, V):
    lib = _lib.load()
    x = rand(rows, V, seed=rows)
    x[:, V // 2:] = x[:, :V - V // 2].flip(1) if V > 1 else x[:, V // 2:]        # every value twice: the first one counts
    for case in range(4):
        y = x.clone()
        if case == 1:
            y[:, V // 3] = float("nan")
            y[:, -1] = float("nan")
        elif case == 2:
            y.fill_(float("-inf"))
        elif case == 3:
            y.fill_(-0.0)
            y[:, V // 2] = 0.0                                   # zeros of either sign are equal
        out = torch.full((rows,), -1, dtype=torch.long, device="cuda")
        assert lib.cobalt_argmax(y.data_ptr(), y.stride(0), rows, V, out.data_ptr(), stream()) == 0
        f = y.float()
        best = f.max(dim=1, keepdim=True).values
        hit = torch.isnan(f) if case == 1 else f == best
        want = torch.where(hit, torch.arange(V, device="cuda")[None], V).min(dim=1).values
        assert torch.equal(out, want), case


@pytest.mark.parametrize("H", [256, 4096, 4352, 8192, 8448, 16384])
@pytest.mark.parametrize("flavor", [0, 1])
def test_norm_of_every_row_length_class(H, flavor):
    """One, two and four 16-byte chunks per thread (their first and last row lengths) against fp64: one bf16 spacing."""
    lib, T = _lib.load(), 5
    h, d, w = rand(T, H, seed=1), rand(T, H, seed=2), rand(H, seed=3, gain=0.2)
    ho, y = torch.empty_like(h), torch.empty_like(h)
    assert lib.cobalt_add_rmsnorm(h.data_ptr(), d.data_ptr(), w.data_ptr(), ho.data_ptr(), y.data_ptr(), T, H, 1e-5, flavor, None, stream()) == 0
    assert torch.equal(ho, (h.float() + d.float()).bfloat16())
    x = ho.double()
    n = x * torch.rsqrt((x * x).mean(1, keepdim=True) + 1e-5)
    ref = n.to(torch.bfloat16).double() * w.double() if flavor == 0 else n * (1.0 + w.double())
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -7 + (n.abs() * w.abs().double() * 2.0 ** -8 if flavor == 0 else 0.0)).all())
