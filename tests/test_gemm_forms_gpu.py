"""Both forms of the prompt GEMM (single CTAs and CTA pairs), its split columns and its fused launch (needs a B200).

Reference: the fp64 product with ``dequantize()`` (bit-exact against the oracle in test_kernels_gpu.py).  Tolerance, per element: one
bf16 spacing (2^-7 of the magnitude at most) for every rounding - of the product, and with a bias of the sum with it, whose
magnitudes differ when the bias cancels the product - plus 1e-4 of the largest value for fp32 sums in another order (5e-5
seen over 14336 columns).
"""
import re

import pytest
import torch

from cobalt_b200 import CobaltSparseLinear
from cobalt_b200.compress import quantize_survivors
from cobalt_b200.linear import FusedProjections

pytestmark = pytest.mark.gpu


def module(K, N, bits, sparsity=0.5, scale2=None, bias=False, seed=0, zero_shift=0.0):
    g = torch.Generator(device="cuda").manual_seed(seed + K + N)
    W = (torch.randn(K, N, generator=g, device="cuda") * 0.02).half().float()
    keep = torch.rand(K, N, generator=g, device="cuda") > sparsity
    q, s, z = quantize_survivors(W, keep, bits)
    z = z.clone()
    z[::3, ::2] += zero_shift                                    # 0.5: zero points off the integer grid
    b = (torch.randn(K, generator=g, device="cuda") * 0.1).bfloat16() if bias else None
    return CobaltSparseLinear(q, s, z, keep, scale2, b, {"nbits": bits})


def check(m, x, y):
    exact = x.double() @ m.dequantize().double().t()
    bound = exact.abs() * 2.0 ** -7 + exact.abs().max() * 1e-4
    if m.bias is not None:
        exact = exact.to(torch.bfloat16).double() + m.bias.double()
        bound = bound + exact.abs() * 2.0 ** -7
    d = (y.double() - exact).abs()
    assert m.device_status() == 0
    assert bool((d <= bound).all()), float((d - bound).max())
    assert float(d.norm() / exact.norm()) <= 2.0 ** -8


def tokens(M, N, seed=1):
    return torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(seed + M), device="cuda").bfloat16()


# rows: less than a tile, tiles minus / plus 16 rows, an odd number of tiles (a pair with an empty half); columns: one group, a tile
# plus one group, ragged tiles; tokens: 17, accumulators minus / plus one, a ragged last tile
@pytest.mark.parametrize("K,N,bits", [(16, 128, 4), (100, 640, 3), (144, 512, 2), (384, 1152, 4), (1000, 4096, 3), (4096, 2048, 4)])
@pytest.mark.parametrize("M", [17, 32, 255, 257, 513, 1500])
def test_forms_match_fp64(K, N, bits, M):
    m, x = module(K, N, bits, bias=K == 384), tokens(M, N)
    check(m, x, m(x))
    assert torch.equal(m(x), m(x))                                # split sums are added in a fixed order


@pytest.mark.parametrize("M", [3, 16, 40, 300, 1100])
@pytest.mark.parametrize("bits", [2, 3, 4])
def test_column_scale(M, bits):
    s2 = torch.exp(torch.randn(1152, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda") * 0.25).half()
    m, x = module(272, 1152, bits, scale2=s2, bias=True), tokens(M, 1152)
    check(m, x, m(x))


@pytest.mark.parametrize("M", [1, 16, 40, 600])
@pytest.mark.parametrize("sparsity", [0.5, -1.0])
def test_column_scale_at_any_address(M, sparsity):
    """A scale off the 16-byte boundary is read one value at a time: the same arithmetic, hence the same bits."""
    buf = torch.exp(torch.randn(1153 + 8, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda") * 0.25).half()
    m, x = module(272, 1152, 4, sparsity=sparsity, scale2=buf[1:1153]), tokens(M, 1152)
    assert m.scale2.data_ptr() % 16 == 0                          # the module keeps an aligned copy of the slice
    want = m(x)
    m.scale2 = buf[1:1153]                                        # a caller's own pointer, as through the C ABI
    assert m.scale2.data_ptr() % 16 == 2
    check(m, x, want)
    assert torch.equal(m(x), want)


@pytest.mark.parametrize("M", [2, 40, 600])
@pytest.mark.parametrize("scaled", [False, True])
def test_zero_points_off_the_grid(M, scaled):
    s2 = (torch.rand(640, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda") + 0.5).half() if scaled else None
    m, x = module(272, 640, 4, scale2=s2, zero_shift=0.5), tokens(M, 640)
    check(m, x, m(x))


@pytest.mark.parametrize("M", [2, 40, 600])
def test_infinite_column_scale_leaves_pruned_positions_alone(M):
    """A column whose scale is infinite only reaches the rows that keep it."""
    s2 = torch.ones(640, device="cuda").half()
    s2[37], s2[300] = float("inf"), 0.5
    m, x = module(64, 640, 3, scale2=s2), tokens(M, 640)
    _, keep = m.unpack()
    y = m(x).float()
    assert bool(torch.isfinite(y[:, ~keep[:, 37]]).all()) and int((~keep[:, 37]).sum()) > 0


@pytest.mark.parametrize("M", [17, 90, 400, 1500])
def test_fused_launch(M):
    mods = [module(K, 1024, 4, seed=i) for i, K in enumerate((512, 128, 200))]
    x = tokens(M, 1024)
    fused = FusedProjections(mods)
    for m, y in zip(mods, fused(x)):
        check(m, x, y)
    assert fused._scratch is not None and fused.device_status() == 0        # the launch's own word: the modules were not called


def launched_form(call):
    """Template arguments of the prompt GEMM's kernel in one call: <bits, CTA pairs, column scale>."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    (form,) = {re.search("<(.*?)>", e.key).group(1) for e in prof.key_averages() if "gemm_tcgen05_kernel" in e.key}
    return form


@pytest.mark.parametrize("K,N,T,n", [(512, 512, 150, 5), (2048, 1024, 200, 8), (6144, 1024, 100, 8), (1024, 1024, 40, 8)])
def test_sums_do_not_depend_on_the_form(K, N, T, n):
    """``sum_tokens``: the rows of n prompts in one launch get the bits that each prompt gets alone, also where one launch takes CTA
    pairs and the other single CTAs (all but the last case)."""
    fused, x = FusedProjections([module(K, N, 4)]), tokens(n * T, N)
    first = x[:T].contiguous()
    alone = torch.cat([fused(x[i * T:(i + 1) * T].contiguous())[0] for i in range(n)])
    assert torch.equal(fused(x, T)[0], alone)
    assert (launched_form(lambda: fused(x, T)) != launched_form(lambda: fused(first))) == (K != 1024)


@pytest.mark.parametrize("how", ["hook", "global hook", "replaced", "subclass"])
def test_fused_launch_does_not_pass_a_module_by(how):
    """Above 16 tokens whatever a call of a module runs is run, as before there was a launch for several modules."""
    class Sub(CobaltSparseLinear):
        def forward(self, x):
            seen.append(x.shape[0])
            return super().forward(x)

    seen = []
    mods = [module(128, 640, 4, seed=i) for i in range(2)]
    fused, x = FusedProjections(mods), tokens(40, 640)
    want = fused(x)
    assert not seen
    note, handle = lambda m, args, *out: seen.append(args[0].shape[0]), None
    if how == "hook":
        handle = mods[1].register_forward_hook(note)
    elif how == "global hook":
        handle = torch.nn.modules.module.register_module_forward_pre_hook(note)
    elif how == "replaced":
        inner = mods[1].forward
        mods[1].forward = lambda x: (seen.append(x.shape[0]), inner(x))[1]
    else:
        mods[1].__class__ = Sub
    try:
        got = fused(x)
    finally:
        if handle is not None:
            handle.remove()
    assert seen == [40] * (2 if how == "global hook" else 1)
    for a, b in zip(got, want):
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 2.0 ** -8


@pytest.mark.parametrize("K,N,bits", [(64, 512, 4), (80, 1152, 4), (512, 2048, 3), (48, 640, 2), (2400, 1536, 4)])
@pytest.mark.parametrize("M", [1, 5, 8, 16])
def test_matrix_without_pruned_positions(K, N, bits, M):
    """Full tiles copied row by row; a ragged last column tile, and rows beyond K (whose tiles are not full), are not."""
    m, x = module(K, N, bits, sparsity=-1.0), tokens(M, N)
    assert m._img_meta["nnz"] == K * N
    check(m, x, m(x))


@pytest.mark.parametrize("missing", [1, 31, 40])
def test_almost_full_tile_in_a_launch_for_full_ones(missing):
    """A tile a few codes short of full can have the bytes of a full one: the kernel must notice even if the survivor count of the
    descriptor says that nothing is pruned."""
    g = torch.Generator(device="cuda").manual_seed(missing)
    W = torch.randn(48, 1024, generator=g, device="cuda") * 0.02
    keep = torch.ones(48, 1024, dtype=torch.bool, device="cuda")
    keep[19, 300:300 + missing] = False
    q, s, z = quantize_survivors(W, keep, 4)
    m, x = CobaltSparseLinear(q, s, z, keep, None, None, {"nbits": 4}), tokens(4, 1024)
    W64 = m.dequantize()
    m._img_meta["nnz"] = 48 * 1024
    m._desc = None
    exact = x.double() @ W64.double().t()
    assert bool(((m(x).double() - exact).abs() <= exact.abs() * 2.0 ** -7 + exact.abs().max() * 1e-4).all())


def test_modules_saved_whole_before_launches_were_kept():
    """Objects of an earlier version, restored with the attributes they had then, run and report their status."""
    import io
    m, x = module(128, 640, 4), tokens(40, 640)
    want = m(x), m(x[:3])
    old = module(128, 640, 4)
    for name in ("_launch",):
        del old.__dict__[name]
    buf = io.BytesIO()
    torch.save(old, buf)
    buf.seek(0)
    again = torch.load(buf, weights_only=False)
    assert torch.equal(again(x), want[0]) and torch.equal(again(x[:3]), want[1]) and again.device_status() == 0
    fused = FusedProjections.__new__(FusedProjections)
    fused.__dict__.update(mods=[again], _scratch=None, _arrays=None)
    assert fused.device_status() == 0
    assert torch.equal(fused(x[:3])[0], want[1]) and torch.equal(fused(x)[0], want[0]) and fused.device_status() == 0


def test_very_many_tokens():
    """More token tiles of the single form than a grid has rows: the pair form takes them.  (4.3 GB of activations.)"""
    M, N, K = 65535 * 256 + 300, 128, 16
    m, few = module(K, N, 4), tokens(300, N)
    x = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    x[:300], x[-300:] = few, few
    y = m(x)
    assert m.device_status() == 0 and y.shape == (M, K)
    check(m, few, y[:300])
    check(m, few, y[-300:])
    assert not bool(y[300:-300].any())
