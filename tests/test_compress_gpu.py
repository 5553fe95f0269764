"""Compression on the GPU (csrc/compress_kernels.cuh) against the torch form of the same recipe on the CPU, which
test_format_cpu.py pins to the reference: masks, codes, scales, zero points and tile images are equal bit for bit."""
import pytest
import torch

from cobalt_b200 import CobaltSparseLinear
from cobalt_b200 import compress as C
from cobalt_b200 import format as F

pytestmark = pytest.mark.gpu


def bits_equal(a, b):
    return torch.equal(a.cpu().contiguous().view(torch.uint8), b.cpu().contiguous().view(torch.uint8))


def make(K, N, dtype, seed, special):
    g = torch.Generator().manual_seed(seed)
    W = (torch.randn(K, N, generator=g) * 0.02).to(dtype)
    norm = torch.randn(N, generator=g).abs() + 0.1
    if special == "ties":                                    # few distinct scores, dead rows, columns and groups, one sign only
        W = (W * 100).round() / 100
        W[::3] = 0
        W[:, ::5] = 0
        W[1::4] = W[1::4].abs()
        norm = norm.round() + 1
        norm[7] = 0
    if special == "inf":                                     # the maximum is not finite: non-finite scores count as zero
        W[0, 0] = float("inf")
        norm[3] = float("nan")
    return W, norm


@pytest.mark.parametrize("K,N,dtype,sparsity,beta,bits,special", [
    (1, 128, torch.float32, 0.5, 0.5, 4, ""), (17, 640, torch.bfloat16, 0.7, 0.5, 3, ""), (300, 1152, torch.float16, 0.3, 1.0, 2, ""),
    (4099, 256, torch.bfloat16, 0.6, 0.5, 3, ""), (64, 5376, torch.float32, 0.999, 0.0, 4, ""), (2, 512, torch.float32, 0.002, 0.5, 4, ""),
    (96, 1024, torch.float32, 0.5, 0.5, 4, "ties"), (96, 1024, torch.float32, 0.8, 0.5, 3, "inf"),
    (4096, 7936, torch.bfloat16, 0.5, 0.5, 4, "")])          # above 32 M elements: the bisected threshold
def test_compression_equals_the_cpu_form(K, N, dtype, sparsity, beta, bits, special):
    W, norm = make(K, N, dtype, K + N, special)
    keep = C.keep_mask(W, norm, sparsity, beta)
    got = C.keep_mask(W.cuda(), norm.cuda(), sparsity, beta)
    assert torch.equal(got.cpu(), keep)
    if special == "inf":
        W = torch.nan_to_num(W, posinf=1.0)                  # an infinite weight has no code
    q, sc, zr = C.quantize_survivors(W, keep, bits)
    q2, sc2, zr2 = C.quantize_survivors(W.cuda(), keep.cuda(), bits)
    assert torch.equal(q2.cpu(), q) and bits_equal(sc2, sc) and bits_equal(zr2, zr)
    if K * N < 10_000_000:
        img = F.pack_tiles(keep, q, sc, zr, bits)
        got = F.pack_tiles(keep.cuda(), q.cuda(), sc.cuda(), zr.cuda(), bits)
        assert torch.equal(got.blob.cpu(), img.blob) and got.meta() == img.meta()
        mod = CobaltSparseLinear._blank()
        mod._install(got, None, None, {})
        codes, k2 = mod.unpack()
        assert torch.equal(codes.cpu(), q) and torch.equal(k2.cpu(), keep)


@pytest.mark.parametrize("density", [0.0, 1.0])
def test_packing_of_empty_and_full_masks(density):
    g = torch.Generator().manual_seed(3)
    q = torch.randint(0, 8, (40, 1152), generator=g)
    keep = (torch.rand(40, 1152, generator=g) < density)
    sc, zr = torch.rand(40, 9, generator=g).half(), torch.randint(0, 8, (40, 9), generator=g).half()
    img = F.pack_tiles(keep, q, sc, zr, 3)
    got = F.pack_tiles(keep.cuda().float(), q.cuda(), sc.cuda(), zr.cuda(), 3)
    assert torch.equal(got.blob.cpu(), img.blob) and got.meta() == img.meta()
    if density:
        q[3, 5] = 8
        for form in (q, q.to(torch.uint8)):                  # a surviving code outside the grid is refused
            with pytest.raises(ValueError):
                F.pack_tiles(keep.cuda(), form.cuda(), sc.cuda(), zr.cuda(), 3)


def test_rounding_under_transforms_on_the_gpu():
    """Derivatives, ``vmap``, empty matrices and wide codes: the torch form, as on the CPU, not a kernel that is handed addresses."""
    g = torch.Generator().manual_seed(4)
    W, keep = torch.randn(6, 256, generator=g), torch.rand(6, 256, generator=g) > 0.5
    Wc, kc = W.cuda(), keep.cuda()
    q, s, z = C.quantize_survivors(W, keep, 4)
    leaf = Wc.clone().requires_grad_()
    q2, s2, z2 = C.quantize_survivors(leaf, kc, 4)
    assert s2.requires_grad and torch.equal(q2.cpu(), q) and bits_equal(s2.detach(), s)
    with torch.no_grad():
        assert not C.quantize_survivors(leaf, kc, 4)[1].requires_grad
    q3 = torch.vmap(lambda w, k: C.quantize_survivors(w, k, 4)[0])(Wc.view(2, 3, 256), kc.view(2, 3, 256))
    assert torch.equal(q3.view(6, 256).cpu(), q)
    assert [tuple(t.shape) for t in C.quantize_survivors(Wc[:0], kc[:0], 4)] == [(0, 256), (0, 2), (0, 2)]
    assert torch.equal(C.quantize_survivors(Wc, kc, 9)[0].cpu(), C.quantize_survivors(W, keep, 9)[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_damaged_weights_show_in_scale_and_zero_point(dtype):
    """A NaN or an infinity among the survivors of a group makes the scale (and zero point) what the torch form makes of it, so that the
    outputs show the damage; the same value at a pruned position changes nothing."""
    nan, inf = float("nan"), float("inf")
    W = (torch.randn(8, 384, generator=torch.Generator().manual_seed(9)) * 0.02).to(dtype)
    keep = torch.ones(8, 384, dtype=torch.bool)
    W[0, 5], W[1, 130], W[2, 383], W[3, 0] = nan, inf, -inf, nan
    keep[3, 0] = False                                       # pruned: harmless
    W[4, :128], W[5, 128:256], W[6, 256:] = inf, -inf, inf
    keep[6, 300] = False                                     # an all-infinite group with and without a pruned position
    W[7, 7], W[7, 8], W[7, 200], keep[7, 200] = inf, -inf, inf, False
    want = C.quantize_survivors(W, keep, 4)
    got = [t.cpu() for t in C.quantize_survivors(W.cuda(), keep.cuda(), 4)]
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a.isnan(), b.isnan()) and bits_equal(a.nan_to_num(nan=1.5), b.nan_to_num(nan=1.5))
    assert bool(got[1][0, 0].isnan()) and not bool(got[1][3, 0].isnan())
