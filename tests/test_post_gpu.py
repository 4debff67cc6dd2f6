"""Parity of the tonemapping and NLM kernels with the reference and the oracle."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_tonemap_matches_reference(ctx, kind):
    """Same per-pixel arithmetic; the log-average is summed in double on the GPU where the
    reference adds floats one by one, so outputs agree to a few ulps of the key."""
    g = np.load(os.path.join(GOLDEN, "tonemap_ref.npz"))
    out, _, _, _ = ctx.tonemap(g["img"], kind, srgb=False)
    np.testing.assert_allclose(out, g[f"tm{kind}"], rtol=2e-5, atol=1e-7)


def test_srgb8_matches_reference_capture_png(ctx):
    """PathTracer::Capture: ACES, clamp, the reference OETF, x*255+0.5 -- within 1 LSB."""
    g = np.load(os.path.join(GOLDEN, "tonemap_ref.npz"))
    _, s8, _, _ = ctx.tonemap(g["img"], 2, srgb=True, ref_oetf=True)
    d = np.abs(s8.astype(int) - g["srgb_aces_ref"].astype(int))
    assert d.max() <= 1 and (d > 0).mean() < 0.01


def test_tonemap_large_image_matches_oracle(ctx, oracle):
    rng = np.random.default_rng(8)
    img = np.exp(rng.normal(0.0, 2.0, size=(540, 960, 3))).astype(np.float32)
    for kind in (0, 1, 2):
        out, _, ave, mx = ctx.tonemap(img, kind, srgb=False)
        o, oave, omx = oracle.tonemap(kind, img)
        assert mx == omx
        assert abs(ave / oave - 1) < 1e-4
        np.testing.assert_allclose(out, o, rtol=2e-4, atol=1e-6)


def test_nlm_ref_matches_reference(ctx):
    g = np.load(os.path.join(GOLDEN, "nlm_ref.npz"))
    out = ctx.nlm_ref(g["rgba"], float(g["coeff"]))
    np.testing.assert_allclose(out, g["out"], rtol=1e-5, atol=1e-6)


def test_nlm_ref_larger_image_matches_oracle(ctx, oracle):
    rng = np.random.default_rng(9)
    rgba = rng.random((70, 90, 4), dtype=np.float32)
    out = ctx.nlm_ref(rgba, 0.15)
    np.testing.assert_allclose(out, oracle.nlm_ref(rgba, 0.15), rtol=1e-5, atol=1e-6)


def test_variance_nlm_matches_oracle(ctx, oracle):
    rng = np.random.default_rng(10)
    clean = np.tile(np.linspace(0.1, 1.0, 64, dtype=np.float32)[None, :, None], (48, 1, 3))
    var = np.full_like(clean, 0.01)
    noisy = clean + rng.normal(0, 0.1, clean.shape).astype(np.float32)
    out = ctx.nlm(noisy, var, search_r=10, patch_r=3, k=0.45)
    ref = oracle.nlm_var(noisy, var, 10, 3, 0.45)
    np.testing.assert_allclose(out, ref, rtol=1e-4, atol=1e-5)
    assert np.mean((out - clean) ** 2) < 0.5 * np.mean((noisy - clean) ** 2)


@pytest.mark.parametrize("ref_oetf", [True, False])
def test_srgb8_equals_the_exact_oetf_of_the_linear_output(ctx, ref_oetf):
    """The sRGB8 encode takes the power from the hardware approximation and falls back to
    powf only near a code boundary: every code must equal the all-powf formula applied to
    the linear output (torch's CUDA pow is powf; the same IEEE operations in the same
    order), here on 12.6M values covering every code the curve reaches (the reference's OETF
    tops out at 1.055^(1/2.4) - 0.055, code 247)."""
    import torch
    rng = np.random.default_rng(21)
    img = np.exp(rng.normal(0.0, 2.0, size=(1024, 4096, 3))).astype(np.float32)
    out, s8, _, _ = ctx.tonemap(img, 0, srgb=True, ref_oetf=ref_oetf)
    y = torch.from_numpy(out).cuda().clamp(0.0, 1.0)
    e = torch.tensor(np.float32(1.0) / np.float32(2.4), device="cuda")
    lin = y <= np.float32(0.0031308)
    if ref_oetf:
        v = torch.pow(y * np.float32(1.055), e) - np.float32(0.055)
    else:
        v = torch.pow(y, e) * np.float32(1.055) - np.float32(0.055)
    v = torch.where(lin, y * np.float32(12.92), v)
    want = (v * np.float32(255.0) + np.float32(0.5)).to(torch.uint8).cpu().numpy()
    assert len(np.unique(want)) == (248 if ref_oetf else 256)
    np.testing.assert_array_equal(s8, want)


# Tiles of the column-walking NLM kernels are 16 rows by 32 - 2P columns (28 for the reference's
# filter): images smaller than a tile, exactly one, and one pixel more each way; search radii
# on both sides of the staged pitches (10, 32), patch radii inside and outside 1..3.
# Tolerance: a weight's exponent is a mean of up to 147 terms, its FP32 error some 20 ulp, and
# matters up to about 20 (e^-20): 20 * 20 * 2^-24 = 2.4e-5 relative, taken as 1e-4.
@pytest.mark.parametrize("h,w", [(5, 7), (16, 26), (17, 27), (33, 61)])
@pytest.mark.parametrize("search_r,patch_r", [(2, 1), (5, 2), (10, 3), (11, 3), (0, 1), (3, 0), (2, 4)])
def test_variance_nlm_at_tile_edges(ctx, oracle, h, w, search_r, patch_r):
    rng = np.random.default_rng(1000 * h + 10 * search_r + patch_r)
    img = rng.random((h, w, 3), dtype=np.float32)
    var = (0.02 * rng.random((h, w, 3), dtype=np.float32) + 1e-3).astype(np.float32)
    out = ctx.nlm(img, var, search_r=search_r, patch_r=patch_r, k=0.6)
    np.testing.assert_allclose(out, oracle.nlm_var(img, var, search_r, patch_r, 0.6), rtol=1e-4, atol=1e-5)


# The exponent here is at most about 10 with 25 non-negative terms: 10 * 10 * 2^-24 = 6e-6.
@pytest.mark.parametrize("h,w", [(3, 5), (16, 28), (17, 29), (40, 57)])
def test_nlm_ref_at_tile_edges(ctx, oracle, h, w):
    rgba = np.random.default_rng(h).random((h, w, 4), dtype=np.float32)
    np.testing.assert_allclose(ctx.nlm_ref(rgba, 0.6), oracle.nlm_ref(rgba, 0.6), rtol=1e-5, atol=1e-6)


def _tonemap_device(ctx, img, out, s8, kind):
    import ctypes as C
    import salty_gb300
    h, w = img.shape[:2]
    ave, mx = C.c_float(), C.c_float()
    ctx.check(salty_gb300.lib().salty_tonemap(ctx.h, kind, w, h, img.data_ptr(), out.data_ptr() if out is not None else None,
                                              s8.data_ptr() if s8 is not None else None, 1, C.byref(ave), C.byref(mx)), "tonemap")
    return np.float32(ave.value), np.float32(mx.value)


def test_tonemap_scale_is_the_hosts(ctx):
    """The curve's scale is key / expf(mean) in the host's arithmetic, bit for bit, whatever the
    device's own exponential rounds to: 4,000 one-pixel images, Reinhard restated in FP32."""
    import torch
    f = np.float32
    rng = np.random.default_rng(31)
    px = np.exp(rng.normal(0.0, 3.0, size=(4000, 1, 1, 3))).astype(f)
    imgs, out = torch.from_numpy(px).cuda(), torch.empty((1, 1, 3), device="cuda")
    for k in range(len(px)):
        ave, mx = _tonemap_device(ctx, imgs[k], out, None, 0)
        c = f(0.18) / ave
        m2 = (mx * c) * (mx * c)
        x = px[k] * c
        y = (x * (f(1.0) + x / m2)) / (f(1.0) + x)
        np.testing.assert_array_equal(out.cpu().numpy(), y)


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("shape", [(1, 1), (1, 3), (1, 4), (5, 1), (37, 29), (33, 1024), (700, 1601)])
def test_tonemap_layouts_agree(ctx, shape, kind):
    """Groups of four pixels, single values, remainders, arrays off the 16-byte boundary and
    tonemapping in place give the same bits; the scale is the same for any order of the sum
    here (to FP32), since it is added in FP64."""
    import torch
    h, w = shape
    n = h * w * 3
    rng = np.random.default_rng(h * w)
    img = torch.from_numpy(np.exp(rng.normal(0.0, 2.0, size=n)).astype(np.float32)).cuda()
    img[0] = 0.0
    got = []
    for off in (0, 1):
        a = torch.empty(n + 4, device="cuda")[off:off + n]
        a.copy_(img)
        o = torch.full((n + 4,), -1.0, device="cuda")
        s = torch.zeros(n + 8, dtype=torch.uint8, device="cuda")
        _tonemap_device(ctx, a.view(h, w, 3), o[off:], s[off:], kind)
        assert (o[off + n:] == -1.0).all() and (s[off + n:] == 0).all()
        got.append((o[off:off + n].cpu().numpy(), s[off:off + n].cpu().numpy()))
        _tonemap_device(ctx, a.view(h, w, 3), a, None, kind)
        got.append((a.cpu().numpy(), got[-1][1]))
    for o, s in got[1:]:
        np.testing.assert_array_equal(o, got[0][0])
        np.testing.assert_array_equal(s, got[0][1])


# Enough tiles for the taller column walks (12 rows; the sizes above take 8), with one row, one
# column and a full tile over.
@pytest.mark.parametrize("h,w,patch_r", [(397, 157, 3), (396, 156, 3), (385, 169, 2), (409, 151, 1)])
def test_variance_nlm_on_tall_tiles(ctx, oracle, h, w, patch_r):
    rng = np.random.default_rng(h + patch_r)
    img = rng.random((h, w, 3), dtype=np.float32)
    var = (0.02 * rng.random((h, w, 3))).astype(np.float32)
    out = ctx.nlm(img, var, search_r=2, patch_r=patch_r, k=0.6)
    np.testing.assert_allclose(out, oracle.nlm_var(img, var, 2, patch_r, 0.6), rtol=1e-4, atol=1e-5)


# The default window, the smallest and the largest radius of the wide tile's kernel, on 12-row
# tiles (more tiles than SMs), against the direct sums in 64 bits.  Bounds as above.
@pytest.mark.parametrize("search_r,patch_r", [(10, 3), (10, 1), (11, 3), (11, 2), (32, 3), (32, 1)])
def test_variance_nlm_search_radii_on_tall_tiles(ctx, search_r, patch_r):
    import torch
    import torch.nn.functional as F
    h, w, k = 397, 157, 0.6
    rng = np.random.default_rng(100 * search_r + patch_r)
    img = rng.random((h, w, 3), dtype=np.float32)
    var = (0.02 * rng.random((h, w, 3)) + 1e-3).astype(np.float32)
    out = ctx.nlm(img, var, search_r=search_r, patch_r=patch_r, k=k)
    R, P = search_r, patch_r
    pad = lambda a: F.pad(torch.from_numpy(a).cuda().double().permute(2, 0, 1)[None], (R + P,) * 4, mode="replicate")[0]
    I, V = pad(img), pad(var)
    cut = lambda a, dy, dx, e: a[:, R + P + dy - e:R + P + dy + h + e, R + P + dx - e:R + P + dx + w + e]
    a, va = cut(I, 0, 0, P), cut(V, 0, 0, P)
    acc, tot = torch.zeros((3, h, w), dtype=torch.float64, device="cuda"), torch.zeros((h, w), dtype=torch.float64, device="cuda")
    for dy in range(-R, R + 1):
        for dx in range(-R, R + 1):
            b, vb = cut(I, dy, dx, P), cut(V, dy, dx, P)
            d = (((a - b) ** 2 - (va + torch.minimum(va, vb))) / (1e-10 + k * k * (va + vb))).sum(0)
            wt = torch.exp(-(F.avg_pool2d(d[None, None], 2 * P + 1, stride=1)[0, 0] / 3.0).clamp_min(0.0))
            acc += wt * cut(I, dy, dx, 0)
            tot += wt
    np.testing.assert_allclose(out, (acc / tot).permute(1, 2, 0).cpu().numpy(), rtol=1e-4, atol=1e-5)


def _aces_fp32(x):
    """ACESFilm (src/s3d_tonemapper.cpp:117-130), every operation rounded to FP32."""
    f = np.float32
    a, b, c, d, e, g, k = f(2.51), f(0.03), f(2.43), f(0.59), f(0.14), f(0.665406), f(12.0)
    with np.errstate(all="ignore"):
        y = (x * (a * x * g / k + b)) / (x * g / k * (c * x * g + d) + e)
    return np.where(y < 0, f(0), np.where(y > 1, f(1), y))


# ACES bit for bit against the FP32 restatement with true quotients: every mantissa of a binade,
# and scaled values on both sides of the range in which a twelfth is taken by a corrected product
# (2^-90 from a bright channel beside tiny ones, 2^90 from a few bright pixels among black ones).
@pytest.mark.parametrize("values", ["mantissas", "tiny", "huge"])
def test_aces_equals_the_fp32_restatement(ctx, values):
    import torch
    f = np.float32
    if values == "mantissas":
        img = (np.arange(1 << 23, dtype=np.uint32) + np.uint32(0x3F800000)).view(f)[:3 * ((1 << 23) // 3)].reshape(1, -1, 3)
    elif values == "tiny":
        e = np.linspace(-100.0, -80.0, 3000)
        img = np.stack([np.ones_like(e), 2.0 ** e, 2.0 ** -e[::-1] * 2.0 ** -180], 1).astype(f)[None]
    else:
        img = np.zeros((100, 1000, 3), f)
        img[0, :, :] = (2.0 ** np.linspace(68.0, 84.0, 3000)).reshape(1000, 3)
    d = torch.from_numpy(np.ascontiguousarray(img)).cuda()
    out = torch.empty_like(d)
    ave, _ = _tonemap_device(ctx, d, out, None, 2)
    x = img * (f(0.27) / ave)
    if values != "mantissas":
        m = np.abs(x[x != 0])
        assert np.count_nonzero((m > 2.0 ** 88) & (m < 2.0 ** 92) | (m > 2.0 ** -92) & (m < 2.0 ** -88)) > 300
    np.testing.assert_array_equal(out.cpu().numpy(), _aces_fp32(x))


# No tonemap of device arrays allocates device memory, the first of a context included.  An
# allocation of 19 KB hides in the driver's 2 MB blocks; those of 256 contexts do not.
def test_first_tonemap_allocates_nothing(salty_lib):
    import torch
    import salty_gb300
    img = torch.rand((33, 47, 3), device="cuda")
    out = torch.empty_like(img)
    many = [salty_gb300.Context(0) for _ in range(257)]
    try:
        _tonemap_device(many[0], img, out, None, 0)  # loads the kernels
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for c in many[1:]:
            _tonemap_device(c, img, out, None, 0)
        assert torch.cuda.mem_get_info()[0] == free
    finally:
        for c in many:
            c.close()


# An image of more rows than a grid's second dimension has tiles for, against its own bands.
def test_variance_nlm_of_a_very_tall_image(ctx):
    import torch
    h, w, R, P = 800000, 3, 1, 1
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    img = torch.rand((h, w, 3), device="cuda", generator=g)
    var = 0.02 * torch.rand((h, w, 3), device="cuda", generator=g)
    out, band = torch.empty_like(img), torch.empty((600, w, 3), device="cuda")
    ctx.nlm(img, var, R, P, out=out)
    for y in (0, 400000, h - 600):
        ctx.nlm(img[y:y + 600].contiguous(), var[y:y + 600].contiguous(), R, P, out=band)
        lo, hi = (0 if y == 0 else 2), (600 if y == h - 600 else 598)  # rows that see the band alone
        torch.testing.assert_close(out[y + lo:y + hi], band[lo:hi], rtol=1e-5, atol=1e-6)
