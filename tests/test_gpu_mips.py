"""GPU mip generation (crngpu_generate_mipmaps) against the reference's own mip levels (golden
fixtures from crnlib's generate_mipmaps resampler) and, at sizes beyond the fixtures, against the
oracle (the CPU restatement pinned to those fixtures): bit-exact, host and device buffers."""
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def cg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import crunch2_gb300
    crunch2_gb300.lib()
    return crunch2_gb300


def cases():
    with open(os.path.join(HERE, "golden", "mips.json")) as fh:
        return json.load(fh)


@pytest.mark.parametrize("name", sorted(cases().keys()))
def test_gpu_mips_match_reference(cg, name):
    m = cases()[name]
    z = np.load(os.path.join(HERE, "golden", "mips.npz"))
    base = z[name + "_base"]
    levels = cg.generate_mipmaps(base, m["filter"], m["filter_scale"], m["srgb"], m["wrap"], alpha=m["comps"] == 4)
    assert len(levels) == m["levels"]
    assert np.array_equal(levels[0], base)
    got = np.concatenate([l.reshape(-1) for l in levels[1:]])
    ref = z[name + "_levels"]
    assert np.array_equal(got, ref), (name, int((got != ref).sum()), got.size)


@pytest.mark.parametrize("filt,srgb,wrap", [("kaiser", True, False), ("lanczos4", False, True), ("box", True, True)])
def test_gpu_mips_match_oracle_device_buffers(cg, filt, srgb, wrap):
    from oracle import mip_oracle
    from crunch2_gb300 import texgen
    img = texgen.colour_texture(203, 130, 77, with_alpha_noise=True)
    want = mip_oracle.generate_mipmaps(img, filt, 0.9, srgb, wrap, alpha=True, levels=4)
    got = cg.generate_mipmaps(torch.from_numpy(img).cuda(), filt, 0.9, srgb, wrap, alpha=True, levels=4)
    for l, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a.cpu().numpy(), b), (filt, l)


# sides below the eight rows / columns and the pairs a warp takes, windows over one staged chunk
# (320 positions in rows, 128 in columns) by size and by filter scale, levels of at most 16 and of
# more samples, power-of-two and other scales, wrap far outside the image
@pytest.mark.parametrize("w,h,filt,scale,wrap,alpha", [
    (1, 1, "kaiser", 0.9, False, True), (1, 37, "kaiser", 0.9, True, True), (41, 2, "tent", 1.2, False, False),
    (9, 7, "box", 0.9, True, True), (66, 34, "mitchell", 0.9, False, True), (700, 9, "lanczos4", 1.0, True, True),
    (11, 530, "kaiser", 0.9, False, False), (128, 64, "kaiser", 9.0, True, True), (530, 133, "lanczos4", 3.0, False, True),
])
def test_gpu_mips_edges_match_oracle(cg, w, h, filt, scale, wrap, alpha):
    from oracle import mip_oracle
    from crunch2_gb300 import texgen
    img = texgen.colour_texture(w, h, w * 7 + h, with_alpha_noise=True)
    levels = max(w, h).bit_length()
    want = mip_oracle.generate_mipmaps(img, filt, scale, True, wrap, alpha=alpha, levels=levels)
    got = cg.generate_mipmaps(torch.from_numpy(img).cuda(), filt, scale, True, wrap, alpha=alpha)
    assert len(got) == levels
    for l in range(1, levels):
        assert np.array_equal(got[l].cpu().numpy(), want[l] if len(want) == levels else want[l - 1]), l


# images of at least 2^21 texels, whose small levels share their row jobs: sides that are not powers of two,
# runs of samples cut unevenly between jobs, windows over many chunks, wrap
@pytest.mark.parametrize("w,h,filt,scale,wrap", [
    (8209, 257, "kaiser", 0.9, False), (1030, 2053, "lanczos4", 1.3, True), (259, 8101, "box", 0.9, False)])
def test_gpu_mips_of_large_images_match_oracle(cg, w, h, filt, scale, wrap):
    from oracle import mip_oracle
    img = np.random.default_rng(w).integers(0, 256, (h, w, 4), dtype=np.uint8)
    levels = 7
    want = mip_oracle.generate_mipmaps(img, filt, scale, True, wrap, alpha=True, levels=levels)
    got = cg.generate_mipmaps(torch.from_numpy(img).cuda(), filt, scale, True, wrap, alpha=True, levels=levels)
    for l in range(1, levels):
        assert np.array_equal(got[l].cpu().numpy(), want[l] if len(want) == levels else want[l - 1]), l


def delayed(stream):
    """Keeps `stream` busy for some milliseconds, so that what is enqueued next waits there."""
    with torch.cuda.stream(stream):
        a = torch.zeros(1 << 28, dtype=torch.uint8, device="cuda")
        for _ in range(40):
            a.add_(1)


def test_calls_on_two_streams_match_oracle(cg):
    """Calls with device buffers return before their kernels have run: a second one of another size, from
    the same thread on another stream, must leave the first one's tables and images alone."""
    from oracle import mip_oracle
    from crunch2_gb300 import texgen
    sizes = [(203, 130), (66, 34), (330, 41)]
    imgs = [torch.from_numpy(texgen.colour_texture(w, h, w, with_alpha_noise=True)).cuda() for w, h in sizes]
    want = [mip_oracle.generate_mipmaps(i.cpu().numpy(), "kaiser", 0.9, True, False, alpha=True, levels=4) for i in imgs]
    for i in imgs:
        cg.generate_mipmaps(i, levels=4)  # plans made, buffers grown
    streams = [torch.cuda.Stream() for _ in imgs]
    torch.cuda.synchronize()
    for rep in range(3):
        delayed(streams[rep])
        got = []
        for k in range(3):
            s = streams[(rep + k) % 3]
            with torch.cuda.stream(s):
                got.append(cg.generate_mipmaps(imgs[k], levels=4, stream=s))
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(g, w)), rep


def test_image_encodes_on_two_streams(cg):
    """The same for compress_image, whose gathered blocks are the thread's."""
    from crunch2_gb300 import texgen
    imgs = [torch.from_numpy(texgen.colour_texture(w, h, w, with_alpha_noise=True)).cuda()
            for w, h in [(256, 128), (64, 44), (200, 180)]]
    fmts = [cg.FMT_DXT5, cg.FMT_DXT1, cg.FMT_DXT5A]
    want = [cg.compress_image(i, f) for i, f in zip(imgs, fmts)]
    streams = [torch.cuda.Stream() for _ in imgs]
    torch.cuda.synchronize()
    for rep in range(3):
        delayed(streams[rep])
        got = []
        for k in range(3):
            s = streams[(rep + k) % 3]
            with torch.cuda.stream(s):
                got.append(cg.compress_image(imgs[k], fmts[k], stream=s))
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want)), rep


def test_plans_of_many_sizes_are_kept(cg):
    """A program whose textures have more than a few sizes pays for each size once: a second round over forty
    sizes, whose plans take milliseconds each to make, goes much faster than the first, with the same bytes."""
    import time
    imgs = [torch.full((211 + 13 * k, 307 + 17 * k, 4), k, dtype=torch.uint8, device="cuda") for k in range(40)]
    rounds = []
    for _ in range(3):
        torch.cuda.synchronize()
        t = time.perf_counter()
        out = [cg.generate_mipmaps(i, "lanczos4", 0.91) for i in imgs]
        torch.cuda.synchronize()
        rounds.append((time.perf_counter() - t, out))
    assert min(r[0] for r in rounds[1:]) < 0.5 * rounds[0][0], [r[0] for r in rounds]
    for _, out in rounds[1:]:
        assert all(torch.equal(a, b) for x, y in zip(out, rounds[0][1]) for a, b in zip(x, y))
