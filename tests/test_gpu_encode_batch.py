"""Batched plain encode (crngpu_encode_batch_*): the mip chains of textures of mixed sizes and
formats, encoded by one gather launch and two persistent encoder launches, must give exactly the
blocks crngpu_compress_image gives on each level -- directly and replayed from the CUDA graph --
and the oracle's on a sample of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def cg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import crunch2_gb300
    crunch2_gb300.lib()
    return crunch2_gb300


# (width, height, format, content, seed): NPOT, 1-texel and tall/wide chains, every format family
CASES = [(32, 32, "DXT1", "colour", 1), (64, 128, "DXT5", "colour_alpha", 2), (100, 60, "DXN_XY", "normal", 3),
         (256, 32, "DXT1", "colour", 4), (48, 48, "DXT5A", "colour_alpha", 5), (1, 1, "DXT1", "colour", 6),
         (128, 64, "DXN_YX", "normal", 7), (512, 512, "DXT1", "colour", 8), (8, 200, "DXT5", "colour_alpha", 9),
         (300, 5, "DXT5A", "colour_alpha", 10)]


def make_items(cg, cases):
    from crunch2_gb300 import texgen
    fmts = {"DXT1": cg.FMT_DXT1, "DXT5": cg.FMT_DXT5, "DXN_XY": cg.FMT_DXN_XY, "DXN_YX": cg.FMT_DXN_YX,
            "DXT5A": cg.FMT_DXT5A}
    items, chains = [], []
    for w, h, fmt, content, seed in cases:
        img = texgen.normal_map(w, h, seed) if content == "normal" else \
            texgen.colour_texture(w, h, seed, with_alpha_noise=(content == "colour_alpha"))
        levels = texgen.mip_chain(img)
        rgba = torch.from_numpy(np.concatenate([l.reshape(-1) for l in levels])).cuda()
        f = fmts[fmt]
        out = torch.zeros(cg.mip_chain_blocks(w, h, len(levels)) * cg.bytes_per_block(f), dtype=torch.uint8,
                          device="cuda")
        items.append((rgba, out, w, h, len(levels), f))
        chains.append(levels)
    return items, chains


@pytest.mark.parametrize("flags", ["perceptual_both", "uniform"])
def test_batch_equals_per_image(cg, flags):
    fl = cg.FLAG_PERCEPTUAL | cg.FLAG_USE_BOTH_BLOCK_TYPES if flags == "perceptual_both" else 0
    items, chains = make_items(cg, CASES)
    with cg.EncodeBatch(items, fl) as b:
        assert b.blocks == sum(cg.mip_chain_blocks(w, h, n) for _, _, w, h, n, _ in items)
        for use_graph in (False, True, True):
            for _, out, *_ in items:
                out.zero_()
            b.launch(use_graph=use_graph)
            torch.cuda.synchronize()
            for (rgba, out, w, h, n, f), levels in zip(items, chains):
                got = out.cpu().numpy()
                ofs = 0
                for l in levels:
                    ref = np.asarray(cg.compress_image(l, f, fl)).reshape(-1)
                    assert np.array_equal(got[ofs:ofs + ref.size], ref), (w, h, f, l.shape, use_graph)
                    ofs += ref.size
                assert ofs == got.size
        grids, ms = b.tuning()
        assert grids[0] > 0 and grids[1] > 0 and len(ms) == 8


def test_batch_rejects_bad_items(cg):
    items, _ = make_items(cg, CASES[:2])
    rgba, out, w, h, n, f = items[0]
    with pytest.raises(cg.CrnGpuError):
        cg.EncodeBatch([(rgba, out, w, h, n + 5, f)])  # more levels than the chain has
    with pytest.raises(cg.CrnGpuError):
        cg.EncodeBatch([(rgba, out, w, h, n, 4)])  # a format this encoder does not write (DXT3)
    with pytest.raises(cg.CrnGpuError):
        cg.EncodeBatch([(rgba, out[:8], w, h, n, f)])  # output too small


@pytest.mark.parametrize("blocks_past_two_rounds", [-1, 0, 1, 5])
@pytest.mark.parametrize("quality", [4, 1])
def test_block_counts_around_two_per_warp_match_short_calls(cg, blocks_past_two_rounds, quality):
    # up to two blocks a search warp (32 warps an SM) are dealt out in turn, more through a counter
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    n = 2 * warps + blocks_past_two_rounds
    rng = np.random.default_rng(n)
    few = rng.integers(0, 256, (n, 4, 4), dtype=np.uint8)  # up to four colours a block
    px = np.take_along_axis(few, rng.integers(0, 4, (n, 16, 1)), axis=1)
    px[..., 3] = 255
    px[::7] = rng.integers(0, 256, px[::7].shape, dtype=np.uint8) | np.uint8([0, 0, 0, 255])
    blocks = torch.from_numpy(px.reshape(n, 64)).cuda()
    got = cg.dxt1_optimize(blocks, quality=quality).cpu().numpy()
    half = n // 2
    want = [cg.dxt1_optimize(b.contiguous(), quality=quality).cpu().numpy() for b in (blocks[:half - 3], blocks[half - 3:n - 9], blocks[n - 9:])]
    assert np.array_equal(got, np.concatenate(want))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 33])
def test_alpha_block_counts_match_single_blocks(cg, n):
    # half a warp a block, eight blocks a CTA: odd counts, short last CTAs, one-value blocks beside full ones
    rng = np.random.default_rng(n)
    img = rng.integers(0, 256, (4, 4 * n, 4), dtype=np.uint8)
    img[..., 3] = np.where(rng.integers(0, 3, (4, 4 * n)) > 0, img[..., 3] // 64 * 60, img[..., 3])
    img[:, 4 * (n // 2):4 * (n // 2) + 4, 3] = 77
    flags = cg.FLAG_USE_BOTH_BLOCK_TYPES
    got = np.asarray(cg.compress_image(img, cg.FMT_DXT5A, flags)).reshape(n, 8)
    for b in range(n):
        want = np.asarray(cg.compress_image(np.ascontiguousarray(img[:, 4 * b:4 * b + 4]), cg.FMT_DXT5A, flags))
        assert np.array_equal(got[b], want.reshape(8)), b


@pytest.mark.parametrize("w,h,skip", [(64, 20, 0), (61, 19, 0), (64, 20, 1), (3, 70, 0), (64, 20, 4)])
def test_images_with_and_without_aligned_rows_match(cg, w, h, skip):
    # rows of 16-byte pieces are read whole, all others by texel: both, with ragged right and lower edges
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    wide = torch.zeros((h, w + skip, 4), dtype=torch.uint8, device="cuda")
    wide[:, skip:] = torch.from_numpy(img).cuda()
    got = cg.compress_image(wide[:, skip:].contiguous(), cg.FMT_DXN_XY, 0)
    flat = torch.zeros(h * w * 4 + 16, dtype=torch.uint8, device="cuda")
    shifted = flat[4 * skip:4 * skip + h * w * 4].view(h, w, 4)
    shifted.copy_(torch.from_numpy(img))
    again = cg.compress_image(shifted, cg.FMT_DXN_XY, 0)
    want = np.asarray(cg.compress_image(img, cg.FMT_DXN_XY, 0))
    to = lambda t: t.cpu().numpy() if hasattr(t, "cpu") else np.asarray(t)
    assert np.array_equal(to(got).reshape(-1), want.reshape(-1)) and np.array_equal(to(again).reshape(-1), want.reshape(-1))


@pytest.mark.parametrize("past", [-1, 0, 1])
def test_block_counts_around_the_few_blocks_search_match(cg, past):
    # up to 16 blocks an SM go to the search with twice the registers: both sides, and one with the other
    n = torch.cuda.get_device_properties(0).multi_processor_count * 16 + past
    rng = np.random.default_rng(n)
    px = rng.integers(0, 256, (n, 16, 4), dtype=np.uint8) // rng.integers(1, 40, (n, 1, 1), dtype=np.uint8)
    px[..., 3] = 255
    blocks = torch.from_numpy(px.reshape(n, 64)).cuda()
    got, err = cg.dxt1_optimize(blocks, with_error=True)
    twice, terr = cg.dxt1_optimize(torch.cat([blocks, blocks]), with_error=True)
    for half in (0, 1):
        assert torch.equal(twice[half * n:(half + 1) * n], got) and torch.equal(terr[half * n:(half + 1) * n], err)


@pytest.mark.parametrize("from_line, n", [(0, 1), (0, 7), (0, 9), (0, 33), (1, -1), (1, 0), (1, 1)])
def test_seeds_of_few_blocks_match_those_of_many(cg, from_line, n):
    # below 40 blocks an SM four lanes take a block: short groups of eight, and both sides of the line,
    # against the same blocks among as many again
    line = torch.cuda.get_device_properties(0).multi_processor_count * 40
    total = line + n if from_line else n
    rng = np.random.default_rng(total)
    px = rng.integers(0, 256, (total, 16, 4), dtype=np.uint8) // rng.integers(1, 60, (total, 1, 4), dtype=np.uint8)
    px[rng.integers(0, 2, (total, 16)) > 0] &= 0xF0
    px[..., 3] = 255
    blocks = torch.from_numpy(px.reshape(total, 64)).cuda()
    for perceptual in (True, False):
        got = cg.dxt1_optimize(blocks, perceptual)
        among = cg.dxt1_optimize(blocks.repeat((line + total) // total + 1, 1), perceptual)
        assert torch.equal(among[:total], got) and torch.equal(among[-total:], got)


def test_launches_on_two_streams_and_in_a_callers_graph(cg):
    """A batch has one set of gathered blocks, seeds and block counter: launches on two streams, directly
    and from the batch's graph, without a wait between them, and from a graph the caller captured."""
    items, _ = make_items(cg, [(512, 512, "DXT1", "colour", 8), (256, 256, "DXT5", "colour_alpha", 2)])
    outs = [it[1] for it in items]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with cg.EncodeBatch(items) as b:
        b.launch()
        torch.cuda.synchronize()
        want = [o.clone() for o in outs]
        for use_graph in (False, True):
            got = []
            for rep in range(6):
                with torch.cuda.stream(streams[0]):
                    for o in outs:
                        o.zero_()
                    b.launch(use_graph=use_graph, stream=streams[0])
                    got.append([o.clone() for o in outs])
                b.launch(use_graph=use_graph, stream=streams[1])  # beside the copies; writes the same bytes
            torch.cuda.synchronize()
            for g in got:
                assert all(torch.equal(x, y) for x, y in zip(g, want)), use_graph
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            b.launch(stream=streams[0])
        for rep in range(3):
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(streams[0]):
                graph.replay()
                got = [o.clone() for o in outs]
            b.launch(stream=streams[1])
            torch.cuda.synchronize()
            assert all(torch.equal(x, y) for x, y in zip(got, want)), rep
