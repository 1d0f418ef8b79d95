"""The transcoder's walk decoder (the largest levels of a plan) against the lane decoder, which has
one serial chain per level: rows that are and are not multiples of eight blocks (row ends of one,
two and three chunks, of two blocks), several table segments, every format, cube maps, batches, and
streams cut short or overwritten (the status and every byte that the two write)."""
import numpy as np
import pytest

import golden_util as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def cg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import crunch2_gb300
    crunch2_gb300.lib()
    return crunch2_gb300


def texture(fmt, w, h, seed):
    from crunch2_gb300 import texgen
    if fmt == "dxn":
        return texgen.normal_map(w, h, seed)
    return texgen.colour_texture(w, h, seed, with_alpha_noise=fmt != "dxt1")


def make(cg, fmt, w, h, seed, levels=3, faces=1, quality=128):
    from crunch2_gb300 import texgen
    f = {"dxt1": cg.FMT_DXT1, "dxt5": cg.FMT_DXT5, "dxn": cg.FMT_DXN_XY, "dxt5a": cg.FMT_DXT5A}[fmt]
    return cg.compress_crn([texgen.mip_chain(texture(fmt, w, h, seed + i), levels) for i in range(faces)], f, quality)


def decode(cg, crn, split, levels=None):
    cg.set_decode_split(split)
    try:
        with cg.unpack_begin(crn) as ctx:
            n = levels or ctx.levels
            out = torch.full((sum(ctx.level_bytes(l) for l in range(n)),), 0xCD, dtype=torch.uint8, device="cuda")
            try:
                ctx.unpack_levels(0, n, out=out)
                code = 0
            except cg.CrnGpuError as e:
                code = e.code
            torch.cuda.synchronize()
            return code, out.cpu().numpy()
    finally:
        cg.set_decode_split(cg.DECODE_SPLIT_DEFAULT)


@pytest.mark.parametrize("fmt,w,h,faces", [
    ("dxt1", 512, 512, 1), ("dxt5", 256, 320, 1), ("dxn", 264, 200, 1), ("dxt5a", 260, 260, 1),
    ("dxt1", 1020, 90, 1), ("dxt5", 332, 180, 1), ("dxt1", 333, 444, 1), ("dxn", 148, 257, 1),
    ("dxt1", 128, 128, 6), ("dxt5", 4096, 32, 1),
])
def test_walk_matches_lane(cg, fmt, w, h, faces):
    crn = make(cg, fmt, w, h, w + h, faces=faces)
    lane = decode(cg, crn, cg.DECODE_LANE_ONLY)
    assert lane[0] == 0
    walk = decode(cg, crn, cg.DECODE_SPLIT_DEFAULT)
    assert walk[0] == 0 and np.array_equal(walk[1], lane[1])


@pytest.mark.parametrize("fmt,quality", [("dxt1", 255), ("dxt5", 192)])
def test_many_segments(cg, fmt, quality):
    crn = make(cg, fmt, 1024, 768, 5, levels=1, quality=quality)
    lane = decode(cg, crn, cg.DECODE_LANE_ONLY)
    walk = decode(cg, crn, cg.DECODE_SPLIT_DEFAULT)
    assert lane[0] == walk[0] == 0 and np.array_equal(walk[1], lane[1])


@pytest.mark.parametrize("fmt,w", [("dxt1", 512), ("dxt5", 300)])
@pytest.mark.parametrize("damage", ["cut", "zeros", "ones", "noise"])
def test_damaged_streams(cg, fmt, w, damage):
    """A level stream overwritten from a point on: the file's own level 0 lies before the others."""
    crn = bytearray(make(cg, fmt, w, 512, 9, levels=1))
    tail = len(crn) // 3
    rng = np.random.default_rng(1)
    fill = {"cut": b"\0" * tail, "zeros": b"\0" * tail, "ones": b"\xff" * tail,
            "noise": rng.integers(0, 256, tail, np.uint8).tobytes()}[damage]
    crn[len(crn) - tail:] = fill
    if damage == "cut":  # the stream ends early: segmented entry with a shorter buffer
        crn = bytes(make(cg, fmt, w, 512, 9, levels=1))
        with cg.unpack_begin(crn) as ctx:
            size = ctx.level_bytes(0)
        outs = []
        for split in (cg.DECODE_LANE_ONLY, cg.DECODE_SPLIT_DEFAULT):
            cg.set_decode_split(split)
            with cg.unpack_begin(crn) as ctx:
                out = torch.full((size,), 0xCD, dtype=torch.uint8, device="cuda")
                import ctypes
                faces = (ctypes.c_void_p * 1)(out.data_ptr())
                half = torch.from_numpy(np.frombuffer(crn[-len(crn) // 2:], np.uint8)[:len(crn) // 3].copy()).cuda()
                pad = torch.cat([half, torch.zeros(64, dtype=torch.uint8, device="cuda")])
                rc = cg.lib().crngpu_unpack_level_segmented(ctx.handle, pad.data_ptr(), half.numel(), faces, size, 0, 0,
                                                            cg.MEM_DEVICE, None)
                torch.cuda.synchronize()
                outs.append((rc, out.cpu().numpy()))
            cg.set_decode_split(cg.DECODE_SPLIT_DEFAULT)
        lane, walk = outs
    else:
        lane, walk = (decode(cg, bytes(crn), s) for s in (cg.DECODE_LANE_ONLY, cg.DECODE_SPLIT_DEFAULT))
    assert walk[0] == lane[0]
    assert np.array_equal(walk[1], lane[1])


def test_batch_of_walks(cg):
    specs = [("dxt1", 512, 256), ("dxt5", 300, 300), ("dxn", 256, 512), ("dxt1", 130, 260), ("dxt1", 64, 64)]
    crns = [make(cg, f, w, h, 20 + i) for i, (f, w, h) in enumerate(specs)]
    want = [decode(cg, c, cg.DECODE_LANE_ONLY)[1] for c in crns]
    ctxs = [cg.unpack_begin(c) for c in crns]
    outs = [torch.zeros(len(w), dtype=torch.uint8, device="cuda") for w in want]
    with cg.UnpackBatch([(c, 0, c.levels, o) for c, o in zip(ctxs, outs)]) as b:
        for graph in (False, True, True):
            for o in outs:
                o.zero_()
            b.launch(use_graph=graph)
            b.status()
            for o, w in zip(outs, want):
                assert np.array_equal(o.cpu().numpy(), w)
    for c in ctxs:
        c.close()


def test_launches_on_two_streams(cg):
    """A batch has one set of index records, walk states and counters: launches on two streams, directly and
    from the batch's graph, without a wait between them."""
    specs = [("dxt1", 512, 256), ("dxt5", 300, 300), ("dxn", 256, 512), ("dxt1", 64, 64)]
    crns = [make(cg, f, w, h, 40 + i) for i, (f, w, h) in enumerate(specs)]
    want = [torch.from_numpy(decode(cg, c, cg.DECODE_LANE_ONLY)[1]).cuda() for c in crns]
    ctxs = [cg.unpack_begin(c) for c in crns]
    outs = [torch.zeros_like(w) for w in want]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with cg.UnpackBatch([(c, 0, c.levels, o) for c, o in zip(ctxs, outs)]) as b:
        b.launch()
        torch.cuda.synchronize()
        for graph in (False, True):
            got = []
            for rep in range(6):
                with torch.cuda.stream(streams[0]):
                    for o in outs:
                        o.zero_()
                    b.launch(use_graph=graph, stream=streams[0])
                    got.append([o.clone() for o in outs])
                b.launch(use_graph=graph, stream=streams[1])  # beside the copies; writes the same bytes
            b.status(streams[0])
            torch.cuda.synchronize()
            for g in got:
                assert all(torch.equal(x, y) for x, y in zip(g, want)), graph
    for c in ctxs:
        c.close()


# What follows runs the walk decoder whatever the cost model would choose, and checks that it ran.

@pytest.fixture
def walk_only(cg):
    cg.set_decode_split(cg.DECODE_WALK_ONLY)
    cg.decode_counters(reset=True)
    yield
    cg.set_decode_split(cg.DECODE_SPLIT_DEFAULT)


@pytest.mark.parametrize("name", sorted(G.manifest().keys()))
def test_walk_alone_writes_golden_levels(cg, walk_only, name):
    """Every level of every fixture, 1 x 1 ones and cube faces included, one at a time and all in one plan."""
    m = G.manifest()[name]
    with cg.unpack_begin(G.crn_bytes(name)) as ctx:
        for lvl, info in enumerate(m["levels"]):
            assert G.sha(ctx.unpack_levels(lvl, 1)) == info["sha256"], (name, lvl)
        allv = ctx.unpack_levels()
    pos = 0
    for lvl, info in enumerate(m["levels"]):
        assert G.sha(allv[pos:pos + info["bytes"]]) == info["sha256"], (name, lvl, "all levels")
        pos += info["bytes"]
    n = cg.decode_counters()
    assert (n["lane"], n["wide"], n["walk"]) == (0, 0, 2 * len(m["levels"]))


# rows of 1, 2, 3, 8, 9, 10, 13 and 1024 blocks: every remainder of the groups of eight, the smallest and
# the widest; the large ones over many segments
@pytest.mark.parametrize("fmt,w,h,segments", [
    ("dxt1", 4, 4, 1), ("dxt5", 8, 12, 1), ("dxn", 12, 100, 1), ("dxt5a", 32, 32, 1), ("dxt5", 36, 60, 1),
    ("dxn", 40, 64, 1), ("dxt1", 52, 44, 1), ("dxt1", 4096, 64, 2), ("dxt5", 1024, 768, 9), ("dxn", 1000, 600, 5),
    ("dxt1", 1024, 768, 5)])
def test_walk_alone_matches_lane(cg, walk_only, fmt, w, h, segments):
    crn = make(cg, fmt, w, h, w + h, levels=1, quality=255)
    lane = decode(cg, crn, cg.DECODE_LANE_ONLY)
    cg.decode_counters(reset=True)
    walk = decode(cg, crn, cg.DECODE_WALK_ONLY)
    n = cg.decode_counters()
    assert (n["lane"], n["wide"], n["walk"]) == (0, 0, 1) and n["walk_segments"] >= segments, n
    assert lane[0] == walk[0] == 0 and np.array_equal(walk[1], lane[1])


@pytest.mark.parametrize("name", ["dxt1_256", "dxt5_256", "dxn_xy_256", "dxt5a_256", "dxt5_cube_64x32"])
def test_walk_alone_on_corrupt_streams(cg, walk_only, name):
    """Random bytes over a level's stream: the lane decoder's status, or its bytes where it still decodes."""
    import struct
    crn = bytes(G.crn_bytes(name))
    nlev = len(G.manifest()[name]["levels"])
    ofs = [struct.unpack(">I", crn[70 + 4 * l:74 + 4 * l])[0] for l in range(nlev)] + [len(crn)]
    rng = np.random.default_rng(12)
    for trial in range(16):
        lvl = trial % 2
        bad = bytearray(crn)
        pos = ofs[lvl] + int(rng.integers(0, max(1, ofs[lvl + 1] - ofs[lvl] - 16)))
        n = int(min(32, ofs[lvl + 1] - pos))
        bad[pos:pos + n] = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
        lane = decode(cg, bytes(bad), cg.DECODE_LANE_ONLY, 2)
        cg.decode_counters(reset=True)
        walk = decode(cg, bytes(bad), cg.DECODE_WALK_ONLY, 2)
        assert cg.decode_counters()["walk"] == 2
        assert walk[0] == lane[0] and (lane[0] or np.array_equal(walk[1], lane[1])), (name, trial)


def test_default_split_walks_a_large_level(cg):
    cg.decode_counters(reset=True)
    code, _ = decode(cg, make(cg, "dxt1", 1024, 1024, 3, levels=1), cg.DECODE_SPLIT_DEFAULT)
    n = cg.decode_counters()
    assert code == 0 and n["walk"] == 1 and n["walk_segments"] > 3, n


@pytest.mark.parametrize("most", [0, 1 << 20])
def test_plans_without_scratch_use_the_other_decoders(cg, most):
    """What a failed allocation of the walk's scratch does too: unpack calls, calls by level and batches."""
    names = ["c1_dxt1_1024", "dxt5_2048", "dxn_xy_2048"]
    man = G.manifest()
    cg.set_decode_scratch(most)
    try:
        cg.decode_counters(reset=True)
        ctxs = [cg.unpack_begin(G.crn_bytes(n)) for n in names]
        outs = [torch.zeros(sum(l["bytes"] for l in man[n]["levels"]), dtype=torch.uint8, device="cuda") for n in names]
        with cg.UnpackBatch([(c, 0, c.levels, o) for c, o in zip(ctxs, outs)]) as b:
            b.launch()
            b.status()
        for n, c, o in zip(names, ctxs, outs):
            got = [o.cpu().numpy(), c.unpack_levels()]
            pos = 0
            for lvl, info in enumerate(man[n]["levels"]):
                for g in got:
                    assert G.sha(g[pos:pos + info["bytes"]]) == info["sha256"], (n, lvl)
                pos += info["bytes"]
                assert G.sha(c.unpack_level(lvl).reshape(-1)) == info["sha256"], (n, lvl)
            c.close()
        assert cg.decode_counters()["walk"] == 0
    finally:
        cg.set_decode_scratch(None)
    cg.decode_counters(reset=True)
    with cg.unpack_begin(G.crn_bytes(names[0])) as c:
        c.unpack_levels()
    assert cg.decode_counters()["walk"] > 0


@pytest.fixture
def waits_run_out(cg, walk_only):
    cg.wait_counters(reset=True)
    cg.force_wait_timeouts(True)
    yield
    cg.force_wait_timeouts(False)


@pytest.mark.parametrize("name", ["c1_dxt1_1024", "dxt5_256", "dxn_xy_256", "dxt5a_256", "dxt1_100x60", "dxt5_cube_64x32"])
def test_levels_whose_walk_gives_up_are_decoded_all_the_same(cg, waits_run_out, name):
    levels = G.manifest()[name]["levels"]
    with cg.unpack_begin(G.crn_bytes(name)) as ctx:
        out = torch.zeros(sum(l["bytes"] for l in levels), dtype=torch.uint8, device="cuda")
        with cg.UnpackBatch([(ctx, 0, len(levels), out)]) as b:
            b.set_variant(0)  # an expansion without waits of its own
            for use_graph in (False, True):
                for forced in (True, False):
                    out.zero_()
                    cg.force_wait_timeouts(forced)
                    cg.wait_counters(reset=True)
                    b.launch(use_graph=use_graph)
                    b.status()
                    n = cg.wait_counters()
                    assert n["expand_stage_timeouts"] == (len(levels) if forced else 0), n
                    assert n["expand_drain_failures"] == 0, n
                    host, pos = out.cpu().numpy(), 0
                    for lvl, info in enumerate(levels):
                        assert G.sha(host[pos:pos + info["bytes"]]) == info["sha256"], (lvl, use_graph, forced)
                        pos += info["bytes"]


def test_a_walk_that_gives_up_keeps_the_status_of_a_corrupt_stream(cg, waits_run_out):
    crn = bytearray(make(cg, "dxt1", 256, 256, 9, levels=1))
    crn[len(crn) - len(crn) // 3:] = b"\xff" * (len(crn) // 3)
    lane = decode(cg, bytes(crn), cg.DECODE_LANE_ONLY)
    walk = decode(cg, bytes(crn), cg.DECODE_WALK_ONLY)
    assert cg.wait_counters()["expand_stage_timeouts"] > 0
    assert walk[0] == lane[0] and (lane[0] or np.array_equal(walk[1], lane[1]))


@pytest.mark.parametrize("name", ["c1_dxt1_1024", "dxt5_256", "dxn_xy_256", "dxt1_cube_64"])
def test_calls_whose_walk_gives_up_decode_again_without_it(cg, waits_run_out, name):
    levels = G.manifest()[name]["levels"]
    with cg.unpack_begin(G.crn_bytes(name)) as ctx:
        out = ctx.unpack_levels()
        n = cg.decode_counters()
        assert n["walk"] == len(levels) and n["lane"] + n["wide"] == len(levels)
        pos = 0
        for lvl, info in enumerate(levels):
            assert G.sha(out[pos:pos + info["bytes"]]) == info["sha256"], lvl
            assert G.sha(ctx.unpack_level(lvl).reshape(-1)) == info["sha256"], lvl
            pos += info["bytes"]
    assert cg.wait_counters()["expand_drain_failures"] == 0
