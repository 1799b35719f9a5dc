"""GPU parity tests of the density path, called through the C ABI (megamol_gb300.p2v -> libp2v.so).

Bars: against the FP64 oracle, max-rel error (max|a-b| / max|b|) <= 1e-6 (the target is 1e-5); against
the reference module's own FP32 output (golden fixtures) the difference is bounded by the reference's
float rounding, <= 2e-5 of the maximum. Integer metadata (resolution, slice distances) must be identical.
"""
import math
import os

import numpy as np
import pytest
import torch

import oracle
from megamol_gb300 import build as nbuild
from megamol_gb300 import p2v, synth
from tests import golden_io as G

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


@pytest.fixture(scope="module")
def ctx():
    nbuild.build()
    c = p2v.Context(0)
    yield c
    c.close()


def run(ctx, lists, bbox, res, cyclic=(1, 1, 1), normalize=False, sigma=1.0, kernel=p2v.KERNEL_BUMP, mass=False,
        out=None, accumulate=p2v.ACCUM_EXACT, surface=False, out_res=None):
    """One frame; `out_res` sizes the host output when the module rewrites the resolution (surface)."""
    ctx.set_params(sizex=int(res[0]), sizey=int(res[1]), sizez=int(res[2]), cyclX=int(cyclic[0]),
                   cyclY=int(cyclic[1]), cyclZ=int(cyclic[2]), normalize=int(bool(normalize)), sigma=float(sigma),
                   kernel=kernel, mass_normalize=int(mass), forSurfaceReconstruction=int(bool(surface)),
                   accumulate=accumulate)
    r = out_res if out_res is not None else res
    if out is None:
        out = np.full(int(r[0]) * int(r[1]) * int(r[2]), np.nan, np.float32)
    meta = ctx.run_frame(lists, bbox, out)
    if isinstance(out, np.ndarray):
        r = meta["resolution"]
        out = out.reshape(int(r[2]), int(r[1]), int(r[0]))
    return out, meta


def maxrel(a, b):
    b = np.asarray(b, np.float64)
    return float(np.abs(np.asarray(a, np.float64) - b).max() / max(np.abs(b).max(), 1e-300))


def golden_lists(c):
    return [p2v.ParticleList(np.ascontiguousarray(L["data"]), L["type"], count=L["count"], stride=L["stride"],
                             global_radius=L["radius"]) for L in c["lists"]]


ACCUM = [p2v.ACCUM_EXACT, p2v.ACCUM_KAHAN]


@pytest.mark.parametrize("accumulate", ACCUM)
@pytest.mark.parametrize("name", G.golden_names())
def test_golden_vs_reference_and_fp64(ctx, name, accumulate):
    c = G.load(name)
    bbox, res = G.grid(c)  # the surface case's adjusted box, restated bit-exactly against the reference
    vol, meta = run(ctx, golden_lists(c), c["bbox"], c["res"], c["cyclic"], bool(c["normalize"]), float(c["sigma"]),
                    accumulate=accumulate, surface=bool(c["surface"]), out_res=res)
    ref = c["volume"]
    assert meta["resolution"] == [int(x) for x in res] and vol.shape == ref.shape
    xyzr = G.case_xyzr(c)
    v64 = oracle.density_f64(xyzr, bbox, res, c["cyclic"], float(c["sigma"]), oracle.BUMP, NT)
    if bool(c["normalize"]):
        v64, _, _ = oracle.normalize_f64(v64, "minmax")
    assert maxrel(vol, v64) <= 1e-6, f"{name}: vs FP64 {maxrel(vol, v64):.3e}"
    assert maxrel(vol, ref) <= 2e-5, f"{name}: vs reference {maxrel(vol, ref):.3e}"
    assert meta["slice_dists"] == [float(x) for x in c["slice_dists"]]
    if int(c["surface"]):
        assert meta["origin"] == [float(x) for x in c["origin"]]
        assert meta["extents"] == [float(x) for x in c["extents"]]
    if bool(c["normalize"]):
        assert meta["min_value"] == 0.0 and meta["max_value"] == 1.0
    else:
        assert abs(meta["max_value"] - float(c["max_value"])) <= 2e-5 * abs(float(c["max_value"]))


@pytest.mark.parametrize("accumulate", ACCUM)
def test_deterministic_bitwise(ctx, accumulate):
    f = synth.uniform(n=200_000, edge=60.0, res=96, seed=3)
    L = [p2v.ParticleList(f.xyzr, p2v.VERTDATA_FLOAT_XYZR)]
    a, _ = run(ctx, L, f.bbox, f.res, accumulate=accumulate)
    b, _ = run(ctx, L, f.bbox, f.res, accumulate=accumulate)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    # the exact mode is independent of the particle order: shuffle the input and compare bitwise
    if accumulate == p2v.ACCUM_EXACT:
        perm = np.random.default_rng(0).permutation(f.n)
        c, _ = run(ctx, [p2v.ParticleList(np.ascontiguousarray(f.xyzr[perm]), p2v.VERTDATA_FLOAT_XYZR)], f.bbox,
                   f.res, accumulate=accumulate)
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32))


def test_device_buffers_match_host_buffers(ctx):
    torch = pytest.importorskip("torch")
    f = synth.uniform(n=50_000, edge=30.0, res=40, seed=4)
    host, _ = run(ctx, [p2v.ParticleList(f.xyzr, p2v.VERTDATA_FLOAT_XYZR)], f.bbox, f.res)
    dx = torch.from_numpy(f.xyzr).cuda()
    dout = torch.empty(40 * 40 * 40, dtype=torch.float32, device="cuda")
    run(ctx, [p2v.ParticleList(dx, p2v.VERTDATA_FLOAT_XYZR, count=f.n)], f.bbox, f.res, out=dout)
    torch.cuda.synchronize()
    assert np.array_equal(dout.cpu().numpy().reshape(40, 40, 40), host)


def test_gauss3_and_mass_normalisation(ctx):
    f = synth.uniform(n=30_000, edge=30.0, res=40, seed=5)
    f.xyzr[:, 3] = np.random.default_rng(1).uniform(0.3, 0.7, f.n).astype(np.float32)
    L = [p2v.ParticleList(f.xyzr, p2v.VERTDATA_FLOAT_XYZR)]
    raw, _ = run(ctx, L, f.bbox, f.res, kernel=p2v.KERNEL_GAUSS3)
    v64 = oracle.density_f64(f.xyzr, f.bbox, f.res, (1, 1, 1), 1.0, oracle.GAUSS3, NT)
    assert maxrel(raw, v64) <= 1e-6
    vm, meta = run(ctx, L, f.bbox, f.res, kernel=p2v.KERNEL_GAUSS3, mass=True)
    h = oracle.spacing_f64(f.bbox, f.res)
    mass = vm.astype(np.float64).sum() * h[0] * h[1] * h[2]
    assert abs(mass - f.n) <= 1e-5 * f.n
    m64, _, _ = oracle.normalize_f64(v64, "mass", f.n, h)
    assert maxrel(vm, m64) <= 1e-6


def test_invalid_particles_are_dropped(ctx):
    f = synth.uniform(n=20_000, edge=20.0, res=24, seed=6)
    x = f.xyzr.copy()
    x[::97, 0] = np.nan
    x[5::101, 3] = 0.0
    x[7::103, 3] = -1.0
    x[9::107, 1] = np.inf
    vol, _ = run(ctx, [p2v.ParticleList(x, p2v.VERTDATA_FLOAT_XYZR)], f.bbox, f.res)
    ok = np.isfinite(x).all(1) & (x[:, 3] > 0)
    v64 = oracle.density_f64(x[ok], f.bbox, f.res, (1, 1, 1), 1.0, oracle.BUMP, NT)
    assert maxrel(vol, v64) <= 1e-6
    st = ctx.stats()
    assert st["particles_dropped"] == int((~ok).sum())
    assert st["particles_binned"] == int(ok.sum())


def test_empty_frame(ctx):
    vol, meta = run(ctx, [], (0, 0, 0, 1, 1, 1), (8, 8, 8), normalize=False)
    assert np.all(vol == 0)
    # the reference divides by (max - min) = 0 when normalising an empty grid; so does this library
    vol, meta = run(ctx, [], (0, 0, 0, 1, 1, 1), (8, 8, 8), normalize=True)
    assert np.all(np.isnan(vol))


@pytest.mark.parametrize("accumulate", ACCUM)
def test_out_of_box_particles_open_and_cyclic(ctx, accumulate):
    rng = np.random.default_rng(8)
    x = np.zeros((8000, 4), np.float32)
    x[:, :3] = rng.uniform(-6, 26, size=(8000, 3))
    x[:, 3] = rng.uniform(0.4, 1.6, 8000)
    for cyc in [(0, 0, 0), (1, 1, 1), (0, 1, 0)]:
        for sigma in (1.0, 1.7):
            vol, _ = run(ctx, [p2v.ParticleList(x, p2v.VERTDATA_FLOAT_XYZR)], (0, 0, 0, 20, 20, 20), (21, 18, 23),
                         cyc, sigma=sigma, accumulate=accumulate)
            v64 = oracle.density_f64(x, (0, 0, 0, 20, 20, 20), (21, 18, 23), cyc, sigma, oracle.BUMP, NT)
            assert maxrel(vol, v64) <= 1e-6, (cyc, sigma)


def test_surface_reconstruction_box(ctx):
    f = synth.uniform(n=5000, edge=10.0, res=16, seed=9)
    m = p2v.ParticlesToDensity(0, sizex=16, sizey=16, sizez=20, forSurfaceReconstruction=1, normalize=0)
    vol, meta = m.get_data([p2v.ParticleList(f.xyzr, p2v.VERTDATA_FLOAT_XYZR)], f.bbox)
    # modifyBBox makes voxels cubic and rewrites sizex / sizey (ParticlesToDensity.cpp:749-799)
    assert meta["resolution"][2] == 20
    sd = meta["slice_dists"]
    assert vol.shape == tuple(meta["resolution"][::-1])
    bb = meta["bbox"]
    assert (tuple(bb), tuple(meta["resolution"])) == oracle.modify_bbox_f32(f.bbox, (16, 16, 20))
    v64 = oracle.density_f64(f.xyzr, bb, meta["resolution"], (1, 1, 1), 1.0, oracle.BUMP, NT)
    assert maxrel(vol, v64) <= 1e-6
    assert m.param("sizex") == meta["resolution"][0]
    assert abs(sd[0] - sd[2]) < 0.2 * sd[2]


def test_surface_reconstruction_rejects_flat_box(ctx):
    """A box without depth would divide by a zero voxel spacing in the box adjustment (the reference's
    float-to-int conversions are then undefined): the frame is rejected and the context stays usable."""
    x = np.zeros((10, 4), np.float32)
    x[:, :2] = np.random.default_rng(1).uniform(0, 1, (10, 2))
    x[:, 3] = 0.5
    ctx.set_params(sizex=8, sizey=8, sizez=8, forSurfaceReconstruction=1, normalize=0, cyclX=0, cyclY=0, cyclZ=0)
    with pytest.raises(p2v.P2VError):
        ctx.run_frame([p2v.ParticleList(x, p2v.VERTDATA_FLOAT_XYZR)], (0, 0, 0, 1, 1, 0), None)
    vol, meta = run(ctx, [p2v.ParticleList(x, p2v.VERTDATA_FLOAT_XYZR)], (0, 0, 0, 1, 1, 1), (8, 8, 8))
    assert meta["resolution"] == [8, 8, 8] and np.isfinite(vol).all()


@pytest.mark.parametrize("seed,accumulate", [(0, p2v.ACCUM_EXACT), (1, p2v.ACCUM_KAHAN)])
def test_lj_liquid_full_size(ctx, seed, accumulate):
    """The headline workload at full size (4M particles, 256^3), against the FP64 oracle."""
    f = synth.lj_liquid(seed=2 + seed)
    vol, meta = run(ctx, [p2v.ParticleList(f.xyzr, p2v.VERTDATA_FLOAT_XYZR)], f.bbox, f.res, accumulate=accumulate)
    v64 = oracle.density_f64(f.xyzr, f.bbox, f.res, (1, 1, 1), 1.0, oracle.BUMP, NT)
    err = maxrel(vol, v64)
    assert err <= 1e-6, err
    st = ctx.stats()
    assert st["particles_binned"] == f.n and st["device_error"] == 0


@pytest.mark.parametrize("cyclic", [(1, 1, 1), (0, 0, 0)])
def test_particles_whose_support_misses_every_node(ctx, cyclic):
    """A frame of flat voxels (3.1 units in z against radii of 0.3-0.9, as in the mixed-phase frame) on the
    radix path (86 cells per particle): the binning sorts the particles whose support holds no node after all
    others and the gather never visits them. The grid is bit-identical to the one of plain cell keys (the AO
    brick order keeps them) and matches the FP64 oracle."""
    rng = np.random.default_rng(77)
    n = 40_000
    x = np.empty((n, 4), np.float32)
    x[:, :2] = rng.uniform(0, 40, (n, 2))
    x[:, 2] = rng.uniform(0, 400, n)
    x[:, 3] = rng.uniform(0.3, 0.9, n)
    bbox, res = (0.0, 0.0, 0.0, 40.0, 40.0, 400.0), (160, 160, 129)
    L = [p2v.ParticleList(x, p2v.VERTDATA_FLOAT_XYZR)]
    ctx.set_params(ao_brick_order=0)
    flagged, _ = run(ctx, L, bbox, res, cyclic=cyclic)
    flagged = flagged.copy()
    keys, order, start = ctx.binning()
    nbins = start.size - 1
    assert ctx.stats()["cell_max_count"] == 0  # the radix path
    miss = oracle.support_misses_nodes_f64(x, bbox, res)
    pf = np.zeros(n, bool)
    pf[order[keys > nbins]] = True
    assert pf.sum() > 0.3 * n and np.all(miss[pf]), (pf.sum(), miss.sum())
    ctx.set_params(ao_brick_order=1)
    try:
        plain, _ = run(ctx, L, bbox, res, cyclic=cyclic)
        assert ctx.binning()[0].max() <= nbins
    finally:
        ctx.set_params(ao_brick_order=0)
    assert np.array_equal(flagged.view(np.uint32), plain.view(np.uint32))
    v64 = oracle.density_f64(x, bbox, res, cyclic, 1.0, oracle.BUMP, NT)
    assert maxrel(flagged, v64) <= 1e-6


def crowd(n, edge, spread, radius, seed):
    """Half the particles in a Gaussian crowd at the box centre, half uniform; radii around `radius`."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(0.0, edge, (n, 3))
    p[::2] = edge / 2 + rng.normal(0.0, spread, ((n + 1) // 2, 3))
    return np.column_stack([np.clip(p, 0.0, edge), rng.uniform(0.8, 1.2, n) * radius]).astype(np.float32)


# n, box edge, crowd spread, radius, resolution: a tile one CTA may just walk alone and the next size, which queues its
# parts; many parts; more crowded tiles than the queue holds; more records than one CTA's sums take, without a queue
CROWDS = [(2 * 32_768, 24.0, 0.2, 0.9, 25), (2 * 32_768 + 2, 24.0, 0.2, 0.9, 25), (300_000, 48.0, 1.5, 0.9, 49),
          (40_000, 64.0, 20.0, 8.0, 65), (20_000, 15.0, 3.0, 5.0, 16), (300_000, 96.0, 1.5, 0.9, 97)]


@pytest.mark.parametrize("kernel", [p2v.KERNEL_BUMP, p2v.KERNEL_GAUSS3])
@pytest.mark.parametrize("n,edge,spread,radius,res", CROWDS)
def test_crowded_tiles(ctx, n, edge, spread, radius, res, kernel):
    """Tiles with tens of thousands of records: the FP64 bar, and the same bits for a shuffled frame. The 3-sigma
    Gaussian's support is three times the bump's: a third of the radius."""
    x = crowd(n, edge, spread, radius / (3 if kernel == p2v.KERNEL_GAUSS3 else 1), n)
    bbox, r = (0, 0, 0, edge, edge, edge), (res, res, res)
    vol, _ = run(ctx, [p2v.ParticleList(x)], bbox, r, kernel=kernel)
    ref = oracle.density_f64(x, bbox, r, (1, 1, 1), 1.0, oracle.GAUSS3 if kernel else oracle.BUMP, NT)
    assert maxrel(vol, ref) <= 1e-6, maxrel(vol, ref)
    again, _ = run(ctx, [p2v.ParticleList(x[np.random.default_rng(1).permutation(n)])], bbox, r, kernel=kernel)
    assert np.array_equal(vol, again)


@pytest.mark.parametrize("tile", [(16, 8, 8), (32, 16, 8)])
def test_crowded_tiles_of_other_shapes(ctx, tile):
    x = crowd(300_000, 48.0, 1.5, 0.9, 9)
    bbox, r = (0, 0, 0, 48.0, 48.0, 48.0), (49, 50, 47)
    ctx.set_params(tile_x=tile[0], tile_y=tile[1], tile_z=tile[2])
    vol, _ = run(ctx, [p2v.ParticleList(x)], bbox, r)
    ctx.set_params(tile_x=0, tile_y=0, tile_z=0)
    ref = oracle.density_f64(x, bbox, r, (1, 1, 1), 1.0, oracle.BUMP, NT)
    assert maxrel(vol, ref) <= 1e-6, maxrel(vol, ref)


@pytest.mark.parametrize("accumulate", [p2v.ACCUM_EXACT, p2v.ACCUM_KAHAN])
@pytest.mark.parametrize("radius", [10.0, 7.3, 1.6])
@pytest.mark.parametrize("kernel", [p2v.KERNEL_BUMP, p2v.KERNEL_GAUSS3])
def test_kernel_values_within_their_error_bound(ctx, kernel, radius, accumulate):
    """One particle on a node of a grid of unit spacing (every squared distance is a whole number): each node within the
    bound its operations give. Bump, x = 1 / w: w is off by at most 2.5 2^-24 (the support's square and its reciprocal,
    2^-24 of d2 / eps2 < 1 each, and the rounding of w), which moves exp(-x) by x^2 of it; the reciprocal's ulp by
    x 2^-23. Gaussian: the argument x by three roundings. __expf: (2 + 1.173 x) ulp as documented. Then the float of the
    sum, and the exact mode's quantum."""
    if kernel == p2v.KERNEL_GAUSS3:
        radius /= 3.0
    res, bbox = (25, 25, 25), (0.0, 0.0, 0.0, 24.0, 24.0, 24.0)
    x = np.array([[12.0, 12.0, 12.0, radius]], np.float32)
    vol, _ = run(ctx, [p2v.ParticleList(x)], bbox, res, cyclic=(0, 0, 0), kernel=kernel, accumulate=accumulate)
    i = np.arange(25, dtype=np.float64) - 12.0
    d2 = i[:, None, None] ** 2 + i[None, :, None] ** 2 + i[None, None, :] ** 2
    r = float(x[0, 3])
    u23 = 2.0 ** -23
    if kernel == p2v.KERNEL_BUMP:
        w = 1.0 - d2 / r ** 2
        arg = 1.0 / np.where(w > 0, w, np.inf)
        v = np.where(w > 0, np.exp(-arg), 0.0)
        rel = arg ** 2 * 1.25 * u23 + arg * u23 + (2.0 + 1.173 * arg) * u23
        err = v * np.expm1(rel)
    else:
        arg = d2 / (2.0 * r ** 2)
        e = np.exp(-arg)
        v = np.where(arg < 4.5, e - np.exp(-4.5), 0.0)
        err = e * np.expm1(1.5 * arg * u23 + (2.0 + 1.173 * arg) * u23) + np.exp(-4.5) * (2.0 + 1.173 * 4.5) * u23
    err = np.where(v > 0, err + v * 2.0 ** -24, 0.0) + 2.0 ** -32
    ref = oracle.density_f64(x, bbox, res, (0, 0, 0), 1.0, oracle.GAUSS3 if kernel else oracle.BUMP, 1)
    assert np.allclose(ref, v, rtol=1e-9, atol=1e-15)
    worst = (np.abs(vol - ref) / err).max()
    assert worst <= 1.0, worst


@pytest.mark.parametrize("n,records", [
    (40_000, lambda limit, chunk: limit), (40_000, lambda limit, chunk: limit + 1),
    (40_000, lambda limit, chunk: 3 * chunk), (40_000, lambda limit, chunk: 3 * chunk + 1),
    (32_768, lambda limit, chunk: 32_768),                           # no queue: the most one CTA walks alone
    (32_769, lambda limit, chunk: 32_769),                           # the smallest frame with a queue, all in one tile
    (1_300_001, lambda limit, chunk: limit), (1_300_001, lambda limit, chunk: limit + 1),
    (1_300_001, lambda limit, chunk: 5 * chunk),                     # limit and parts from n / SMs
])
def test_tiles_at_the_split_limit(ctx, n, records):
    """One isolated tile (16^3 nodes, the cells from one below it on) whose records all lie in one cell, so that their
    number is known: the last that its own CTA walks, the first that is queued, parts that end on its last record and one
    before it. The FP64 bar, and the same bits for a shuffled frame."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = records(max(4096, min(32_768, n // sms)), max(2048, min(8192, n // (4 * sms))))
    rng = np.random.default_rng(m)
    x = np.empty((n, 4), np.float32)
    x[:m, :3] = rng.uniform(24.05, 24.95, (m, 3))
    x[m:, 0] = rng.uniform(33.0, 126.0, n - m)                       # no other tile shares that cell's records
    x[m:, 1:3] = rng.uniform(0.0, 126.0, (n - m, 2))
    x[:, 3] = 0.9
    bbox, r = (0.0, 0.0, 0.0, 127.0, 127.0, 127.0), (128, 128, 128)
    vol, _ = run(ctx, [p2v.ParticleList(x)], bbox, r, cyclic=(0, 0, 0))
    ref = oracle.density_f64(x, bbox, r, (0, 0, 0), 1.0, oracle.BUMP, NT)
    assert maxrel(vol, ref) <= 1e-6, maxrel(vol, ref)
    again, _ = run(ctx, [p2v.ParticleList(x[rng.permutation(n)])], bbox, r, cyclic=(0, 0, 0))
    assert np.array_equal(vol, again)


@pytest.mark.parametrize("n,radius,tile", [(30_000, 0.9, 16), (30_000, 3.0, 16), (400_000, 2.0, 16), (30_000, 0.9, 8)])
def test_mass_sum_is_the_sum_of_the_grid(ctx, n, radius, tile):
    """stats["mass_sum"] is the sum of the floats of the raw grid: exact integers within a tile, one FP64 rounding per tile
    is the most it may lack (a sum of the unrounded fixed-point values is off by about 1e-9 of it). Nodes below and above
    1, crowded tiles that are written by their last part."""
    x = crowd(n, 40.0, 1.5, radius, n)
    res = (49, 50, 47)
    if tile != 16:
        ctx.set_params(tile_x=16, tile_y=8, tile_z=8)
    vol, _ = run(ctx, [p2v.ParticleList(x)], (0, 0, 0, 40.0, 40.0, 40.0), res)
    ctx.set_params(tile_x=0, tile_y=0, tile_z=0)
    exact = math.fsum(vol.ravel().tolist())
    tiles = 4 * 4 * 3 if tile == 16 else 4 * 7 * 6
    assert vol.max() > 1.0
    assert abs(ctx.stats()["mass_sum"] - exact) <= (tiles + 2) * 2.0 ** -53 * exact


@pytest.mark.parametrize("res", [(17, 17, 17), (48, 47, 49), (80, 81, 79), (97, 97, 96)])
@pytest.mark.parametrize("n,spread", [(1_000, 0.5), (60_000, 1.0), (60_000, 6.0)])
def test_kahan_gather_of_crowded_tiles(ctx, res, n, spread):
    """Grids of so few tiles that an SM holds one CTA, two and three (they stage 6400, 2816 and 1728 records at a time), with
    tiles of fewer records than that and of many chunks: the FP64 bar, and the same bits again."""
    x = crowd(n, 24.0, spread, 1.2 * 24.0 / 96, n + res[0])
    bbox = (0, 0, 0, 24.0, 24.0, 24.0)
    vol, _ = run(ctx, [p2v.ParticleList(x)], bbox, res, accumulate=p2v.ACCUM_KAHAN)
    ref = oracle.density_f64(x, bbox, res, (1, 1, 1), 1.0, oracle.BUMP, NT)
    assert maxrel(vol, ref) <= 1e-6, maxrel(vol, ref)
    again, _ = run(ctx, [p2v.ParticleList(x)], bbox, res, accumulate=p2v.ACCUM_KAHAN)
    assert np.array_equal(vol, again)
