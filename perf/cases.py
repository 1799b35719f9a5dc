"""Workloads of the particle-to-volume path, for timing: what a program that uses this library calls, over the
sizes its configurations, tests and benchmark name.

A case is a dict of plain values. `listed()` are the named cases, `draw(rng)` gives another one of the same
ranges, `prepare(case, seed)` makes what a program holds before the call (inputs, context, network), `run(state)`
makes one call through the public entry points, `work(case)` is what the call cannot do without, and
`exact(case, seed)` is the same result in 64-bit arithmetic from plain torch.

The particles are generated on the GPU from the seed alone, with the distributions of the library's synthetic
frames: a uniform gas, a jittered FCC liquid, the mixed-phase slab with gas above it, and Gaussian blobs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from megamol_gb300 import p2v

# The AO of the benchmark: 8 cones x 32 samples over a 3-level pyramid of the normalised density, normals down
# the density gradient computed by the library
AO_BENCH = dict(ao_volume=p2v.AOVOL_DENSITY, ao_volume_scale=1.0, ao_cones=8, ao_steps=32, ao_levels=3, ao_apex_deg=50.0,
                ao_offset=0.01, ao_strength=1.0, ao_cone_length=0.8, ao_early_exit=1,
                ao_normals=p2v.NORMALS_GRADIENT)
EDGES = (64, 96, 128, 160, 192, 224, 256)  # grid edges of trajectory frames


def listed():
    return [
        # A small frame in an interactive session (the size of the smoke check): the density grid alone, where
        # launches and latency are the cost.
        frame("density_20k", "uniform", 20_000, (48, 48, 48)),
        # The small plain-method configuration: 100k particles with one global radius (FLOAT_XYZ), the 3-sigma
        # Gaussian, a 128^3 grid and the plain cone march.
        frame("uniform_100k_cone", "uniform", 100_000, (128, 128, 128), kernel="gauss3", ao="cone", vertex="xyz"),
        # A renderer's MDAO mode with the reference's defaults (3 cones, geometric steps, the 8-bit occupancy
        # volume of 128 voxels along the longest edge): two lists (float and double positions) with their own
        # directions, an odd count and a ragged grid.
        frame("mdao_250k_lists", "liquid", 250_003, (100, 75, 113), ao="mdao", vertex="xyz+double", normals="list"),
        # The AOSphereRenderer's main-axes AO of a frame whose density is Kahan-compensated and mass-normalised.
        frame("aosphere_864k_kahan", "liquid", 864_000, (154, 154, 154), ao="aosphere", normals="list",
              accumulate="kahan", normalize="mass"),
        # The module as MegaMol calls it: host arrays in, host volume out, the intensity aggregator.
        frame("intensity_600k_host", "uniform", 600_000, (129, 127, 130), aggregator=1, memory="host"),
        # The vector aggregator (velocity field on a grid), open boundaries.
        frame("vector_500k", "liquid", 500_000, (96, 96, 96), aggregator=2, cyclic=0, normalize="none"),
        # The LJ-liquid configuration with the plain cone march, and with the learned AO.
        frame("lj_4M_cone", "liquid", 4_000_000, (256, 256, 256), ao="cone"),
        frame("lj_4M_learned", "liquid", 4_000_000, (256, 256, 256), ao="learned"),
        # The learned AO's inference set: 16M particles of the small configuration's structure.
        frame("uniform_16M_learned", "uniform", 16_000_000, (695, 695, 695), kernel="gauss3", ao="learned"),
        # The large mixed-phase frame, the benchmark's default.
        frame("mixed_64M_learned", "mixed", 64_000_000, (512, 512, 512), ao="learned"),
        # A batch of trajectory frames of uneven particle counts and grids, plain AO.
        dict(name="trajectory_32", kind="batch", frames=32, nmin=50_000, nmax=2_000_000),
        # One forward + backward pass of the learned AO's training kernels at the default batch size.
        dict(name="train_2048", kind="train", n=2048),
    ]


def frame(name, cloud, n, res, kernel="bump", ao="none", vertex="xyzr", normals="gradient", aggregator=0,
          accumulate="exact", normalize="minmax", cyclic=1, memory="device"):
    return dict(name=name, kind="frame", cloud=cloud, n=int(n), sx=int(res[0]), sy=int(res[1]), sz=int(res[2]),
                kernel=kernel, ao=ao, vertex=vertex, normals=normals, aggregator=aggregator, accumulate=accumulate,
                normalize=normalize, cyclic=cyclic, memory=memory)


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(n, per_voxel, lo, hi):
        # about `per_voxel` particles per voxel, the edges a few per cent apart (odd sizes among them)
        e = (n / per_voxel) ** (1.0 / 3.0)
        return tuple(int(min(hi, max(lo, round(e * rng.uniform(0.93, 1.07))))) for _ in range(3))

    kind = rng.choice(["density", "gauss", "mdao", "aosphere", "intensity", "vector", "liquid", "liquid", "gas",
                       "mixed", "batch", "train"])
    if kind == "density":
        n = log_int(2_000, 1_000_000)
        c = frame("", rng.choice(["uniform", "liquid"]), n, grid(n, rng.uniform(0.05, 0.5), 16, 256),
                  vertex=rng.choice(["xyzr", "xyz", "double"]), cyclic=rng.choice([0, 1]))
    elif kind == "gauss":
        n = log_int(20_000, 1_000_000)
        c = frame("", "uniform", n, grid(n, 0.0477, 32, 280), kernel="gauss3", ao="cone",
                  vertex=rng.choice(["xyz", "xyzr"]))
    elif kind == "mdao":
        n = log_int(50_000, 1_000_000)
        c = frame("", "liquid", n, grid(n, 0.25, 32, 160), ao="mdao", vertex=rng.choice(["xyz+double", "xyzr"]),
                  normals="list")
    elif kind == "aosphere":
        n = log_int(50_000, 2_000_000)
        c = frame("", "liquid", n, grid(n, 0.25, 32, 200), ao="aosphere", normals="list",
                  accumulate=rng.choice(["kahan", "exact"]), normalize="mass")
    elif kind == "intensity":
        n = log_int(50_000, 2_000_000)
        c = frame("", "uniform", n, grid(n, 0.28, 32, 192), aggregator=1, memory=rng.choice(["host", "device"]))
    elif kind == "vector":
        n = log_int(50_000, 1_000_000)
        c = frame("", "liquid", n, grid(n, 0.5, 24, 128), aggregator=2, cyclic=rng.choice([0, 1]), normalize="none")
    elif kind == "liquid":
        n = log_int(100_000, 4_000_000)
        c = frame("", "liquid", n, grid(n, 0.25, 48, 256), ao=rng.choice(["cone", "learned"]))
    elif kind == "gas":
        n = log_int(500_000, 16_000_000)
        c = frame("", "uniform", n, grid(n, 0.0477, 128, 695), kernel="gauss3", ao="learned")
    elif kind == "mixed":
        n = log_int(4_000_000, 60_000_000)
        c = frame("", "mixed", n, grid(n, 0.5, 128, 500), ao="learned")
    elif kind == "batch":
        c = dict(kind="batch", frames=rng.randint(4, 32), nmin=log_int(20_000, 100_000), nmax=log_int(400_000, 2_000_000))
    else:
        c = dict(kind="train", n=log_int(256, 65_536))
    c.pop("name", None)
    return c


# ---- inputs -------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _fcc(ncells, spacing, n, gen, jitter):
    """The first n sites (z-major cells) of an FCC lattice of ncells = (x, y, z) cells, jittered; float64."""
    cx, cy, cz = ncells
    i = torch.arange(n, device="cuda")
    c, b = i // 4, i % 4
    base = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], dtype=torch.float64, device="cuda")
    p = torch.stack([c % cx, (c // cx) % cy, c // (cx * cy)], 1).to(torch.float64) + base[b]
    return p * spacing + jitter * torch.randn(n, 3, generator=gen, device="cuda")


def _cloud(case, gen):
    """(xyzr float32 on the GPU, bbox)"""
    n, cloud = case["n"], case["cloud"]
    out = torch.empty(n, 4, device="cuda")
    if cloud == "uniform":
        edge = float(np.float32(100.0 * (n / 100_000) ** (1.0 / 3.0)))
        out[:, :3] = torch.rand(n, 3, generator=gen, device="cuda") * edge
        out[:, 3] = 0.5
        return out, (0.0, 0.0, 0.0, edge, edge, edge)
    if cloud == "liquid":
        cells = math.ceil((n / 4) ** (1.0 / 3.0) - 1e-9)
        edge = cells * 1.12
        p = _fcc((cells, cells, cells), 1.12, n, gen, 0.08)
        edge = float(np.float32(edge))
        below = float(np.nextafter(np.float32(edge), np.float32(0)))
        out[:, :3] = torch.remainder(p, edge).to(torch.float32).clamp(max=below)
        out[:, 3] = 0.4 + 0.2 * torch.rand(n, generator=gen, device="cuda")
        return out, (0.0, 0.0, 0.0, edge, edge, edge)
    # mixed phase: an FCC slab and, above it, a gas at 1/20 of its density
    half = n // 2
    side = math.ceil((half / 4.0) ** (1.0 / 3.0) * 1.6)
    thick = math.ceil(half / (4.0 * side * side))
    edge, z0 = side * 1.12, thick * 1.12
    height = (n - half) / (4.0 / 1.12 ** 3 / 20.0) / (edge * edge)
    out[:half, :3] = _fcc((side, side, thick), 1.12, half, gen, 0.05).to(torch.float32)
    gas = torch.rand(n - half, 3, generator=gen, device="cuda")
    out[half:, 0] = gas[:, 0] * edge
    out[half:, 1] = gas[:, 1] * edge
    out[half:, 2] = z0 + gas[:, 2] * height
    s = torch.rand(n, generator=gen, device="cuda")
    out[:, 3] = torch.where(s < 0.6, 0.5, torch.where(s < 0.9, 0.8, 1.2))
    lo, hi = out[:, :3].amin(0).tolist(), out[:, :3].amax(0).tolist()
    return out, (*lo, *hi)


def _unit(n, gen):
    v = torch.randn(n, 3, generator=gen, device="cuda")
    return v / v.norm(dim=1, keepdim=True)


def _frame_inputs(case, seed):
    """Everything the frame's values depend on: xyzr as the library reads it (float32), bbox, and the lists' arrays."""
    gen = _gen(seed)
    xyzr, bbox = _cloud(case, gen)
    n = case["n"]
    d = dict(xyzr=xyzr, bbox=bbox)
    if case["vertex"] != "xyzr":
        xyzr[:, 3] = 0.5
    if case["normals"] == "list" or case["aggregator"] == 2:
        d["normals"] = _unit(n, gen)
    if case["aggregator"] == 1:
        d["colour"] = torch.rand(n, generator=gen, device="cuda")
    if case["ao"] == "learned":
        d["weights"] = _weights(gen)
    return d


def _weights(gen):
    """A network as training leaves it: hidden layers of the library's initial scale, a wider last layer."""
    w = torch.rand(p2v.MLP_PARAMS, generator=gen, device="cuda") * 2 - 1
    h, k = p2v.MLP_HIDDEN, p2v.MLP_INPUTS
    o1, o2, o3 = h * k + h, h * k + h + h * h + h, p2v.MLP_PARAMS - 1
    w[:o1] *= 2.0 / math.sqrt(k)
    w[o1:o2] *= 2.0 / math.sqrt(h)
    w[o2:o3] *= 4.0 / math.sqrt(h)
    return w


def _lists(case, d, ao):
    n, xyzr = case["n"], d["xyzr"]
    host = case["memory"] == "host"

    def place(t):
        return t.cpu().numpy() if host else t

    def part(key, a, b):
        return place(d[key][a:b].contiguous()) if key in d else None

    if case["vertex"] == "xyz+double":
        cuts = [(0, n // 3, p2v.VERTDATA_FLOAT_XYZ), (n // 3, n, p2v.VERTDATA_DOUBLE_XYZ)]
    else:
        kind = {"xyzr": p2v.VERTDATA_FLOAT_XYZR, "xyz": p2v.VERTDATA_FLOAT_XYZ, "double": p2v.VERTDATA_DOUBLE_XYZ}
        cuts = [(0, n, kind[case["vertex"]])]
    out = []
    for a, b, vt in cuts:
        data = xyzr[a:b] if vt == p2v.VERTDATA_FLOAT_XYZR else xyzr[a:b, :3]
        data = data.to(torch.float64) if vt == p2v.VERTDATA_DOUBLE_XYZ else data
        kw = {}
        if "colour" in d:
            kw = dict(colour=part("colour", a, b), colour_type=p2v.COLDATA_FLOAT_I)
        out.append(p2v.ParticleList(place(data.contiguous()), vt, count=b - a, global_radius=0.5,
                                    normals=part("normals", a, b), ao_out=None if ao is None else ao[a:b], **kw))
    return out


def _params(case):
    p = dict(sizex=case["sx"], sizey=case["sy"], sizez=case["sz"], cyclX=case["cyclic"], cyclY=case["cyclic"],
             cyclZ=case["cyclic"], sigma=1.0, aggregator=case["aggregator"],
             kernel=p2v.KERNEL_GAUSS3 if case["kernel"] == "gauss3" else p2v.KERNEL_BUMP,
             accumulate=p2v.ACCUM_KAHAN if case["accumulate"] == "kahan" else p2v.ACCUM_EXACT,
             normalize=int(case["normalize"] == "minmax"), mass_normalize=int(case["normalize"] == "mass"))
    if case["ao"] == "cone":
        p.update(AO_BENCH, ao_mode=p2v.AO_CONE)
    elif case["ao"] == "learned":
        p.update(AO_BENCH, ao_mode=p2v.AO_LEARNED)
    elif case["ao"] == "mdao":
        p.update(ao_mode=p2v.AO_CONE, ao_volume=p2v.AOVOL_MDAO)
    elif case["ao"] == "aosphere":
        p.update(ao_mode=p2v.AO_AOSPHERE_AXES)
    return p


def _blobs(case):
    """(count, grid edge) of every trajectory frame: counts spread over their logarithm, edges in turn."""
    f, lo, hi = case["frames"], case["nmin"], case["nmax"]
    out = []
    for k in range(f):
        u = ((k * 7) % f + 0.5) / f  # a fixed order that mixes small and large frames
        out.append((int(math.exp(math.log(lo) + u * (math.log(hi) - math.log(lo)))), EDGES[(k * 3) % len(EDGES)]))
    return out


def _blob_frame(n, res, gen):
    """1 to 8 Gaussian blobs (standard deviations 2 to 10) of a frame whose extent suits a grid of `res` voxels of 0.5."""
    k = int(torch.randint(1, 9, (1,), generator=gen, device="cuda"))
    edge = max(10.0, 0.5 * res - 30.0)
    centres = torch.rand(k, 3, generator=gen, device="cuda") * edge
    std = 2.0 + 8.0 * torch.rand(k, generator=gen, device="cuda")
    share = torch.rand(k, generator=gen, device="cuda") + 0.05
    which = torch.multinomial(share, n, replacement=True, generator=gen)
    out = torch.empty(n, 4, device="cuda")
    out[:, :3] = centres[which] + torch.randn(n, 3, generator=gen, device="cuda") * std[which, None]
    out[:, 3] = 0.5
    lo, hi = out[:, :3].amin(0).tolist(), out[:, :3].amax(0).tolist()
    return out, (*lo, *hi)


def _train_inputs(case, seed):
    gen = _gen(seed)
    n = case["n"]
    x = torch.rand(n, p2v.MLP_INPUTS, generator=gen, device="cuda")
    x[:, -6:-3] = _unit(n, gen)
    return x, torch.rand(n, generator=gen, device="cuda"), _weights(gen)


def prepare(case, seed):
    if case["kind"] == "train":
        x, t, w = _train_inputs(case, seed)
        ctx = p2v.Context(0)
        ctx.mlp_set_weights(w.cpu().numpy())
        return dict(kind="train", ctx=ctx, x=x.cpu().numpy(), t=t.cpu().numpy())
    if case["kind"] == "batch":
        gen = _gen(seed)
        ctx = p2v.Context(0)
        ctx.set_params(normalize=1, ao_mode=p2v.AO_CONE, **AO_BENCH)
        frames = []
        for n, res in _blobs(case):
            xyzr, bbox = _blob_frame(n, res, gen)
            ao = torch.empty(n, device="cuda")
            frames.append(dict(lists=[p2v.ParticleList(xyzr, ao_out=ao)], bbox=bbox, size=(res, res, res),
                               out=torch.empty(res, res, res, device="cuda")))
        torch.cuda.synchronize()
        return dict(kind="batch", ctx=ctx, frames=frames)
    d = _frame_inputs(case, seed)
    shape = (case["sz"], case["sy"], case["sx"]) + ((3,) if case["aggregator"] == 2 else ())
    if case["memory"] == "host":
        module = p2v.ParticlesToDensity(0, **_params(case))
        state = dict(kind="host", module=module, lists=_lists(case, d, None), bbox=d["bbox"])
    else:
        ctx = p2v.Context(0)
        ctx.set_params(**_params(case))
        if "weights" in d:
            ctx.mlp_set_weights(d["weights"].cpu().numpy())
        ao = torch.empty(case["n"], device="cuda") if case["ao"] != "none" else None
        state = dict(kind="frame", ctx=ctx, lists=_lists(case, d, ao), bbox=d["bbox"], ao=ao,
                     grid=torch.empty(shape, device="cuda"))
    torch.cuda.synchronize()
    return state


def run(state):
    if state["kind"] == "train":
        grad, loss = state["ctx"].mlp_gradients(state["x"], state["t"])
        return {"grad": grad, "loss": float(loss)}
    if state["kind"] == "batch":
        state["ctx"].run_batch(state["frames"])
        return {"grids": [f["out"] for f in state["frames"]], "ao": [f["lists"][0].ao_out for f in state["frames"]]}
    if state["kind"] == "host":
        volume, _ = state["module"].get_data(state["lists"], state["bbox"])
        return {"grid": volume}
    state["ctx"].run_frame(state["lists"], state["bbox"], state["grid"])
    out = {"grid": state["grid"]}
    if state["ao"] is not None:
        out["ao"] = state["ao"]
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------

def _per_particle_nodes(case, hx):
    """In-support nodes of an average particle (mean cube of the kernel's radius over the voxel volume)."""
    if case["kernel"] == "gauss3":
        r3 = 1.5 ** 3
    elif case["vertex"] != "xyzr" or case["cloud"] == "uniform":
        r3 = 0.5 ** 3
    else:
        r3 = 0.5 ** 3 * 1.04 if case["cloud"] == "liquid" else 0.6 * 0.5 ** 3 + 0.3 * 0.8 ** 3 + 0.1 * 1.2 ** 3
    return 4.0 / 3.0 * math.pi * r3 / hx


def work(case):
    if case["kind"] == "train":
        per = 2 * (p2v.MLP_INPUTS * p2v.MLP_HIDDEN + p2v.MLP_HIDDEN ** 2 + p2v.MLP_HIDDEN)
        return {"bytes": 4 * case["n"] * (p2v.MLP_INPUTS + 1) + 8 * p2v.MLP_PARAMS, "flops": 3 * per * case["n"]}
    if case["kind"] == "batch":
        b = f = 0
        for n, res in _blobs(case):
            b += n * (16 + 4) + 4 * res ** 3
            f += n * (20 * 8 + 8 * 32 * 20)
        return {"bytes": b, "flops": f}
    n, v = case["n"], case["sx"] * case["sy"] * case["sz"]
    record = {"xyzr": 16, "xyz": 12, "double": 24, "xyz+double": 20}[case["vertex"]]
    comps = 3 if case["aggregator"] == 2 else 1
    b = n * record + 4 * comps * v
    if case["normals"] == "list" or case["aggregator"] == 2:
        b += 12 * n
    if case["aggregator"] == 1:
        b += 4 * n
    if case["cloud"] == "uniform":
        volume = 10.0 * n
    elif case["cloud"] == "liquid":
        volume = (math.ceil((n / 4) ** (1.0 / 3.0) - 1e-9) * 1.12) ** 3
    else:
        volume = (n // 2) * 1.12 ** 3 / 4 * 21
    f = 20 * n * _per_particle_nodes(case, volume / v) * (1 if comps == 1 else 4)
    if case["ao"] != "none":
        b += 4 * n
    if case["ao"] == "cone":
        f += n * 8 * 32 * 20
    elif case["ao"] == "mdao":
        f += n * 3 * 8 * 20
    elif case["ao"] == "learned":
        f += n * (48 * 20 + 2 * (54 * 64 + 64 * 64 + 64))
    elif case["ao"] == "aosphere":
        f += n * 80
    return {"bytes": int(b), "flops": int(f)}


# ---- the same results in 64 bits ---------------------------------------------------------------------------------

CHUNK = 1 << 20


def _density64(xyzr, weights, bbox, res, cyclic, kernel):
    """Kernel sums of the particles on the node grid, one volume per weight column (None: unweighted): (z, y, x) float64.
    The reference's integer decisions (cell, footprint) are taken in float32 as it takes them; distances are exact."""
    dev = xyzr.device
    nw = 1 if weights is None else weights.shape[1]
    grid = torch.zeros(nw, res[0] * res[1] * res[2], dtype=torch.float64, device=dev)
    lo = [float(np.float32(v)) for v in bbox[:3]]
    hi = [float(np.float32(v)) for v in bbox[3:]]
    h = [(hi[a] - lo[a]) / (res[a] - 1) for a in range(3)]
    h32 = [float(np.float32(np.float32(hi[a]) - np.float32(lo[a])) / np.float32(res[a] - 1)) for a in range(3)]
    for c0 in range(0, xyzr.shape[0], 4 * CHUNK):
        p = xyzr[c0:c0 + 4 * CHUNK]
        r = p[:, 3].to(torch.float64)
        w = None if weights is None else weights[c0:c0 + 4 * CHUNK].to(torch.float64)
        cell, reach, base = [], [], []
        for a in range(3):
            q = (p[:, a] - lo[a]) / torch.tensor(h32[a], dtype=torch.float32, device=dev)
            if kernel == "gauss3":
                cell.append(q.floor().to(torch.int64))
                reach.append(torch.full_like(cell[-1], int(math.ceil(3.0 * float(r.max()) / h[a])) + 1))
            else:
                cell.append(q.trunc().to(torch.int64))
                reach.append((p[:, 3] / torch.tensor(h32[a], dtype=torch.float32, device=dev)).ceil().to(torch.int64))
            base.append(p[:, a].to(torch.float64) - lo[a])
        far = [int(x.max()) for x in reach]

        def axis(a, o):
            k = cell[a] + o
            ok = (reach[a] >= abs(o))
            if cyclic:
                idx = torch.remainder(k, res[a])
            else:
                ok = ok & (k >= 0) & (k < res[a])
                idx = k.clamp(0, res[a] - 1)
            return idx, (k.to(torch.float64) * h[a] - base[a]) ** 2, ok

        eps2 = (3.0 * r if kernel == "gauss3" else r) ** 2
        ax = [{o: axis(a, o) for o in range(-far[a], far[a] + 1)} for a in range(3)]
        for oz in range(-far[2], far[2] + 1):
            for oy in range(-far[1], far[1] + 1):
                iz, dz, kz = ax[2][oz]
                iy, dy, ky = ax[1][oy]
                row, dyz, kyz = iz * res[1] + iy, dy + dz, ky & kz
                for ox in range(-far[0], far[0] + 1):
                    ix, dx, kx = ax[0][ox]
                    d2 = dyz + dx
                    hit = torch.nonzero(kyz & kx & (d2 < eps2)).squeeze(1)
                    if hit.numel() == 0:
                        continue
                    x = d2[hit] / eps2[hit]
                    v = torch.exp(-4.5 * x) - math.exp(-4.5) if kernel == "gauss3" else torch.exp(-1.0 / (1.0 - x))
                    v = torch.where(v < 2.0 ** -149, 0.0, v)  # a kernel value is a float: tails below its range are zero
                    node = row[hit] * res[0] + ix[hit]
                    for k in range(nw):
                        grid[k].index_add_(0, node, v if w is None else v * w[hit, k])
    return grid.view(nw, res[2], res[1], res[0])


def _sample64(vol, q, edge):
    """GL LINEAR sample of a (z, y, x) volume at normalised points q (n, 3): border 0, or clamped to the edge."""
    dims = (vol.shape[2], vol.shape[1], vol.shape[0])
    flat = vol.reshape(-1)
    i0, fr = [], []
    for a in range(3):
        c = q[:, a] * dims[a] - 0.5
        f = torch.floor(c)
        i0.append(f.to(torch.int64))
        fr.append(c - f)
    out = torch.zeros_like(q[:, 0])
    for corner in range(8):
        w, idx, ok = None, [], None
        for a in range(3):
            b = (corner >> a) & 1
            i = i0[a] + b
            wa = fr[a] if b else 1.0 - fr[a]
            w = wa if w is None else w * wa
            inside = (i >= 0) & (i < dims[a])
            ok = inside if ok is None else ok & inside
            idx.append(i.clamp(0, dims[a] - 1))
        v = flat[(idx[2] * dims[1] + idx[1]) * dims[0] + idx[0]]
        out += w * (v if edge else torch.where(ok, v, 0.0))
    return out


def _gradient_normals64(grid, xyz, lo, h, res):
    """Unit vectors down the density gradient (periodic axes), trilinear between the nodes' central differences."""
    flat = grid.reshape(-1)
    i0, i1, fr = [], [], []
    for a in range(3):
        u = ((xyz[:, a] - lo[a]) / h[a]).clamp(0.0, res[a] - 1.0)
        k = u.floor().to(torch.int64).clamp(max=res[a] - 1)
        i0.append(k)
        i1.append((k + 1).clamp(max=res[a] - 1))
        fr.append(u - k)
    g = torch.zeros_like(xyz)
    for corner in range(8):
        idx = [(i1 if (corner >> a) & 1 else i0)[a] for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (fr[a] if (corner >> a) & 1 else 1.0 - fr[a])
        for a in range(3):
            up, dn = list(idx), list(idx)
            up[a], dn[a] = torch.remainder(idx[a] + 1, res[a]), torch.remainder(idx[a] - 1, res[a])
            d = flat[(up[2] * res[1] + up[1]) * res[0] + up[0]] - flat[(dn[2] * res[1] + dn[1]) * res[0] + dn[0]]
            g[:, a] += w * d / (2.0 * h[a])
    l = g.norm(dim=1, keepdim=True)
    return torch.where(l > 0, -g / l, 0.0)


def _cone_ao64(xyzr, grid, bbox, res, weights=None):
    """The cone march (AO_BENCH) of every particle over the pyramid of a (z, y, x) grid, gradient normals; with
    weights, the network on the march's samples at six of its steps instead."""
    lo = [float(np.float32(v)) for v in bbox[:3]]
    hi = [float(np.float32(v)) for v in bbox[3:]]
    h = [(hi[a] - lo[a]) / (res[a] - 1) for a in range(3)]
    levels = [grid.clamp(0.0, 1.0)]
    for _ in range(2):
        levels.append(torch.nn.functional.avg_pool3d(levels[-1][None, None], 2)[0, 0])
    apex, cones, steps = math.radians(50.0), 8, 32
    edge = 2.0 * math.tan(0.5 * apex)
    height, radius = math.sqrt(1.0 - edge * edge / 12.0), edge / (2.0 * math.sin(math.pi / cones))
    dirs = []
    for k in range(cones):
        v = (math.cos(k / cones * 2 * math.pi) * radius, height, math.sin(k / cones * 2 * math.pi) * radius)
        l = math.sqrt(sum(c * c for c in v))
        dirs.append([c / l for c in v])
    t = [0.0101 * (0.8 / 0.0101) ** (k / steps) for k in range(steps)]
    lod = [min(max(math.log2(x * edge * min(res)), 0.0), 2.0) for x in t]

    def visible(u, d, k):
        q = u + t[k] * d
        l0 = min(int(lod[k]), 2)
        f = lod[k] - l0
        v = _sample64(levels[l0], q, False)
        return v if f <= 0 or l0 == 2 else (1.0 - f) * v + f * _sample64(levels[l0 + 1], q, False)

    out = torch.empty(xyzr.shape[0], dtype=torch.float64, device=xyzr.device)
    for c0 in range(0, xyzr.shape[0], CHUNK):
        p = xyzr[c0:c0 + CHUNK].to(torch.float64)
        nn = _gradient_normals64(grid, p[:, :3], lo, h, res)
        none = nn.norm(dim=1) == 0
        x = p[:, :3] + p[:, 3:] * nn
        xn = x / x.norm(dim=1, keepdim=True)
        ex = torch.linalg.cross(nn, xn)
        ez = torch.linalg.cross(ex, nn)
        u = torch.stack([(x[:, a] - (lo[a] - 0.5 * h[a])) / (res[a] * h[a]) for a in range(3)], 1)
        if weights is None:
            total = torch.zeros_like(u[:, 0])
            for d in dirs:
                v = ex * d[0] + nn * d[1] + ez * d[2]
                acc = torch.zeros_like(total)
                for k in range(steps):
                    acc = torch.where(acc > 0.99, acc, acc + (1.0 - acc) * visible(u, v, k))
                total += acc
            ao = 1.0 - (total / cones).clamp(0.0, 1.0)
        else:
            f = []
            for d in dirs:
                v = ex * d[0] + nn * d[1] + ez * d[2]
                f += [visible(u, v, round(j * (steps - 1) / 5)) for j in range(6)]
            ao = _forward64(weights, torch.cat([torch.stack(f, 1), nn, u], 1))
        out[c0:c0 + CHUNK] = torch.where(none, 1.0, ao)
    return out


def _forward64(w, x):
    h, k = p2v.MLP_HIDDEN, p2v.MLP_INPUTS
    s = torch.nn.functional.silu
    o = [0, h * k, h * k + h, h * k + h + h * h, h * k + 2 * h + h * h, h * k + 3 * h + h * h]
    a = s(x @ w[o[0]:o[1]].view(h, k).T + w[o[1]:o[2]])
    a = s(a @ w[o[2]:o[3]].view(h, h).T + w[o[3]:o[4]])
    return torch.sigmoid(a @ w[o[4]:o[5]] + w[o[5]])


def _aosphere64(xyzr, normals, bbox):
    """AOSphereRenderer's main-axes AO with its defaults: a 32^3 volume with a one-voxel border, three taps."""
    s, si = 32, 30
    lo = torch.tensor(bbox[:3], dtype=torch.float64, device=xyzr.device)
    ext = torch.tensor(bbox[3:], dtype=torch.float64, device=xyzr.device) - lo
    q = (xyzr[:, :3] - lo.float()) / ext.float() * float(si)
    c = q.to(torch.int64).clamp(0, si - 1) + 1
    p, r = xyzr[:, :3].to(torch.float64), xyzr[:, 3].to(torch.float64)
    vol = torch.zeros(s ** 3, dtype=torch.float64, device=xyzr.device)
    vol.index_add_(0, (c[:, 2] * s + c[:, 1]) * s + c[:, 0], 4.0 / 3.0 * math.pi * r ** 3 / float((ext / si).prod()))
    vol = vol.view(s, s, s)
    full = ext / (1.0 - 2.0 / s)
    at = (p - (lo - full / s)) / full
    off = (r[:, None] + 0.5 * ext / s) / full
    nn = normals.to(torch.float64)
    nn = nn / nn.norm(dim=1, keepdim=True)
    ao = torch.zeros_like(r)
    for a in range(3):
        x = at.clone()
        x[:, a] += torch.where(nn[:, a] > 0, off[:, a], -off[:, a])
        ao += nn[:, a] ** 2 * (1.0 - _sample64(vol, x, True))
    return ao


def _minmax(v, lo, hi):
    return (v - lo) / (hi - lo)


def exact(case, seed):
    if case["kind"] == "train":
        x, t, w = (v.to(torch.float64) for v in _train_inputs(case, seed))
        w.requires_grad_(True)
        loss = ((_forward64(w, x) - t) ** 2).mean()
        loss.backward()
        return {"grad": w.grad.cpu().numpy(), "loss": float(loss.detach())}
    if case["kind"] == "batch":
        gen = _gen(seed)
        grids, aos = [], []
        for n, res in _blobs(case):
            xyzr, bbox = _blob_frame(n, res, gen)
            v = _density64(xyzr, None, bbox, (res,) * 3, True, "bump")[0]
            grids.append(_minmax(v, v.min(), v.max()))
            aos.append(_cone_ao64(xyzr, grids[-1], bbox, (res,) * 3))
        return {"grids": grids, "ao": aos}
    d = _frame_inputs(case, seed)
    res, xyzr, bbox = (case["sx"], case["sy"], case["sz"]), d["xyzr"], d["bbox"]
    if case["aggregator"] == 2:
        v = _density64(xyzr, torch.cat([d["normals"], torch.ones_like(xyzr[:, :1])], 1), bbox, res, case["cyclic"],
                       case["kernel"])
        v3 = (v[:3] / torch.where(v[3] == 0, 1.0, v[3])).permute(1, 2, 3, 0)
        return {"grid": v3.contiguous()}
    w = d["colour"][:, None] if case["aggregator"] == 1 else None
    v = _density64(xyzr, w, bbox, res, case["cyclic"], case["kernel"])[0]
    if case["normalize"] == "mass":
        h = [(float(np.float32(bbox[a + 3])) - float(np.float32(bbox[a]))) / (res[a] - 1) for a in range(3)]
        v = v * (case["n"] / (float(v.sum()) * h[0] * h[1] * h[2]))
    elif case["normalize"] == "minmax":
        v = _minmax(v, v.min(), v.max())
    out = {"grid": v.cpu().numpy() if case["memory"] == "host" else v}
    if case["ao"] in ("cone", "learned"):
        out["ao"] = _cone_ao64(xyzr, v, bbox, res, d["weights"].to(torch.float64) if case["ao"] == "learned" else None)
    elif case["ao"] == "aosphere":
        out["ao"] = _aosphere64(xyzr, d["normals"], bbox)
    elif case["ao"] == "mdao":
        out["ao"] = None  # the 8-bit occupancy volume is defined by its own rounding
    return out
