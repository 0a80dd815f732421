"""Timed cases of the framework: whole simulations from host arrays through
`GrainHandler`, and the allocation-free convolution of one box.

A network case is what a user's program does for one microstructure: create a
handler, load the input from (page-locked) host memory, initialise, run a
fixed number of timesteps and read every grain's statistics, once at the end
or after every step as a monitoring program does.  A handler takes one
network, so there is none to keep between runs: the program holds the input
arrays and the settings.  The networks are Poisson-Voronoi tessellations at
20 to 32 grid points per grain (the reference's resolution), a Matern
cluster mix for uneven grain sizes, and polygon input as a restart reads it.
"""
import math

import numpy as np
import torch

from gragles2d_b200 import gg
from gragles2d_b200 import microstructure as ms

BORDER = 7  # DomainBorderSize, the default

STATS = np.dtype([("id", "i4"), ("state", "i4"), ("motion_regular", "i4"), ("intersects_boundary", "i4"),
                  ("n_neighbours", "i4"), ("contour_points", "i4"), ("box", "i4", (4,)), ("area", "f8"),
                  ("energy", "f8"), ("perimeter", "f8"), ("mean_da", "f8")])


def listed():
    return [
        # one box on a caller's own buffers: a box of ordinary size, and the largest the entry point takes
        {"name": "box_45", "kind": "box", "n": 45},
        {"name": "box_128", "kind": "box", "n": 128},
        # a small sample followed step by step: launches and latency count
        network("small_60_each", "batched", 60, 160, "iso", 40, read="each"),
        # the 1,000-grain isotropic benchmark network in both forms
        network("iso_1000", "batched", 1000, 800, "iso", 25),
        network("plain_iso_1000", "plain", 1000, 800, "iso", 12),
        # the bench's network, its statistics read after every step
        network("rs_20000_each", "batched", 20000, 3600, "rs", 20, read="each"),
        # mobility model and triple-junction drag, at scale
        network("drag_50000", "batched", 50000, 5600, "drag", 8),
        # the largest: uneven grain sizes
        network("clustered_100000", "batched", 100000, 8192, "rs", 4, source="clustered"),
        # recrystallisation-like runs: the stored-energy driving force, on an odd grid
        network("stored_2000", "batched", 2000, 1131, "stored", 15),
        # a run resumed from contours
        network("contours_1500", "batched", 1500, 968, "rs", 15, source="contours"),
        # the FP64 form that reproduces the reference, at the profiling case's size
        network("plain_rs_5000", "plain", 5000, 1800, "rs", 8),
        # calibration: areas with their parameter derivatives
        network("tangent_300", "plain", 300, 433, "drag", 8, tangents=True),
    ]


def network(name, form, grains, grid, physics, steps, source="voronoi", read="end", tangents=False):
    case = {"kind": "network", "form": form, "grains": grains, "grid": grid, "physics": physics, "steps": steps,
            "source": source, "read": read, "tangents": tangents}
    return {"name": name, **case} if name else case


def log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    if rng.random() < 0.15:
        return {"kind": "box", "n": log_int(rng, 2, 128)}
    form = "batched" if rng.random() < 0.65 else "plain"
    tangents = form == "plain" and rng.random() < 0.3
    most, budget = (100000, 400000) if form == "batched" else (600, 2400) if tangents else (5000, 40000)
    source = "voronoi" if tangents else rng.choice(["voronoi"] * 3 + ["contours"] + ["clustered"] * (form == "batched"))
    # a contour file is read on the host; an uneven network takes many grains to be one
    grains = log_int(rng, 5000 if source == "clustered" else 30, min(most, 4000) if source == "contours" else most)
    per_grain = rng.uniform(23, 29)
    if source == "contours":
        per_grain = int(per_grain)  # NumberOfPointsPerGrain is a whole number
    physics = rng.choice(["iso", "rs", "rs", "drag"] if tangents or source == "contours"
                         else ["iso", "rs", "rs", "drag", "stored", "magnetic"])
    steps = min(rng.randint(3, 40), max(2, budget // grains))
    return network("", form, grains, int(math.sqrt(grains) * per_grain), physics, steps, source,
                   rng.choice(["each", "end"]), tangents)


# ---- inputs ----------------------------------------------------------------

def cluster_seeds(rng, n, nn):
    """Matern cluster mix of the uneven-box network: 90% daughters, 60 per cluster, radius 100 grid spacings."""
    daughters = int(round(0.9 * n))
    parents = rng.random((max(1, daughters // 60), 2))
    owner = rng.integers(0, len(parents), 2 * daughters)
    r, t = 100 / nn * np.sqrt(rng.random(2 * daughters)), 2 * np.pi * rng.random(2 * daughters)
    pts = parents[owner] + np.stack([r * np.cos(t), r * np.sin(t)], axis=1)
    pts = pts[(pts >= 0).all(axis=1) & (pts < 1).all(axis=1)][:daughters]
    return np.concatenate([pts, rng.random((n - len(pts), 2))])


def nearest_seed(seeds, nn):
    """Labels 1..n of the nn x nn pixel centres by nearest seed, on the GPU: blocks of 512 x 512 pixels, in each
    32 x 32 tile only the seeds that can be nearest to one of its pixels."""
    dev, big, small = "cuda", 512, 32
    s = torch.tensor(seeds, device=dev) * nn
    out = torch.empty(nn, nn, dtype=torch.int32, device=dev)
    half = small / 2
    per = torch.arange(small, device=dev, dtype=torch.float64) + 0.5
    py, px = [a.reshape(-1) for a in torch.meshgrid(per, per, indexing="ij")]
    first_reach = 6 * nn / math.sqrt(len(seeds))
    for y0 in range(0, nn, big):
        for x0 in range(0, nn, big):
            ny, nx = -(-min(big, nn - y0) // small), -(-min(big, nn - x0) // small)
            ty, tx = [a.reshape(-1) for a in torch.meshgrid(
                y0 + small * torch.arange(ny, device=dev, dtype=torch.float64),
                x0 + small * torch.arange(nx, device=dev, dtype=torch.float64), indexing="ij")]
            reach = first_reach
            while True:
                near = ((s[:, 0] > x0 - reach) & (s[:, 0] < x0 + big + reach) &
                        (s[:, 1] > y0 - reach) & (s[:, 1] < y0 + big + reach)).nonzero().reshape(-1)
                if len(near) == len(seeds):
                    break
                if len(near):
                    d = torch.cdist(torch.stack([tx + half, ty + half], 1), s[near])
                    if float(d.min(1).values.max()) + 3 * half <= reach:
                        break
                reach *= 2
            c = s[near]
            d = torch.cdist(torch.stack([tx + half, ty + half], 1), c)
            k = int((d <= d.min(1, keepdim=True).values + 2.9 * half).sum(1).max())
            cand = d.topk(k, largest=False).indices
            lab = torch.empty(ny * nx, small * small, dtype=torch.int32, device=dev)
            step = max(1, 40_000_000 // (k * small * small))
            for t in range(0, ny * nx, step):
                q = c[cand[t:t + step]]
                dx = (tx[t:t + step, None] + px)[:, :, None] - q[:, None, :, 0]
                dy = (ty[t:t + step, None] + py)[:, :, None] - q[:, None, :, 1]
                best = (dx * dx + dy * dy).argmin(2)
                lab[t:t + step] = near[cand[t:t + step].gather(1, best)].to(torch.int32) + 1
            lab = lab.reshape(ny, nx, small, small).permute(0, 2, 1, 3).reshape(ny * small, nx * small)
            out[y0:y0 + big, x0:x0 + big] = lab[:min(big, nn - y0), :min(big, nn - x0)]
    return out


def grain_boxes(labels, n):
    """(xmin, xmax, ymin, ymax, pixel count) of every grain, as a .uds header holds them."""
    nn, dev = labels.shape[0], labels.device
    g = labels.reshape(-1).long() - 1
    at = torch.arange(nn, device=dev, dtype=torch.int32)
    x, y = at.repeat(nn), at.repeat_interleave(nn)
    box = torch.zeros(n, 5, dtype=torch.int32, device=dev)
    for k, (v, how) in enumerate([(x, "amin"), (x, "amax"), (y, "amin"), (y, "amax")]):
        box[:, k] = torch.zeros(n, dtype=torch.int32, device=dev).scatter_reduce(0, g, v, how, include_self=False)
    box[:, 4] = torch.bincount(g, minlength=n).to(torch.int32)
    return box


def lattice_contours(rng, case):
    """Closed polygons of a jittered honeycomb (rows of staggered cells) that tile the domain, with a point every
    grid spacing or so along each edge, as a restart file's contours have."""
    n, nn = case["grains"], case["grid"]
    rows = max(2, int(math.sqrt(n)))
    cols = [n // rows + (j < n % rows) for j in range(rows)]
    # x positions of the cell walls of every row, staggered and jittered; a row boundary carries the wall ends of both rows
    walls = []
    for j, c in enumerate(cols):
        w = (np.arange(c + 1) + np.where(np.arange(c + 1) % c == 0, 0.0, 0.25 * (-1) ** j)) / c
        w[1:c] += rng.uniform(-0.12, 0.12, c - 1) / c
        walls.append(w)
    lines = []
    for j in range(rows + 1):
        x = np.unique(np.concatenate([walls[k] for k in (j - 1, j) if 0 <= k < rows]))
        y = np.full(len(x), j / rows)
        if 0 < j < rows:
            y += rng.uniform(-0.12, 0.12, len(x)) / rows
        lines.append((x, y))
    polygons = []
    for j in range(rows):
        (xb, yb), (xt, yt) = lines[j], lines[j + 1]
        for i in range(cols[j]):
            lo, hi = walls[j][i], walls[j][i + 1]
            b, t = (xb >= lo) & (xb <= hi), (xt >= lo) & (xt <= hi)
            p = np.concatenate([np.stack([xb[b], yb[b]], 1), np.stack([xt[t], yt[t]], 1)[::-1]])
            p = np.concatenate([p, p[:1]])
            m = np.maximum(1, (np.hypot(*(p[1:] - p[:-1]).T) * nn).astype(int))
            f = np.concatenate([np.arange(k) / k for k in m])
            q = np.repeat(p[:-1], m, 0) + f[:, None] * np.repeat(p[1:] - p[:-1], m, 0)
            polygons.append(np.concatenate([q, p[:1]]))
    return polygons


def settings(case):
    over = {"precision": gg.PRECISION_BATCHED if case["form"] == "batched" else gg.PRECISION_PLAIN,
            "is_isotropic_network": int(case["physics"] == "iso"), "analysis_timestep": 100,
            "constant_sector_radius": 3.0, "interpolating_sector_radius": 2.0,
            "number_of_particles": case["grains"],
            "number_of_points_per_grain": int(case["grid"] / math.sqrt(case["grains"]) + 1e-9)}
    if case["physics"] == "drag":
        over.update(use_mobility_model=1, triple_point_drag=0.1 / (0.69 / math.sqrt(case["grains"])))
    if case["physics"] == "stored":
        over.update(use_stored_elastic_energy=1, dislocation_energy_per_m=1.0, box_default_stored_elastic_energy=500.0)
    if case["source"] == "clustered":
        over["list_capacity"] = 128  # uneven grains have longer neighbour lists than the default holds
    s = gg.Settings(**over)
    if case["source"] == "contours":
        s.p.microstructure_gen_mode = 0
    if case["physics"] == "magnetic":
        s.p.use_magnetic_field = 1
        s.p.vacuum_permeability, s.p.delta_mag_sys, s.p.magnetic_force_field = 1.0, 1600.0, 1.0
        s.p.magnetic_vector[0], s.p.magnetic_vector[2] = 0.6, 0.8
    return s


def microstructure(case, seed):
    """Labels (on the GPU), Euler angles, boxes and stored energies of a voxelized case."""
    rng = np.random.Generator(np.random.PCG64([seed, case["grains"], case["grid"]]))
    n = case["grains"]
    seeds = cluster_seeds(rng, n, case["grid"]) if case["source"] == "clustered" else rng.random((n, 2))
    euler = ms.quaternion_to_bunge(ms.shoemake_quaternions(rng, n))
    labels = nearest_seed(seeds, case["grid"])
    stored = rng.uniform(0, 3000, n) if case["physics"] == "stored" else None
    return labels, euler, grain_boxes(labels, n).cpu().numpy(), stored


def box_input(case, seed):
    """A grain's signed distance field, clamped to +-delta as the framework keeps it, and its network's grid."""
    n = case["n"]
    rng = np.random.Generator(np.random.PCG64([seed, n]))
    nn = 3600
    y, x = np.mgrid[0:n, 0:n]
    r = max(0.5, n / 2 - BORDER) * rng.uniform(0.8, 1.2) * (
        1 + 0.1 * np.cos(3 * np.arctan2(y - n / 2, x - n / 2) + rng.uniform(0, 6)))
    d = (r - np.hypot(x - n / 2 + rng.uniform(-1, 1), y - n / 2 + rng.uniform(-1, 1))) / nn
    return np.clip(d, -BORDER / nn, BORDER / nn), 0.8 / nn ** 2 * 25 / 2 / 5.0, nn


def prepare(case, seed):
    if case["kind"] == "box":
        field, dt, nn = box_input(case, seed)
        d = torch.tensor(field, device="cuda")
        return {"case": case, "in": d, "out": torch.empty_like(d), "dt": dt, "nn": nn}
    state = {"case": case, "settings": settings(case)}
    if case["source"] == "contours":
        rng = np.random.Generator(np.random.PCG64([seed, case["grains"]]))
        state["contours"] = lattice_contours(rng, case)
        state["quats"] = ms.shoemake_quaternions(rng, case["grains"])
        return state
    labels, state["euler"], state["boxes"], state["stored"] = microstructure(case, seed)
    ids = torch.empty(labels.shape, dtype=torch.int32, pin_memory=True)
    ids.copy_(labels)
    state["ids"] = ids.numpy()
    state["keep"] = ids
    return state


# ---- one pass --------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "box":
        gg.convolve_box_static(state["in"].data_ptr(), state["out"].data_ptr(), case["n"], state["dt"], state["nn"],
                               torch.cuda.current_stream().cuda_stream)
        return {"out": state["out"]}
    h = gg.GrainHandler(state["settings"])
    try:
        if case["source"] == "contours":
            h.load_contours(state["contours"], state["quats"])
        else:
            h.load_voxels(state["ids"], state["euler"], state["boxes"], state["stored"])
        if case["tangents"]:
            h.enable_tangents()
        h.distanceInitialisation()
        h.find_neighbors()
        stats = None
        if case["read"] == "each":
            for _ in range(case["steps"]):
                h.step(1)
                stats = h.grain_stats(stats)
        else:
            h.step(case["steps"])
            stats = h.grain_stats()
        out = {"tangents": h.area_tangents()} if case["tangents"] else {}
    finally:
        h.close()
    s = np.frombuffer(stats, STATS, case["grains"])
    # the batched form computes in FP32, so its numbers are kept in that type
    real = np.float32 if case["form"] == "batched" else np.float64
    for key in ("area", "perimeter", "energy", "mean_da"):
        out[key] = np.where(s["state"] == 1, s[key], 0.0).astype(real)
    out["state"], out["neighbours"] = s["state"].copy(), np.where(s["state"] == 1, s["n_neighbours"], 0)
    return out


def work(case):
    if case["kind"] == "box":
        n = case["n"]
        return {"bytes": 16 * n * n, "flops": 2 * 2.5 * n * n * math.log2(max(2, n * n)) + n * n}
    n, nn, steps = case["grains"], case["grid"], case["steps"]
    size = 4 if case["form"] == "batched" else 8
    # box edge of a Poisson-Voronoi grain with its border; every step reads and writes each box's field and the
    # competing-grain map, and convolves, compares and redistances each cell; four derivative fields with tangents
    edge = 1.2 * nn / math.sqrt(n) + 2 * BORDER
    cells = n * edge * edge * steps * (5 if case["tangents"] else 1)
    load = 4 * nn * nn if case["source"] != "contours" else 0
    return {"bytes": load + 88 * n * (steps if case["read"] == "each" else 1) + 2 * (size + 4) * cells,
            "flops": cells * (2 * 2.5 * math.log2(edge * edge) + 30)}


# ---- 64-bit values ---------------------------------------------------------

def exact(case, seed):
    """The box by numpy's FFT; areas and perimeters of small isotropic networks by a numpy restatement of the
    level-set step.  Anisotropic networks would need the whole corrector restated, larger ones too long."""
    if case["kind"] == "box":
        field, dt, nn = box_input(case, seed)
        return {"out": gaussian(field, dt, nn)}
    if case["physics"] != "iso" or case["source"] != "voronoi" or case["grains"] * case["steps"] > 3000:
        return None
    labels, _, boxes, _ = microstructure(case, seed)
    area, perimeter = isotropic(case, labels.cpu().numpy(), boxes)
    none = {k: None for k in ("energy", "mean_da", "state", "neighbours", "tangents")}
    return {"area": area, "perimeter": perimeter, **none}


def gaussian(field, dt, nn):
    n = len(field)
    f = np.minimum(np.arange(n), n - np.arange(n)).astype(np.float64)
    k2 = f[:, None] ** 2 + f[None, :n // 2 + 1] ** 2
    g = np.exp(-math.sqrt(2 / math.pi) * k2 * 4.0 * dt * nn ** 2 / n ** 2 * math.pi ** 2)
    return np.fft.irfft2(np.fft.rfft2(field) * g, s=(n, n))


def square(box, m):
    x0, x1, y0, y1 = (int(v) for v in box)
    w, h = x1 - x0, y1 - y0
    if w == h:
        return x0, x1, y0, y1
    if w > h:
        y0, y1 = y0 - (w - h) // 2, y1 + (w - h) // 2 + (w - h) % 2
    else:
        x0, x1 = x0 - (h - w) // 2, x1 + (h - w) // 2 + (h - w) % 2
    dx = -x0 if x0 < 0 else min(0, m - 1 - x1)
    dy = -y0 if y0 < 0 else min(0, m - 1 - y1)
    return x0 + dx, x1 + dx, y0 + dy, y1 + dy


def meet(a, b):
    return max(a[0], b[0]), min(a[1], b[1]), max(a[2], b[2]), min(a[3], b[3])


def part(field, box, of):
    """The view of `field` (stored on `box`) over the box `of` inside it."""
    return field[of[2] - box[2]:of[3] - box[2], of[0] - box[0]:of[1] - box[0]]


def sweep(out, given, r0, r1, c0, c1, h):
    """Forward and backward along axis 0; `given` holds the input in rows r0..r1, columns c0..c1."""
    o, p, k = out[:, c0:], given[:, c0:], c1 - c0
    for i in range(r0, len(o) - 1):
        into = np.sign(o[i + 1])
        if i < r1 - 1:
            a, c = p[i, :k], p[i + 1, :k]
            slope = (c - a) / h
            dz = -a / slope
            hit = (a * c <= 0) & (np.abs(o[i, :k]) > np.abs(dz))
            o[i, :k][hit] = (-dz * np.sign(slope))[hit]
            into[:k] = np.sign(c)
        cand = o[i] + into * h
        o[i + 1] = np.where(np.abs(cand) < np.abs(o[i + 1]), cand, o[i + 1])
    for i in range(r1 - 1, 0, -1):
        into = np.sign(o[i - 1])
        if i > r0:
            into[:k] = np.sign(p[i - 1, :k])
        cand = o[i] + into * h
        o[i - 1] = np.where(np.abs(cand) < np.abs(o[i - 1]), cand, o[i - 1])


def redistance(field, box, to, h, delta):
    x0, x1, y0, y1 = meet(box, to)
    out = np.full((to[3] - to[2], to[1] - to[0]), -1.0)
    given = np.zeros_like(out)
    part(given, to, (x0, x1, y0, y1))[:] = part(field, box, (x0, x1, y0, y1))
    r0, r1, c0, c1 = y0 - to[2], y1 - to[2], x0 - to[0], x1 - to[0]
    with np.errstate(divide="ignore", invalid="ignore"):
        sweep(out, given, r0, r1, c0, c1, h)
        sweep(out.T[:, r0:], given.T[:, r0:], c0, c1, 0, r1 - r0, h)
    return np.clip(out, -delta, delta)


def wall_distance(box, m, h):
    def signed(at):
        low, high = BORDER - at, at - (m - BORDER)
        return np.where(np.abs(low) < np.abs(high), low, high).astype(np.float64)
    dx, dy = np.meshgrid(signed(np.arange(box[0], box[1])), signed(np.arange(box[2], box[3])))
    return h * np.where((dx > 0) & (dy > 0), np.hypot(dx, dy), np.where((dx < 0) & (dy < 0), np.maximum(dx, dy),
                                                                       np.maximum(np.maximum(dx, dy), 0)))


def contour(field):
    """Marching squares from the first pixel inside, as points (x, y) in the box; None if there is none."""
    n_y, n_x = field.shape
    inside = np.zeros((n_y + 2, n_x + 2), dtype=int)
    inside[1:-1, 1:-1] = field >= 0
    if not inside.any():
        return None
    inside, v = inside.tolist(), field.tolist()
    r = next(k for k, row in enumerate(inside) if any(row))
    c = inside[r].index(1)
    left, top, points = c - 2, r - 2, []  # the cell whose lower right corner is the first pixel
    end, came = (left, top), None
    go = {1: "u", 2: "r", 3: "r", 4: "l", 5: "u", 7: "r", 8: "d", 10: "d", 11: "d", 12: "l", 13: "u", 14: "l"}
    while True:
        a, b = inside[top + 1], inside[top + 2]
        mask = a[left + 1] + 2 * a[left + 2] + 4 * b[left + 1] + 8 * b[left + 2]
        if mask == 6:
            move = "r" if came == "u" else "l"
        elif mask == 9:
            move = "d" if came == "r" else "u"
        else:
            move = go[mask]
            right, bottom = left + 1, top + 1
            if move == "l":
                p = (left, bottom - v[bottom][left] / (v[bottom][left] - v[top][left]) if top >= 0 else bottom)
            elif move == "r":
                p = (right, top + v[top][right] / (v[top][right] - v[bottom][right]) if bottom < n_y else top)
            elif move == "u":
                p = (left + v[top][left] / (v[top][left] - v[top][right]) if right < n_x else left, top)
            else:
                p = (right - v[bottom][right] / (v[bottom][right] - v[bottom][left]) if left >= 0 else right, bottom)
            if not points or points[-1] != p:
                points.append(p)
        left += (move == "r") - (move == "l")
        top += (move == "d") - (move == "u")
        came = move
        if (left, top) == end:
            break
    if points[0] != points[-1]:
        points.append(points[0])
    return np.array(points, dtype=np.float64)


def isotropic(case, labels, boxes):
    n, nn, b = case["grains"], case["grid"], BORDER
    m, h, delta = nn + 2 * b, 1.0 / nn, b / nn
    dt = 0.8 / nn ** 2 * int(nn / math.sqrt(n)) / 2 / 5.0
    padded = np.zeros((m + 1, m + 1), dtype=labels.dtype)
    padded[b:b + nn, b:b + nn] = labels
    box, phi = {}, {}
    for g in range(1, n + 1):
        x0, x1, y0, y1, count = boxes[g - 1]
        if count:
            box[g] = square((x0, min(x1 + 2 * b, m), y0, min(y1 + 2 * b, m)), m)
            x0, x1, y0, y1 = box[g]
            phi[g] = redistance(np.where(padded[y0:y1, x0:x1] == g, h, -h), box[g], box[g], h, delta)
    area, perimeter = np.zeros(n), np.zeros(n)
    for _ in range(case["steps"]):
        conv = {g: gaussian(f, dt, nn) for g, f in phi.items()}
        area[:], perimeter[:], new_box, new_phi = 0, 0, {}, {}
        for g, own in conv.items():
            x0, x1, y0, y1 = at = box[g]
            rival = np.full_like(own, -1.0)
            for q, field in conv.items():
                over = meet(at, box[q])
                if q != g and over[0] < over[1] and over[2] < over[3]:
                    view = part(rival, at, over)
                    np.maximum(view, part(field, box[q], over), out=view)
            if not (x0 > 2 * b and x1 < m - 2 * b and y0 > 2 * b and y1 < m - 2 * b):
                rival = np.maximum(rival, wall_distance(at, m, h))
            field = np.where(np.abs(own) < 0.7 * delta, 0.5 * (own - rival), own)
            points = contour(field)
            if points is None:
                continue
            ys, xs = np.nonzero(field >= 0)
            to = square((max(0, x0 + xs.min() - b), min(m, x0 + xs.max() + b),
                         max(0, y0 + ys.min() - b), min(m, y0 + ys.max() + b)), m)
            p = points + np.array([x0, y0])
            d = p[1:] - p[:-1]
            area[g - 1] = abs(np.sum((p[:-1, 1] + p[1:, 1]) * -d[:, 0])) * h * h * 0.5
            perimeter[g - 1] = np.sum(np.hypot(d[:, 0], d[:, 1])) * h
            new_box[g], new_phi[g] = to, redistance(field, at, to, h, delta)
        box, phi = new_box, new_phi
    return area, perimeter
