"""Performance cases: what programs have this framework do, through its public entry points.

A case is a dict of plain values.  ``kind`` names the call:

* ``train``    one training iteration (``trainer.GraphStep.step``: march, cull, field, render,
               losses, adjoint, Adam, an occupancy update every 8 iterations);
* ``sdf``      ``SDFNetwork.sdf`` at given points and its gradients w.r.t. the parameters;
* ``gradient`` ``SDFNetwork.sdf_and_gradient`` and its (second-order) gradients;
* ``lattice``  ``mesh.sdf_lattice``: the SDF on a res^3 lattice, the input of mesh extraction;
* ``mesh``     ``mesh.marching_cubes`` of such a lattice;
* ``march``    ``nerfacc.ray_marching`` of camera rays through an occupancy grid;
* ``weights``  nerfacc's patch weights and accumulation, forward and backward;
* ``patches``  ``NeuSRenderer.render_samples`` of culled samples, forward and backward;
* ``view``     ``NeuSRenderer.render`` in eval mode over the patches of an image.

The field of every case is the shipped network (16 levels x 2 features, 35 -> 64 -> 16) in a
state like a trained one: a surface near the sphere of radius 0.5, hash-table entries that fall
with the level's resolution, and an occupancy grid that is full inside the surface.
"""
from __future__ import annotations

import math

import torch

from supernormal_gb300 import mesh, nerfacc, scenes
from supernormal_gb300.fields import SDFNetwork, SingleVarianceNetwork
from supernormal_gb300.renderer import NeuSRenderer, near_far_from_sphere
from supernormal_gb300.trainer import FusedTrainer, GraphStep, TrainConfig

DEV = "cuda"
LEVELS, BASE, SCALE, HIDDEN = 16, 16, 1.447, 64
VARIANCE = 0.5            # inv_s = exp(5): ~25 kept samples per centre ray at a step of 2/1024
RADIUS = 0.5
VIEW_H, VIEW_W, VIEW_FOV = 512, 612, 40.0


def listed():
    return [
        # a small reconstruction (table 2^15, coarse steps): launches and latency count
        dict(name="train_small", kind="train", patches=256, table=15, inv_step=64, method="dfd",
             precision="fp32", patch=3),
        # the reference's training configuration: 2048 3x3 patches, table 2^19, <= 1024 samples a chord
        dict(name="train_full", kind="train", patches=2048, table=19, inv_step=512, method="dfd",
             precision="fp32", patch=3),
        # a served object's iteration: 512 patches, the largest table, mixed precision
        dict(name="train_served_mixed", kind="train", patches=512, table=21, inv_step=512, method="dfd",
             precision="mixed", patch=3),
        # a few scattered SDF queries with gradients (a caller's own regulariser)
        dict(name="sdf_small", kind="sdf", points=2053, table=15, layout="scattered"),
        # the field evaluation of a training step: samples of neighbouring rays
        dict(name="sdf_rays", kind="sdf", points=500003, table=19, layout="rays"),
        # normals by differentiation ('ad'), differentiated again for the normal loss
        dict(name="gradient_rays", kind="gradient", points=100003, table=19, layout="rays"),
        # the lattice of a validation mesh
        dict(name="lattice_256", kind="lattice", res=256, table=19),
        # the mesh of that lattice
        dict(name="mesh_256", kind="mesh", res=256),
        # the centre rays of a whole 612x512 image
        dict(name="march_image", kind="march", rays=VIEW_H * VIEW_W, inv_step=512),
        # the operators of a renderer that keeps its own alpha: 2048 patches, ~27 samples each
        dict(name="weights_2048", kind="weights", patches=2048, samples=27, patch=3),
        # the renderer as a module in the caller's own training loop, at the first marching step 1e-2
        dict(name="patches_2048", kind="patches", patches=2048, inv_step=100, table=19, patch=3),
        # a normal map at a new pose
        dict(name="view_300", kind="view", res=300, inv_step=512, table=19),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "sdf", "gradient", "lattice", "mesh", "march", "weights", "patches", "view"])
    c = dict(kind=kind)
    if kind == "train":
        c["patch"] = rng.choice([3, 3, 3, 5])
        c["patches"] = _log(rng, 64, 2047 if c["patch"] == 3 else 512)
        c["table"] = rng.randint(15, 21 if c["patches"] <= 512 else 19)
        c["inv_step"] = _log(rng, 64, 512)
        c["method"] = rng.choice(["dfd", "dfd", "ad"])
        c["precision"] = rng.choice(["fp32", "mixed"]) if c["method"] == "dfd" else "fp32"
    elif kind == "sdf":
        c.update(points=_log(rng, 1, 500000), table=rng.randint(15, 20), layout=rng.choice(["rays", "scattered"]))
    elif kind == "gradient":
        c.update(points=_log(rng, 1, 100000), table=rng.randint(15, 20), layout=rng.choice(["rays", "scattered"]))
    elif kind == "lattice":
        c.update(res=_log(rng, 32, 255), table=rng.randint(15, 20))
    elif kind == "mesh":
        c.update(res=_log(rng, 32, 255))
    elif kind == "march":
        c.update(rays=_log(rng, 100, VIEW_H * VIEW_W - 1), inv_step=_log(rng, 64, 511))
    elif kind == "weights":
        p = rng.choice([3, 3, 5])
        c.update(patches=_log(rng, 64, 2047 if p == 3 else 700), samples=_log(rng, 4, 27), patch=p)
    elif kind == "patches":
        p = rng.choice([3, 3, 5])
        c.update(patches=_log(rng, 64, 2047 if p == 3 else 700), inv_step=_log(rng, 50, 100),
                 table=rng.randint(15, 19), patch=p)
    else:
        c.update(res=3 * _log(rng, 10, 99), inv_step=_log(rng, 64, 511), table=rng.randint(15, 19))
    return c


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _encoding(table):
    return dict(otype="HashGrid", n_levels=LEVELS, n_features_per_level=2, log2_hashmap_size=table,
                base_resolution=BASE, per_level_scale=SCALE)


def _field(table, seed):
    """The shipped network, its surface near the sphere of radius 0.5 and every level in use."""
    torch.manual_seed(seed)
    net = SDFNetwork(3, 16, HIDDEN, 1, skip_in=(-1,), bias=RADIUS, encoding_config=_encoding(table),
                     input_concat=True).to(DEV)
    g = _generator(seed)
    offsets, res, _ = _levels(table)
    with torch.no_grad():
        t = net.encoding.params.view(-1, 2)
        for l in range(LEVELS):
            n = offsets[l + 1] - offsets[l]
            t[offsets[l]:offsets[l + 1]] = (torch.rand((n, 2), device=DEV, generator=g) - 0.5) * (1.0 / res[l])
        v = net.lin0.weight_v
        v[:, 3:] = 0.05 * torch.randn((HIDDEN, 2 * LEVELS), device=DEV, generator=g)
        net.lin0.weight_g.copy_(v.norm(dim=1, keepdim=True))
    net.bindwidth = LEVELS
    return net


def _plain_sdf(net, x):
    """The network without its encoding: near enough to place an occupancy grid."""
    with torch.no_grad():
        w0 = net.lin0.weight_v[:, :3]
        h = torch.nn.functional.softplus(x @ w0.T + net.lin0.bias, beta=100)
        w1 = (net.lin1.weight_g * net.lin1.weight_v / net.lin1.weight_v.norm(dim=1, keepdim=True))[0]
        return h @ w1 + net.lin1.bias[0]


def _fill_grid(grid, net):
    r = int(grid.resolution[0])
    u = (torch.arange(r, device=DEV) + 0.5) / r * 2.0 - 1.0
    for i in range(r):
        x = torch.stack(torch.meshgrid(u[i:i + 1], u, u, indexing="ij"), -1).reshape(-1, 3)
        grid.occs.view(r, -1)[i] = torch.sigmoid(-80.0 * _plain_sdf(net, x))
    grid._binary.copy_((grid.occs > min(float(grid.occs.mean()), 0.1)).view(r, r, r))


def _rig(views):
    return scenes.ring_cameras(views, VIEW_H, VIEW_W, radius=3.0, elevation_deg=30.0, fov_deg=VIEW_FOV)


def _batch(patches, patch, seed):
    ds = scenes.SyntheticDataset(scenes.sphere(RADIUS), _rig(4), torch.device(DEV))
    return ds.gen_random_patches(patches, patch, patch, generator=_generator(seed + 1))


def _points(n, layout, seed):
    """Field points: uniform in the cube, or 32 consecutive samples of each ray near the surface."""
    g = _generator(seed + 2)
    if layout == "scattered":
        return torch.rand((n, 3), device=DEV, generator=g) * 2.0 - 1.0
    rays = (n + 31) // 32
    patch = (rays + 8) // 9                       # nine neighbouring rays a patch
    d = torch.nn.functional.normalize(torch.randn((patch, 3), device=DEV, generator=g), dim=-1)
    side = torch.nn.functional.normalize(torch.randn((patch, 3), device=DEV, generator=g), dim=-1)
    off = torch.stack(torch.meshgrid(torch.arange(3.0), torch.arange(3.0), indexing="ij"), -1).reshape(9, 2).to(DEV)
    up = torch.linalg.cross(d, side)
    o = (RADIUS + 0.03) * d
    o = o[:, None] + 0.003 * (off[:, :1] * side[:, None] + off[:, 1:] * up[:, None])     # (patch, 9, 3)
    t = torch.arange(32.0, device=DEV) * (2.0 / 1024)
    x = o[:, None] - t[None, :, None, None] * d[:, None, None]                            # (patch, 32, 9, 3)
    return x.reshape(-1, 3)[:n].contiguous()


def _weights_of(net):
    return [net.encoding.params, net.lin0.weight_g, net.lin0.weight_v, net.lin0.bias,
            net.lin1.weight_g, net.lin1.weight_v, net.lin1.bias]


def _prepare_train(c, seed):
    net = _field(c["table"], seed)
    var = SingleVarianceNetwork(VARIANCE).to(DEV)
    # iterations past the schedules: the rate constant and so small that repeated passes keep the same work
    cfg = TrainConfig(batch_size=c["patches"], patch_h=c["patch"], patch_w=c["patch"],
                      step_size=1.0 / c["inv_step"], learning_rate=5e-6, learning_rate_alpha=1.0,
                      gradient_method=c["method"], precision=c["precision"], seed=seed & 0xFFFF)
    tr = FusedTrainer(net, var, cfg, device=DEV)
    _fill_grid(tr.grid, net)
    g = _generator(seed + 3)
    tr.exp_avg.copy_(torch.randn(tr.n_params, device=DEV, generator=g) * 1e-5)
    tr.exp_avg_sq.copy_((torch.rand(tr.n_params, device=DEV, generator=g) + 0.5) * 1e-8)
    tr.iter_step = 5001
    tr.iter_dev.fill_(tr.iter_step)
    graph = GraphStep(tr)
    batch = _batch(c["patches"], c["patch"], seed)
    graph.prepare()
    return dict(kind="train", tr=tr, graph=graph, batch=batch)


def _prepare_patches(c, seed):
    """Samples as marching and culling leave them: consecutive steps of the patches that see the surface."""
    p = c["patch"]
    net = _field(c["table"], seed)
    ro, rd, pn, vinv, _, _ = _batch(c["patches"], p, seed)
    oc, dc = ro[:, p // 2, p // 2], rd[:, p // 2, p // 2]
    b = (oc * dc).sum(-1)
    reach = b * b - (oc * oc).sum(-1) + (RADIUS + 0.03) ** 2
    dt = 1.0 / c["inv_step"]
    g = _generator(seed + 4)
    # the fifth of the patches that come closest to the centre; always the same number of samples in all
    hits = reach.argsort(descending=True)[: max(1, c["patches"] // 5)]
    steps = torch.zeros(c["patches"], dtype=torch.int64, device=DEV)
    steps[hits] = c["inv_step"] // 12 + torch.arange(hits.numel(), device=DEV) % (c["inv_step"] // 12)
    first = -b - reach.clamp_min(0).sqrt() + dt * torch.rand(c["patches"], device=DEV, generator=g)
    idx = torch.repeat_interleave(torch.arange(c["patches"], device=DEV), steps)
    k = torch.arange(idx.numel(), device=DEV) - (steps.cumsum(0) - steps)[idx]
    t = first[idx] + k * dt
    ts, te = t[:, None].contiguous(), (first[idx] + (k + 1) * dt)[:, None].contiguous()
    var = SingleVarianceNetwork(0.35).to(DEV)
    n, s = c["patches"], idx.numel()
    grads = [torch.randn((n, p, p, 3), device=DEV, generator=g) / n, torch.randn((n, p, p, 1), device=DEV, generator=g) / n,
             torch.randn((s, p, p, 3), device=DEV, generator=g) / max(1, s * p * p)]
    return dict(kind="patches", renderer=NeuSRenderer(net, var), args=(ro, rd, pn, vinv, idx, ts, te), grads=grads,
                leaves=_weights_of(net) + [var.variance])


def _prepare_view(c, seed):
    net = _field(c["table"], seed)
    r = NeuSRenderer(net, SingleVarianceNetwork(VARIANCE).to(DEV))
    _fill_grid(r.occupancy_grid, net)
    r.sampling_step_size = 1.0 / c["inv_step"]
    rig = scenes.ring_cameras(8, c["res"], c["res"], radius=3.0, elevation_deg=10.0 + seed % 30, fov_deg=VIEW_FOV)
    v = seed % 8
    d, vinv = scenes.view_rays(rig, v, torch.device(DEV))
    n = c["res"] // 3
    blocks = lambda t: t.reshape(n, 3, n, 3, *t.shape[2:]).transpose(1, 2).reshape(n * n, 3, 3, *t.shape[2:]).contiguous()
    rd, vinv = blocks(d), blocks(vinv)
    pose = rig.poses[v].to(DEV).float()
    ro = pose[:3, 3].expand(rd.shape).contiguous()
    near, far = near_far_from_sphere(ro[:, 1, 1], rd[:, 1, 1])
    return dict(kind="view", renderer=r, rays=(ro, rd, pose[:3, 2].expand(n * n, 3).contiguous(), near, far, vinv),
                jitter=_generator(seed + 5))


def _prepare_march(c, seed):
    """The rays of one view, or that many of its pixels, beginning at a pixel that the seed gives."""
    grid = nerfacc.OccupancyGrid([-1.0, -1.0, -1.0, 1.0, 1.0, 1.0], 128).to(DEV)
    _fill_grid(grid, _field(15, 0))
    d, _ = scenes.view_rays(_rig(8), 1, torch.device(DEV))
    rd = d.reshape(-1, 3)
    if c["rays"] < rd.shape[0]:
        rd = rd[torch.randperm(rd.shape[0], device=DEV, generator=_generator(6))[: c["rays"]]]
    rd = rd.roll(int(torch.randint(1, c["rays"], (1,), device=DEV, generator=_generator(seed + 6))), 0).contiguous()
    ro = _rig(8).poses[1, :3, 3].to(DEV).float().expand(rd.shape).contiguous()
    near, far = near_far_from_sphere(ro, rd)
    return dict(kind="march", grid=grid, rays=(ro, rd, near, far), step=1.0 / c["inv_step"])


def _prepare_weights(c, seed):
    g = _generator(seed + 8)
    n, p = c["patches"], c["patch"] ** 2
    counts = (torch.arange(n, device=DEV) % (2 * c["samples"] + 1))[torch.randperm(n, device=DEV, generator=g)]
    idx = torch.repeat_interleave(torch.arange(n, device=DEV), counts)
    s = idx.numel()
    alphas = torch.rand((s, p, 1), device=DEV, generator=g).square() * 0.6
    values = torch.randn((s, p, 3), device=DEV, generator=g)
    grads = [torch.randn((n, p, 3), device=DEV, generator=g), torch.randn((n, p, 1), device=DEV, generator=g)]
    return dict(kind="weights", idx=idx, alphas=alphas.requires_grad_(), values=values.requires_grad_(), n=n, grads=grads)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "train":
        return _prepare_train(c, seed)
    if kind == "patches":
        return _prepare_patches(c, seed)
    if kind == "view":
        return _prepare_view(c, seed)
    if kind == "march":
        return _prepare_march(c, seed)
    if kind == "weights":
        return _prepare_weights(c, seed)
    if kind == "mesh":
        r = c["res"]
        u = torch.linspace(-1.0, 1.0, r, device=DEV)
        x, y, z = torch.meshgrid(u, u, u, indexing="ij")
        g = _generator(seed + 9)
        bumps = 0.02 * torch.sin(12.0 * x) * torch.sin(9.0 * y) * torch.sin(15.0 * z)
        u = RADIUS - (x * x + y * y + z * z).sqrt() + bumps
        # a distance that is off by up to a tenth: other vertices on the same edges
        return dict(kind="mesh", u=u * (1.0 + 0.1 * torch.rand(u.shape, device=DEV, generator=g)))
    net = _field(c["table"], seed)
    if kind == "lattice":
        return dict(kind="lattice", net=net, res=c["res"])
    g = _generator(seed + 10)
    n = c["points"]
    s = dict(kind=kind, net=net, x=_points(n, c["layout"], seed), leaves=_weights_of(net),
             gs=torch.randn((n, 1), device=DEV, generator=g) / n)
    if kind == "gradient":
        s["gg"] = torch.randn((n, 3), device=DEV, generator=g) / n
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    s, kind = state, state["kind"]
    if kind == "train":
        loss = s["graph"].step(s["batch"])
        tr = s["tr"]
        return dict(loss=loss, params=tr.params, exp_avg=tr.exp_avg, exp_avg_sq=tr.exp_avg_sq)
    if kind == "sdf":
        y = s["net"].sdf(s["x"])
        return [y, *torch.autograd.grad(y, s["leaves"], s["gs"])]
    if kind == "gradient":
        y, n = s["net"].sdf_and_gradient(s["x"])
        return [y, n, *torch.autograd.grad([y, n], s["leaves"], [s["gs"], s["gg"]])]
    if kind == "lattice":
        return mesh.sdf_lattice(s["net"], (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), s["res"])
    if kind == "mesh":
        return mesh.marching_cubes(s["u"], 0.0, (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0))
    if kind == "march":
        ro, rd, near, far = s["rays"]
        return nerfacc.ray_marching(ro, rd, t_min=near, t_max=far, grid=s["grid"], render_step_size=s["step"])
    if kind == "weights":
        w = nerfacc.render_weight_from_alpha_patch_based(s["alphas"], s["idx"], n_rays=s["n"])
        normal = nerfacc.accumulate_along_rays_patch_based(w, s["idx"], values=s["values"], n_patches=s["n"])
        mask = nerfacc.accumulate_along_rays_patch_based(w, s["idx"], n_patches=s["n"])
        return [w, normal, mask, *torch.autograd.grad([normal, mask], [s["alphas"], s["values"]], s["grads"])]
    if kind == "patches":
        out = s["renderer"].render_samples(*s["args"])
        got = [out["comp_normal"], out["weight_sum"], out["gradients"]]
        return got + list(torch.autograd.grad(got, s["leaves"], s["grads"]))
    ro, rd, pn, near, far, vinv = s["rays"]
    normals, masks = [], []
    with torch.no_grad():
        for a in range(0, ro.shape[0], 4096):
            b = min(a + 4096, ro.shape[0])
            out = s["renderer"].render(ro[a:b], rd[a:b], pn[a:b], near[a:b], far[a:b], vinv[a:b], mode="eval",
                                       generator=s["jitter"])
            normals.append(out["comp_normal"])
            masks.append(out["weight_sum"])
    return [torch.cat(normals), torch.cat(masks)]


def _entries(table):
    return _levels(table)[0][-1]


def work(case):
    c, kind = case, case["kind"]
    point = 2.0 * (35 * HIDDEN + HIDDEN)                    # one evaluation of the MLP's sdf
    if kind == "train":
        p = c["patch"] ** 2
        kept = 0.22 * max(2.0, 0.22 * c["inv_step"])        # samples of a centre ray that pass the culling
        n = c["patches"] * kept
        params = 2 * _entries(c["table"])
        batch = c["patches"] * p * (3 + 3 + 9 + 3 + 1) * 4
        return dict(bytes=params * 24.0 + batch, flops=n * point + n * p * point * (6 if c["method"] == "ad" else 3))
    if kind in ("sdf", "gradient"):
        k = 1 if kind == "sdf" else 4
        return dict(bytes=16.0 * _entries(c["table"]) + c["points"] * (12.0 + 8.0 * k),
                    flops=c["points"] * point * (3 if kind == "sdf" else 6))
    if kind == "lattice":
        return dict(bytes=8.0 * _entries(c["table"]) + 4.0 * c["res"] ** 3, flops=c["res"] ** 3 * point)
    if kind == "mesh":
        return dict(bytes=4.0 * c["res"] ** 3 + 2.4 * c["res"] ** 2 * (12 + 24), flops=0.0)
    if kind == "march":
        return dict(bytes=c["rays"] * 32.0 + 128 ** 3 + c["rays"] * 0.217 * c["inv_step"] * 16.0, flops=0.0)
    if kind == "weights":
        p = c["patch"] ** 2
        n = c["patches"] * c["samples"] * p
        return dict(bytes=n * 4.0 * (1 + 1 + 3 + 1 + 3) + c["patches"] * p * 32.0, flops=n * 30.0)
    if kind == "patches":
        p = c["patch"] ** 2
        n = c["patches"] / 5 * c["inv_step"] / 8 * p
        return dict(bytes=16.0 * _entries(c["table"]) + n * 24.0, flops=n * point * 3)
    n = (c["res"] // 3) ** 2 * 0.22 * max(2.0, 0.22 * c["inv_step"])
    return dict(bytes=8.0 * _entries(c["table"]) + c["res"] ** 2 * 76.0, flops=n * 10 * point)


# ---------------------------------------------------------------------------
# the same in 64 bits, with plain torch
# ---------------------------------------------------------------------------
def _levels(table):
    """Offsets, resolutions and float32 scales of the levels (Instant-NGP's geometry)."""
    pls = float(torch.tensor(math.log2(float(torch.tensor(SCALE, dtype=torch.float32))), dtype=torch.float32))
    offsets, res, scales = [0], [], []
    for l in range(LEVELS):
        s = float(torch.tensor(2.0 ** (l * pls) * BASE - 1.0, dtype=torch.float32))
        r = int(math.ceil(s)) + 1
        offsets.append(offsets[-1] + min((r ** 3 + 7) // 8 * 8, 1 << table))
        res.append(r)
        scales.append(s)
    return offsets, res, scales


def _encode64(x, entries, table, x64):
    """The encoding of float32 points (cells and fractions are float32 by definition), in 64 bits."""
    offsets, res, scales = _levels(table)
    out = []
    for l in range(LEVELS):
        pos = (x.double() * scales[l] + 0.5).float()
        cell = pos.floor()
        xs = x64 * scales[l]
        f = (pos - cell).double() + (xs - xs.detach())
        q = cell.long() & 0xFFFFFFFF
        size, r = offsets[l + 1] - offsets[l], res[l]
        acc = 0.0
        for k in range(8):
            i = [(q[:, d] + ((k >> d) & 1)) & 0xFFFFFFFF for d in range(3)]
            if r ** 3 <= size:
                idx = (i[0] + i[1] * r + i[2] * (r * r)) & 0xFFFFFFFF
            else:
                idx = i[0] ^ ((i[1] * 2654435761) & 0xFFFFFFFF) ^ ((i[2] * 805459861) & 0xFFFFFFFF)
            e = entries.index_select(0, offsets[l] + idx % size)
            w = 1.0
            for d in range(3):
                w = w * (f[:, d] if (k >> d) & 1 else 1.0 - f[:, d])
            acc = acc + w[:, None] * e
        out.append(acc)
    return torch.cat(out, 1)


def _sdf64(x, leaves, table, x64=None):
    t, g0, v0, b0, g1, v1, b1 = leaves
    x64 = x.double() if x64 is None else x64
    h = torch.cat([x64, _encode64(x, t.view(-1, 2), table, x64)], 1)
    h = h @ (g0 * v0 / v0.norm(dim=1, keepdim=True)).T + b0
    h = torch.where(h * 100.0 > 20.0, h, torch.log1p(torch.exp((h * 100.0).clamp(max=20.0))) / 100.0)
    return h @ (g1 * v1 / v1.norm(dim=1, keepdim=True))[:1].T + b1[:1]


def _leaves64(leaves):
    return [p.detach().double().requires_grad_() for p in leaves]


def _grads64(outs, leaves, grads):
    got = torch.autograd.grad(outs, leaves, [g.double() for g in grads], allow_unused=True)
    return [torch.zeros_like(p) if g is None else g for p, g in zip(leaves, got)]


def _exact_patches(s, c):
    ro, rd, pn, vinv, idx, ts, te = s["args"]
    n, p = ro.shape[0], c["patch"]
    leaves = _leaves64(s["leaves"])
    # sample positions are float32 numbers, as the field's inputs are
    dot = lambda a, b: (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]
    dc = dot(rd[:, p // 2, p // 2], pn)[idx][:, None, None]
    dp = dot(rd, pn[:, None, None].expand_as(rd))[idx]
    t0, t1 = (ts[:, :, None] * dc / dp), (te[:, :, None] * dc / dp)
    x0 = ro[idx] + rd[idx] * t0[..., None]
    x1 = ro[idx] + rd[idx] * t1[..., None]
    last = torch.cat([ts[1:], ts[-1:]])[:, 0] != te[:, 0]
    f = _sdf64(torch.cat([x0, x1[last]]).reshape(-1, 3), leaves[:7], c["table"]).reshape(-1, p, p)
    s0 = f[: idx.numel()]
    s1 = torch.cat([s0[1:], s0[-1:]])
    s1 = s1.index_copy(0, last.nonzero()[:, 0], f[idx.numel():])
    inv_s = torch.exp(leaves[7] * 10.0).clip(1e-6, 1e6)
    a, b = torch.sigmoid(s0 * inv_s), torch.sigmoid(s1 * inv_s)
    alpha = ((a - b + 1e-5) / (a + 1e-5)).clip(0.0, 1.0)
    w = alpha * _transmittance64(alpha.reshape(-1, p * p), idx, n).reshape(alpha.shape)
    x = x0.double()
    dx, dy = (x[:, :, 1:] - x[:, :, :-1]).norm(dim=-1), (x[:, 1:] - x[:, :-1]).norm(dim=-1)
    gx = torch.cat([(s0[:, :, 1:2] - s0[:, :, :1]) / dx[:, :, :1],
                    (s0[:, :, 2:] - s0[:, :, :-2]) / (dx[:, :, :-1] + dx[:, :, 1:]),
                    (s0[:, :, -1:] - s0[:, :, -2:-1]) / dx[:, :, -1:]], 2)
    gy = torch.cat([(s0[:, 1:2] - s0[:, :1]) / dy[:, :1], (s0[:, 2:] - s0[:, :-2]) / (dy[:, :-1] + dy[:, 1:]),
                    (s0[:, -1:] - s0[:, -2:-1]) / dy[:, -1:]], 1)
    g = torch.stack([(s1 - s0) / (t1.double() - t0.double()), gx, gy], -1)
    g = (vinv.double()[idx] @ g[..., None])[..., 0]
    comp = torch.zeros((n, p, p, 3), dtype=torch.float64, device=DEV).index_add(0, idx, w[..., None] * g)
    mask = torch.zeros((n, p, p), dtype=torch.float64, device=DEV).index_add(0, idx, w)[..., None]
    return [comp, mask, g, *_grads64([comp, mask, g], leaves, s["grads"])]


def _transmittance64(alpha, idx, n):
    """prod of 1 - alpha over the earlier samples of the same patch, per pixel."""
    counts = torch.bincount(idx, minlength=n)
    k = torch.arange(idx.numel(), device=DEV) - (counts.cumsum(0) - counts)[idx]
    width = int(counts.max()) + 1
    rest = torch.ones((n * width, alpha.shape[1]), dtype=torch.float64, device=DEV)
    rest = rest.index_copy(0, idx * width + k + 1, 1.0 - alpha) if width > 1 else rest
    return rest.reshape(n, width, -1).cumprod(1).reshape(n * width, -1)[idx * width + k]


def exact(case, seed):
    """None for training iterations, views and marching: which samples they keep is decided by comparisons
    of float32 values, one after another along a ray."""
    c, kind = case, case["kind"]
    if kind in ("train", "view", "march"):
        return None
    s = prepare(case, seed)
    if kind == "mesh":
        u, r = s["u"].double(), c["res"]
        inside, verts = u > 0.0, []
        for axis in range(3):
            m = r - 1
            cut = (inside.narrow(axis, 0, m) != inside.narrow(axis, 1, m)).nonzero()
            lo, hi = (u.narrow(axis, k, m)[cut[:, 0], cut[:, 1], cut[:, 2]] for k in (0, 1))
            pos = cut.double()
            pos[:, axis] += -lo / (hi - lo)
            verts.append(pos * (2.0 / (r - 1)) - 1.0)
        return [torch.cat(verts), None]
    if kind == "weights":
        a, v = s["alphas"].detach().double().requires_grad_(), s["values"].detach().double().requires_grad_()
        w = a * _transmittance64(a[..., 0], s["idx"], s["n"])[..., None]
        zero = torch.zeros((s["n"], a.shape[1], 3), dtype=torch.float64, device=DEV)
        normal, mask = zero.index_add(0, s["idx"], w * v), zero[..., :1].index_add(0, s["idx"], w)
        return [w, normal, mask, *_grads64([normal, mask], [a, v], s["grads"])]
    if kind == "patches":
        return _exact_patches(s, c)
    if kind == "lattice":
        leaves, r = [p.detach().double() for p in _weights_of(s["net"])], c["res"]
        u = torch.linspace(-1.0, 1.0, r, device=DEV, dtype=torch.float64).float()
        out = torch.empty((r, r, r), dtype=torch.float64, device=DEV)
        with torch.no_grad():
            for i in range(0, r, 8):
                x = torch.stack(torch.meshgrid(u[i:i + 8], u, u, indexing="ij"), -1).reshape(-1, 3)
                out[i:i + 8] = -_sdf64(x, leaves, c["table"]).reshape(-1, r, r)
        return out
    leaves = _leaves64(s["leaves"])
    if kind == "sdf":
        y = _sdf64(s["x"], leaves, c["table"])
        return [y, *_grads64([y], leaves, [s["gs"]])]
    x = s["x"].double().requires_grad_()
    y = _sdf64(s["x"], leaves, c["table"], x)
    (n,) = torch.autograd.grad(y.sum(), x, create_graph=True)
    return [y, n, *_grads64([y, n], leaves, [s["gs"], s["gg"]])]
