"""The launches that an iteration joins give what the separate entry points give,
bit for bit, at the edges of their tiles."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

from supernormal_gb300._lib import CopyBuffer, SupernormalError, WeightNormLayer, call, stream_handle


def _samples(n, gen):
    """Sample starts and ends, about one in nine of which leaves a gap."""
    dt = 0.01
    gap = torch.rand(n, device="cuda", generator=gen) < 0.11
    ts = torch.cumsum(torch.full((n,), dt, device="cuda") + gap * 0.05, 0)
    te = torch.cat([ts[1:], ts[-1:] + dt]) - torch.cat([gap[1:], gap[:1]]) * 0.05
    return ts, te


@pytest.mark.parametrize("n,live", [(1, None), (63, None), (64, 65), (65, 65), (256, 255), (1023, None),
                                    (1024, None), (1025, 1025), (3000, 2049), (70001, None), (500, 0)])
def test_ranked_points_equal_the_scanned_ones(n, live):
    gen = torch.Generator(device="cuda").manual_seed(n)
    P, H, W, B = 9, 3, 3, 7
    ts, te = _samples(n, gen)
    ridx = torch.sort(torch.randint(0, B, (n,), device="cuda", generator=gen))[0]
    ro, rd = torch.randn(2, B, P, 3, device="cuda", generator=gen)
    pn = torch.randn(B, 3, device="cuda", generator=gen)
    ro_c, rd_c = ro[:, 4].contiguous(), rd[:, 4].contiguous()
    count = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    m = n if live is None else min(n, live)
    st = stream_handle()
    i32 = dict(dtype=torch.int32, device="cuda")
    diff, packed, ends = torch.zeros(n, **i32), torch.zeros((n, 2), **i32), torch.zeros(1, **i32)
    call("sn_end_diff", n, count, ts, te, diff, st)
    ws = torch.empty(call("sn_scan_workspace_bytes", n), dtype=torch.uint8, device="cuda")
    call("sn_pack_counts_n", n, torch.tensor([m], **i32), diff, packed, ends, ws, st)
    rws = torch.empty(call("sn_end_ranks_workspace_bytes", n), dtype=torch.uint8, device="cuda")

    def buffers(k):
        return [torch.full((2 * n * k, 3), -7.0, device="cuda"), torch.full((1,), -1, **i32)]

    xyz, q = buffers(1)
    call("sn_center_points", n, count, ridx, ts, te, ro_c, rd_c, packed, ends, xyz, q, st)
    got, got_ends, (gxyz, gq) = torch.zeros((n, 2), **i32), torch.full((1,), -1, **i32), buffers(1)
    call("sn_end_ranks", n, count, ts, te, got, rws, st)
    call("sn_center_points_ranked", n, count, ridx, ts, te, ro_c, rd_c, rws, got, got_ends, gxyz, gq, st)
    assert torch.equal(got[:m], packed[:m]) and torch.equal(got_ends, ends)
    assert torch.equal(gxyz, xyz) and torch.equal(gq, q)

    xyz, q = buffers(P)
    tps, tpe, gtps, gtpe = torch.zeros(4, n, P, device="cuda")
    call("sn_patch_points", n, count, H, W, ridx, ts, te, ro, rd, pn, packed, ends, xyz, tps, tpe, q, st)
    gxyz, gq = buffers(P)
    call("sn_end_ranks", n, count, ts, te, got, rws, st)
    call("sn_patch_points_ranked", n, count, H, W, ridx, ts, te, ro, rd, pn, rws, got, got_ends, gxyz, gtps,
         gtpe, gq, st)
    assert torch.equal(got[:m], packed[:m]) and torch.equal(got_ends, ends)
    assert torch.equal(gxyz, xyz) and torch.equal(gq, q)
    assert torch.equal(gtps, tps) and torch.equal(gtpe, tpe)


@pytest.mark.parametrize("eps,thre", [(1e-8, 0.0), (1e-3, 0.02), (0.0, 0.0)])
def test_center_visibility_equals_alpha_then_visibility(eps, thre):
    gen = torch.Generator(device="cuda").manual_seed(3)
    steps = torch.tensor([0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 0, 300, 5], dtype=torch.int32, device="cuda")
    R, n = steps.numel(), int(steps.sum())
    packed = torch.stack([torch.cumsum(steps, 0, dtype=torch.int32) - steps, steps], 1).contiguous()
    ts, te = _samples(n, gen)
    st = stream_handle()
    i32 = dict(dtype=torch.int32, device="cuda")
    diff, endp, ends = torch.zeros(n, **i32), torch.zeros((n, 2), **i32), torch.zeros(1, **i32)
    call("sn_end_diff", n, None, ts, te, diff, st)
    call("sn_pack_counts", n, diff, endp, ends, torch.empty(call("sn_scan_workspace_bytes", n), dtype=torch.uint8,
                                                            device="cuda"), st)
    # falling through the surface half-way along a ray, some rays never
    j = torch.arange(n, device="cuda") - torch.repeat_interleave(packed[:, 0].long(), steps.long())
    sdf = (0.3 - 0.011 * j)[:, None] + 0.01 * torch.randn(n, 1, device="cuda", generator=gen)
    sdf = torch.cat([sdf, 0.05 * torch.randn(n, 1, device="cuda", generator=gen)])
    var = torch.tensor([0.45], device="cuda")
    alpha = torch.zeros(n, device="cuda")
    call("sn_center_alpha", n, None, sdf, 1, endp, var, alpha, st)
    vis, gvis = torch.full((2, n), 9, dtype=torch.uint8, device="cuda")
    counts, gcounts = torch.full((2, R), -1, **i32)
    call("sn_visibility_from_alpha", R, packed, alpha, eps, thre, vis, counts, st)
    call("sn_center_visibility", R, packed, n, None, sdf, 1, endp, var, eps, thre, gvis, gcounts, st)
    assert eps == 0.0 or 0 < int(counts.sum()) < n
    assert torch.equal(gvis, vis) and torch.equal(gcounts, counts)


@pytest.mark.parametrize("B", [1, 31, 257, 2100])
def test_step_ends_equal_the_separate_launches(B):
    gen = torch.Generator(device="cuda").manual_seed(B)
    P, st = 9, stream_handle()
    i32 = dict(dtype=torch.int32, device="cuda")
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    mask, ro, rd = torch.rand(B, P, device="cuda", generator=gen), 0.4 * rand(B, P, 3), rand(B, P, 3)
    it = torch.tensor([5], **i32)
    shapes = [(64, 35), (1, 64)]
    v, g = [rand(*s) for s in shapes], [rand(s[0]) for s in shapes]

    def layers(buf):
        return [C.byref(WeightNormLayer(*s, v[l].data_ptr(), g[l].data_ptr(), *(t.data_ptr() for t in buf[l])))
                for l, s in enumerate(shapes)]

    def outputs():
        return [[rand(*s), rand(s[0]), rand(*s), rand(*s), rand(s[0])] for s in shapes]   # w, norms, grad w, v, g

    a, b = outputs(), outputs()
    one = [torch.zeros(B, P, device="cuda"), torch.zeros(1, device="cuda"), *torch.zeros(3, B, device="cuda"),
           *torch.zeros(2, B, 3, device="cuda")]
    two = [torch.zeros_like(t) for t in one]
    call("sn_mask_prep", B * P, mask, one[0], one[1], st)
    call("sn_near_far_sphere", B, ro, rd, 3 * P, one[2], one[3], one[4], 11, it, one[5], one[6], st)
    for l, s in enumerate(shapes):
        call("sn_weightnorm_fwd", *s, v[l], g[l], a[l][0], a[l][1], st)
    call("sn_step_begin", B * P, mask, two[0], two[1], B, ro, rd, 3 * P, two[2], two[3], two[4], 11, it, two[5],
         two[6], *layers(b), st)
    for x, y in zip(one, two):
        assert torch.equal(x.nan_to_num(-9.0), y.nan_to_num(-9.0))
    for l in (0, 1):
        assert torch.equal(a[l][0], b[l][0]) and torch.equal(a[l][1], b[l][1])
        assert not b[l][2].any()
        b[l][2].copy_(a[l][2])
        call("sn_weightnorm_bwd", *shapes[l], v[l], g[l], a[l][1], a[l][2], a[l][3], a[l][4], st)
    call("sn_weightnorm_pair_bwd", *layers(b), st)
    for l in (0, 1):
        assert torch.equal(a[l][3], b[l][3]) and torch.equal(a[l][4], b[l][4])

    steps = torch.randint(0, 4, (B,), device="cuda", generator=gen, dtype=torch.int32)
    packed = torch.stack([torch.cumsum(steps, 0, dtype=torch.int32) - steps, steps], 1).contiguous()
    S = max(1, int(steps.sum()))
    endp = torch.randint(0, 2, (S, 2), device="cuda", generator=gen, dtype=torch.int32)
    carry, partials, var = rand(B, P), rand(B, 4), torch.tensor([0.3], device="cuda")
    d0 = rand(2 * S, P)
    d1, out, gout, gv, ggv = d0.clone(), *torch.zeros(2, 5, device="cuda"), *torch.ones(2, 1, device="cuda")
    call("sn_patch_carry_fixup", B, P, packed, None, S, endp, carry, d0, st)
    call("sn_patch_finalize", B, P, partials, None, S, var, one[1], 1.0, 0.5, 0.25, out, gv, st)
    call("sn_patch_finish", B, P, packed, None, S, endp, carry, d1, partials, var, one[1], 1.0, 0.5, 0.25, gout,
         ggv, st)
    assert torch.equal(d0, d1) and torch.equal(out, gout) and torch.equal(gv, ggv)
    sums = partials.double().sum(0)
    want = torch.stack([sums[1] / one[1].double()[0], sums[2] / (B * P), sums[3] / (S * P)])
    # float rounding of the three quotients
    assert torch.allclose(out[1:4].double(), want, rtol=3e-7, atol=0.0)

    src = [rand(k)[o:] for k, o in ((B, 0), (4 * B + 3, 1), (6, 2), (1, 0))]
    dst = [torch.zeros_like(s) for s in src]
    call("sn_copy_many", 4, (CopyBuffer * 4)(*(CopyBuffer(d.data_ptr(), s.data_ptr(), s.numel())
                                               for d, s in zip(dst, src))), st)
    assert all(torch.equal(d, s) for d, s in zip(dst, src))


def _net(d_out, weight_norm=True):
    from supernormal_gb300.fields import SDFNetwork

    torch.manual_seed(3)
    net = SDFNetwork(3, d_out, 64, 1, weight_norm=weight_norm, input_concat=True, encoding_config=dict(
        otype="HashGrid", n_levels=4, n_features_per_level=2, log2_hashmap_size=11, base_resolution=8,
        per_level_scale=1.5)).cuda()
    net.bindwidth = 3
    with torch.no_grad():
        for p in net.parameters():
            p.add_(0.1 * torch.randn_like(p))
    return net


@pytest.mark.parametrize("n", [0, 1, 300])
@pytest.mark.parametrize("d_out,second_order", [(1, False), (5, False), (1, True)])
def test_weight_normalised_field_equals_its_layers(n, d_out, second_order):
    """One node for layers and field: the values of the layer-by-layer route bit
    for bit, its gradients up to the order of the sums (norm-wise 1e-5: at most
    300 points, 128 to a sum taken in order, at float's 6e-8), for every form of
    the parameters that the layers take and with parameters frozen."""
    from supernormal_gb300.fields import _FieldFn, _FieldGradFn

    net = _net(d_out)
    x = (2 * torch.rand(n, 3, device="cuda") - 1).requires_grad_(not second_order)

    def layered():
        w0, b0, w1, b1 = net.mlp_tensors()
        args = (net.encoding.params, w0.contiguous(), b0.contiguous(), w1.contiguous(), b1.contiguous(), net)
        return _FieldGradFn.apply(x, *args) if second_order else (_FieldFn.apply(x, *args, d_out),)

    def fused():
        return net.sdf_and_gradient(x) if second_order else (net.forward(x),)

    lin0 = net.lin0
    forms = {
        "all": lambda: None,
        "rows strided": lambda: setattr(lin0, "weight_v", torch.nn.Parameter(
            torch.cat([lin0.weight_v.data] * 2, 1)[:, : lin0.in_features])),
        "double": lambda: setattr(lin0, "weight_g", torch.nn.Parameter(lin0.weight_g.data.double())),
        "frozen first layer": lambda: [p.requires_grad_(False) for p in lin0.parameters()],
        "frozen weights": lambda: [p.requires_grad_(False) for l in (lin0, net.lin1)
                                   for k, p in l.named_parameters() if k != "bias"],
    }
    for name, change in forms.items():
        change()
        if n == 0:   # an empty tensor has no address: refused either way
            for route in (layered, fused):
                with pytest.raises(SupernormalError, match="null buffer"):
                    route()
            continue
        a, b = layered(), fused()
        ga = [torch.randn_like(t) for t in a]
        leaves = [p for p in net.parameters() if p.requires_grad] + ([] if second_order else [x])
        da = torch.autograd.grad(a, leaves, ga, allow_unused=True)
        db = torch.autograd.grad(b, leaves, ga, allow_unused=True)
        for u, v in zip(a, b):
            assert torch.equal(u, v), name
        for u, v in zip(da, db):
            assert u.shape == v.shape and u.dtype == v.dtype, name
            assert float((u - v).norm()) <= 1e-5 * float(u.norm()) + 1e-30, name
    if n:
        assert torch.equal(net.sdf_raw(x.detach()), net.sdf(x.detach()))


def test_plain_layers_keep_their_route():
    net = _net(1, weight_norm=False)
    assert net._weight_norm_params() is None and _net(1)._weight_norm_params() is not None
    y = net.sdf(torch.rand(50, 3, device="cuda"))
    g = torch.autograd.grad(y.sum(), [net.lin0.weight, net.lin1.weight])
    assert all(bool(t.abs().sum() > 0) for t in g)


@pytest.mark.parametrize("n", [1, 127, 129, 5000])
def test_kept_and_regathered_encodings_agree(n, monkeypatch):
    """The backward that reads kept encodings and the one that gathers them again:
    the same dL/dx bit for bit (summed per point), the other gradients up to the
    order of their atomic sums (norm-wise 2e-5: float's 6e-8 over sums of up to
    5,000 terms, 128 to a block, whose rounding errors add like their square root)."""
    from supernormal_gb300 import fields

    net = _net(1)
    x = (2 * torch.rand(n, 3, device="cuda") - 1).requires_grad_()
    gy = torch.randn(n, 1, device="cuda")
    leaves = [x, *net.parameters()]
    kept = torch.autograd.grad(net.sdf(x), leaves, gy)
    monkeypatch.setattr(fields, "_KEPT_ENCODING_BYTES", 0)
    again = torch.autograd.grad(net.sdf(x), leaves, gy)
    assert torch.equal(kept[0], again[0])
    for u, v in zip(kept, again):
        assert float((u - v).norm()) <= 2e-5 * float(u.norm())


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1028, 400_003])
@pytest.mark.parametrize("eps", [1e-8, 0.0])
def test_adam_untouched_entries_equal_the_general_path(n, eps):
    """Entries that an update leaves as they are: the bits of the path that writes
    everything (taken where a half-precision copy is kept)."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    p, g, m = torch.randn(3, n, device="cuda", generator=gen)
    v = torch.rand(n, device="cuda", generator=gen)
    untouched = (torch.rand((n + 7) // 8, device="cuda", generator=gen) < 0.6).repeat_interleave(8)[:n]
    for t in (g, m, v):
        t[untouched] = 0.0
    g[::5] = 0.0
    g[3::64] = -0.0
    st = stream_handle()
    out = []
    for half in (None, torch.zeros(n, dtype=torch.float16, device="cuda")):
        a = [torch.empty(n + 4, device="cuda")[:n].copy_(t) for t in (p, g, m, v)]
        call("sn_adam_step", n, *a, half, None, None, 1e-3, 7, 0.9, 0.999, eps, 1, st)
        out.append(a)
    for x, y in zip(*out):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))


@pytest.mark.parametrize("R", [1, 7, 8, 9, 129, 4096, 4097, 9000])
def test_compaction_from_counts_equals_the_packed_one(R):
    gen = torch.Generator(device="cuda").manual_seed(R)
    i32 = dict(dtype=torch.int32, device="cuda")
    steps = torch.randint(0, 150, (R,), generator=gen, **i32) * (torch.rand(R, device="cuda", generator=gen) < 0.4)
    steps[-1] = 3
    steps = steps.to(torch.int32)
    n = int(steps.sum())
    packed = torch.stack([torch.cumsum(steps, 0, dtype=torch.int32) - steps, steps], 1).contiguous()
    vis = (torch.rand(n, device="cuda", generator=gen) < 0.5).to(torch.uint8)
    rows = torch.repeat_interleave(torch.arange(R, device="cuda"), steps.long())
    counts = torch.zeros(R, device="cuda").index_add_(0, rows, vis.float()).to(torch.int32)
    ts, te = torch.rand(2, n, device="cuda", generator=gen)
    st, ws = stream_handle(), torch.empty(call("sn_scan_workspace_bytes", R), dtype=torch.uint8, device="cuda")
    outs = []
    for joined in (False, True):
        po, total = torch.full((R, 2), -1, **i32), torch.full((1,), -1, **i32)
        o = [torch.full((n,), -1, dtype=torch.int64, device="cuda"), *torch.full((2, n), -1.0, device="cuda")]
        if joined:
            call("sn_compact_counts", R, packed, vis, counts, po, total, ws, rows, ts, te, *o, st)
        else:
            call("sn_pack_counts", R, counts, po, total, ws, st)
            call("sn_compact_samples", R, packed, vis, po, rows, ts, te, *o, st)
        outs.append([po, total, *o])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("R", [1, 3, 4, 5, 1000, 4096, 4097])
def test_expansion_from_counts_equals_the_packed_one(R):
    gen = torch.Generator(device="cuda").manual_seed(R)
    i32 = dict(dtype=torch.int32, device="cuda")
    o = 0.3 * torch.randn(R, 3, device="cuda", generator=gen)
    d = torch.nn.functional.normalize(torch.randn(R, 3, device="cuda", generator=gen), dim=-1)
    t0, t1 = torch.zeros(R, device="cuda"), torch.ones(R, device="cuda")
    roi = torch.tensor([-1.0, -1, -1, 1, 1, 1], device="cuda")
    grid = (torch.rand(32, 32, 32, device="cuda", generator=gen) < 0.3).to(torch.uint8)
    st, ws = stream_handle(), torch.empty(call("sn_scan_workspace_bytes", R), dtype=torch.uint8, device="cuda")
    march = (R, o, d, t0, t1, None, roi, grid, 32, 32, 32, 0, 0.01, None, 0.0, 0)
    counts, status = torch.empty(R, **i32), torch.zeros(1, **i32)
    runs = torch.empty(call("sn_march_runs_bytes", R), dtype=torch.uint8, device="cuda")
    call("sn_march_runs", *march, 0, counts, runs, status, st)
    n = int(counts.sum())
    outs = []
    for joined in (False, True):
        po, total = torch.full((R, 2), -1, **i32), torch.full((1,), -1, **i32)
        s = [torch.full((n,), -1, dtype=torch.int64, device="cuda"), *torch.full((2, n), -1.0, device="cuda")]
        if joined:
            call("sn_march_expand_counts", *march, counts, po, total, ws, runs, n, *s, status, st)
        else:
            call("sn_pack_counts", R, counts, po, total, ws, st)
            call("sn_march_expand", *march, po, runs, n, *s, status, st)
        outs.append([po, total, *s])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("cols,offset", [(1, 0), (1, 1), (3, 0), (3, 2), (4, 0), (16, 0)])
@pytest.mark.parametrize("n", [1, 5, 127, 4099, 70_001])
def test_output_bias_gradient_of_cancelling_terms(n, cols, offset):
    """The output biases' gradients are column sums whose terms nearly cancel: no
    further off 64 bits than the rounding of the result and 2^-39 of the terms'
    sizes (the sums in float carry their errors; at most 9 terms a thread and 17
    levels of merging, so what the errors themselves lose is below (26 x 2^-24)^2 / 2
    of them).  Rows past the device's count are not read."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    net = _net(cols)
    g = 1e3 * torch.randn(n, cols, device="cuda", generator=gen)
    if n > 1:
        g[-1] = 0.0
        g[-1] = (1e-3 - g.double().sum(0)).float()
    buf = torch.full((n * cols + 2 * cols + 8,), float("nan"), device="cuda")
    buf[offset:offset + n * cols] = g.reshape(-1)
    go, want, size = buf[offset:], g.double().sum(0), g.double().abs().sum(0)
    x = 2 * torch.rand(n + 2, 3, device="cuda", generator=gen) - 1
    w0, b0, w1, b1 = (t.detach().contiguous() for t in net.mlp_tensors())
    mlp, grid, table = C.byref(net._mlp_desc(w0, b0, w1, b1)), C.byref(net.encoding.desc), net.encoding.params
    st = stream_handle()
    for cap, count in ((n, None), (n + 2, torch.tensor([n], dtype=torch.int32, device="cuda"))):
        gb1 = torch.zeros(cols, device="cuda")
        call("sn_field_bwd", cap, count, x, go, cols, table, grid, 3, mlp, None, None, None, None, gb1, None, st)
        assert bool(((gb1.double() - want).abs() <= 2.0**-24 * want.abs() + 2.0**-39 * size).all())
        if cols == 1:
            gb1, gx = torch.zeros(1, device="cuda"), torch.zeros(n + 2, 3, device="cuda")
            call("sn_field_grad_bwd", cap, count, x, gx, go, table, grid, 3, mlp, None, None, None, None, gb1, st)
            assert bool(((gb1.double() - want).abs() <= 2.0**-24 * want.abs() + 2.0**-39 * size).all())
    go[0] = float("inf")
    gb1 = torch.zeros(cols, device="cuda")
    call("sn_field_bwd", n, None, x, go, cols, table, grid, 3, mlp, None, None, None, None, gb1, None, st)
    assert float(gb1[0]) == float("inf")


@pytest.mark.parametrize("second_order", [False, True])
def test_output_weight_gradient_does_not_depend_on_the_order_of_blocks(second_order):
    """The parts of the output layer's weight gradient cancel; summed in a fixed
    order in a block and in double over the blocks they leave weight_g's and
    weight_v's gradients the same at every call, up to a last bit of the result and
    2^-40 of the terms' sizes (double, any order: 152 x 2^-53)."""
    net, n = _net(1), 60_001
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = 2 * torch.rand(n, 3, device="cuda", generator=gen) - 1
    gy = 1e3 * torch.randn(n, 1, device="cuda", generator=gen)
    gy -= gy.mean()
    leaves, got = [net.lin1.weight_g, net.lin1.weight_v], []
    for _ in range(12):
        y = net.sdf_and_gradient(x)[0] if second_order else net.sdf(x)
        got.append([t.double() for t in torch.autograd.grad(y, leaves, gy)])
    with torch.no_grad():   # terms of dW1: |g| times an activation of at most the largest pre-activation + log(2) / beta
        w0, b0, w1, _ = net.mlp_tensors()
        size = float(gy.double().abs().sum()) * float((w0.abs().sum(1) + b0.abs()).max() + 0.01)
    for t in zip(*got):
        t = torch.stack(t)
        spread = t.max(0).values - t.min(0).values
        assert bool((spread <= 2.0**-23 * t.abs().max(0).values + 2.0**-40 * size).all())


@pytest.mark.parametrize("variance", [0.3, -0.7, 1.5, -1.5])
@pytest.mark.parametrize("B", [1, 31, 255, 257, 2049, 20_000])
def test_loss_sums_against_double(B, variance):
    """Every number that the finishing launch writes, formed here in double.  The sums
    are in double there too; behind them come expf (2 ulp), two products and a sum in
    float: 2^-21 of the numbers' sizes.  Past the clip of exp(10 variance) (1.5 and
    -1.5) the variance has no gradient."""
    gen = torch.Generator(device="cuda").manual_seed(B)
    P, S, st, i32 = 9, 3 * B, stream_handle(), dict(dtype=torch.int32, device="cuda")
    partials = torch.randn(B, 4, device="cuda", generator=gen)
    var, mask = torch.tensor([variance], device="cuda"), torch.tensor([0.37 * B], device="cuda")
    packed = torch.stack([3 * torch.arange(B, **i32), torch.full((B,), 3, **i32)], 1).contiguous()
    endp, carry, d_sdf = torch.ones((S, 2), **i32), torch.zeros(B, P, device="cuda"), torch.zeros(2 * S, P, device="cuda")
    sums, size = partials.double().sum(0), partials.double().abs().sum(0)
    scale = torch.stack([10 * torch.exp(10 * var.double()[0]) * (abs(variance) < 1.3), 1 / mask.double()[0],
                         torch.tensor(1 / (B * P), device="cuda"), torch.tensor(1 / (S * P), device="cuda")])
    terms, weights = sums * scale, torch.tensor([0.0, 1.0, 0.25, 0.5], device="cuda", dtype=torch.float64)
    want = torch.cat([terms, (weights * terms).sum()[None]])
    room = 2.0**-21 * torch.cat([terms.abs(), (weights * terms).abs().sum()[None]])
    for name, head in (("sn_patch_finalize", (B, P, partials, None, S)),
                       ("sn_patch_finish", (B, P, packed, None, S, endp, carry, d_sdf, partials))):
        out, gv = torch.full((5,), 7.0, device="cuda"), torch.ones(1, device="cuda")
        call(name, *head, var, mask, 1.0, 0.5, 0.25, out, gv, st)
        assert bool(((out.double() - want).abs() <= room).all()), name
        assert abs(float(gv) - (1 + float(want[0]))) <= float(room[0]) + 2.0**-24 * abs(1 + float(want[0])), name


@pytest.mark.parametrize("R", [3, 300, 4097])
@pytest.mark.parametrize("short,counted", [(1, False), (70, True), (200, False)])
def test_compaction_stops_at_the_capacity(R, short, counted):
    """A packed table that goes past the capacity: samples up to there alone, though
    the bytes behind (here in reach) read as visible, and nothing past the output."""
    gen = torch.Generator(device="cuda").manual_seed(R + short)
    i32 = dict(dtype=torch.int32, device="cuda")
    steps = torch.randint(100, 150, (R,), generator=gen, **i32)
    n = int(steps.sum())
    live = n - short
    packed = torch.stack([torch.cumsum(steps, 0, dtype=torch.int32) - steps, steps], 1).contiguous()
    vis = (torch.rand(n + 256, device="cuda", generator=gen) < 0.5).to(torch.uint8)
    vis[live - 1:] = 1   # the last sample below the capacity, and every byte behind
    rows = torch.arange(R, device="cuda").repeat_interleave(steps.long())
    rows = torch.cat([rows, torch.full((256,), -5, device="cuda")])
    ts, te = torch.rand(2, n + 256, device="cuda", generator=gen)
    seen = (vis[:live] > 0).nonzero()[:, 0]
    counts = torch.bincount(rows[seen], minlength=R).to(torch.int32)
    want_packed = torch.stack([torch.cumsum(counts, 0, dtype=torch.int32) - counts, counts], 1)
    cap, count = (n + 256, torch.tensor([live], **i32)) if counted else (live, None)
    out = [torch.full((seen.numel() + 256,), -1, dtype=torch.int64, device="cuda"),
           *torch.full((2, seen.numel() + 256), -1.0, device="cuda")]
    po, total = torch.full((R, 2), -1, **i32), torch.full((1,), -1, **i32)
    ws = torch.empty(call("sn_scan_workspace_bytes", R), dtype=torch.uint8, device="cuda")
    call("sn_compact_counts_n", R, packed, cap, count, vis, counts, po, total, ws, rows, ts, te, *out, stream_handle())
    assert torch.equal(po, want_packed) and int(total) == seen.numel()
    for got, src in zip(out, (rows, ts, te)):
        assert torch.equal(got[:seen.numel()], src[seen]) and bool((got[seen.numel():] == -1).all())


def test_softplus_derivative_keeps_subnormals():
    """beta x = -92: z = exp(-92) = 1.1e-40 is subnormal, and so is softplus' there;
    output weights of 1e20 bring it back to sizes that show.  1e-4: half of z's last
    place is 7e-6 of it, and the exponent's rounding (133 x 2^-24) as much again."""
    net = _net(1)
    with torch.no_grad():
        net.lin0.weight_v.zero_()[:, 0] = 1.0
        net.lin0.weight_g.fill_(1.0)
        net.lin0.bias.fill_(-0.92)
        net.lin1.weight_v.fill_(1.0)
        net.lin1.weight_g.fill_(8e20)
    z = torch.exp(net.lin0.bias.detach().double() * 100)
    x = torch.zeros(5, 3, device="cuda")
    for y in (net.sdf(x), net.sdf_and_gradient(x)[0]):
        (b0,) = torch.autograd.grad(y.sum(), [net.lin0.bias])
        assert torch.allclose(b0.double(), 5e20 * z, rtol=1e-4, atol=0.0)
    n = net.gradient(x)[:, 0].detach()
    assert torch.allclose(n[:, 0].double(), (1e20 * z.sum()).expand(5), rtol=1e-4, atol=0.0)
    x.requires_grad_()
    (gx,) = torch.autograd.grad(net.sdf(x).sum(), [x])
    assert torch.allclose(gx[:, 0].double(), (1e20 * z.sum()).expand(5), rtol=1e-4, atol=0.0)


@pytest.mark.parametrize("n,live", [(4096 * 1024, None), (4096 * 1024 + 1, None), (4096 * 1024 + 1, 700_001),
                                    (9_000_001, 8_999_937)])
def test_ranked_points_of_many_samples(n, live):
    """At the capacity from which the tiles' totals are scanned, and past it: the slots,
    the centre points and the points of 1 x 1 patches that the scanned flags give."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    B, st, i32 = 7, stream_handle(), dict(dtype=torch.int32, device="cuda")
    ts, te = _samples(n, gen)
    ridx = torch.sort(torch.randint(0, B, (n,), device="cuda", generator=gen))[0]
    ro, rd = torch.randn(2, B, 3, device="cuda", generator=gen)
    pn = torch.randn(B, 3, device="cuda", generator=gen)
    count = None if live is None else torch.tensor([live], **i32)
    m = n if live is None else live
    diff, packed, ends = torch.zeros(n, **i32), torch.zeros((n, 2), **i32), torch.zeros(1, **i32)
    call("sn_end_diff", n, count, ts, te, diff, st)
    ws = torch.empty(call("sn_scan_workspace_bytes", n), dtype=torch.uint8, device="cuda")
    call("sn_pack_counts_n", n, torch.tensor([m], **i32), diff, packed, ends, ws, st)
    rws = torch.empty(call("sn_end_ranks_workspace_bytes", n), dtype=torch.uint8, device="cuda")
    got, got_ends = torch.zeros((n, 2), **i32), torch.full((1,), -1, **i32)
    xyz, gxyz = torch.full((2, 2 * n, 3), -7.0, device="cuda")
    q, gq = torch.full((2, 1), -1, **i32)
    call("sn_center_points", n, count, ridx, ts, te, ro, rd, packed, ends, xyz, q, st)
    call("sn_end_ranks", n, count, ts, te, got, rws, st)
    call("sn_center_points_ranked", n, count, ridx, ts, te, ro, rd, rws, got, got_ends, gxyz, gq, st)
    assert torch.equal(got[:m], packed[:m]) and torch.equal(got_ends, ends)
    assert torch.equal(gxyz, xyz) and torch.equal(gq, q) and int(ends) > m // 10
    tps, tpe, gtps, gtpe = torch.zeros(4, n, 1, device="cuda")
    xyz.fill_(-7.0), gxyz.fill_(-7.0)
    call("sn_patch_points", n, count, 1, 1, ridx, ts, te, ro, rd, pn, packed, ends, xyz, tps, tpe, q, st)
    call("sn_end_ranks", n, count, ts, te, got, rws, st)
    call("sn_patch_points_ranked", n, count, 1, 1, ridx, ts, te, ro, rd, pn, rws, got, got_ends, gxyz, gtps, gtpe,
         gq, st)
    assert torch.equal(got[:m], packed[:m]) and torch.equal(got_ends, ends)
    assert torch.equal(gxyz, xyz) and torch.equal(gq, q)
    assert torch.equal(gtps, tps) and torch.equal(gtpe, tpe)


def test_replaced_weights_are_asked_for(monkeypatch):
    """A subclass' or an instance's own mlp_tensors, and a layer's own
    effective_weight, count in every evaluation of the field."""
    from supernormal_gb300.fields import SDFNetwork, WeightNormLinear

    class Doubled(SDFNetwork):
        def mlp_tensors(self):
            w0, b0, w1, b1 = super().mlp_tensors()
            return w0, b0, 2.0 * w1, 2.0 * b1

    def values(net):
        x = torch.linspace(-0.9, 0.9, 60, device="cuda").reshape(20, 3)
        return [t.detach() for t in (net.sdf(x), net.forward(x), net.sdf_raw(x), *net.sdf_and_gradient(x))]

    def doubled(net):
        own = net.lin1.effective_weight
        return lambda: 2.0 * own()

    want = [2.0 * t for t in values(_net(3))]
    net = _net(3)
    net.__class__ = Doubled
    instance = _net(3)
    instance.mlp_tensors = lambda: [k * t for k, t in zip((1, 1, 2.0, 2.0), SDFNetwork.mlp_tensors(instance))]
    layer = _net(3)
    layer.lin1.effective_weight = doubled(layer)
    with torch.no_grad():
        layer.lin1.bias.mul_(2.0)
    for got in (values(net), values(instance), values(layer)):
        for a, b in zip(got, want):   # a power of two: every rounding is the same
            assert torch.equal(a, b)
    patched, own = _net(3), WeightNormLinear.effective_weight
    with torch.no_grad():
        patched.lin1.bias.mul_(2.0)
    monkeypatch.setattr(WeightNormLinear, "effective_weight",
                        lambda lin: own(lin) * (2.0 if lin is patched.lin1 else 1.0))
    for a, b in zip(values(patched), want):
        assert torch.equal(a, b)


def test_kept_encodings_are_bounded_together(monkeypatch):
    """Evaluations that wait for their backwards share one network's bound; a
    backward, or a graph dropped without one, gives its share back, and the network's
    switch keeps nothing.  The gradients do not depend on it."""
    import copy
    import pickle

    from supernormal_gb300 import fields

    net, n = _net(1), 4096
    x = 2 * torch.rand(n, 3, device="cuda") - 1
    one = 8 * 3 * n
    monkeypatch.setattr(fields, "_KEPT_ENCODING_BYTES", 2 * one + one // 2)
    leaves = list(net.parameters())
    grads = lambda y: torch.autograd.grad(y.sum(), leaves, retain_graph=True)

    def kept():
        before = torch.cuda.memory_allocated()
        y = net.sdf(x)
        return y, torch.cuda.memory_allocated() - before >= one

    ys = [kept() for _ in range(4)]
    assert [k for _, k in ys] == [True, True, False, False]
    want = grads(ys[2][0])
    for u, v in zip(grads(ys[0][0]), want):
        assert float((u - v).norm()) <= 2e-5 * float(v.norm())
    grads(ys[0][0])                                 # a second backward gives nothing back twice
    assert net._encoding_budget().held == one and kept()[1]
    del ys
    assert net._encoding_budget().held == 0
    with torch.no_grad():
        assert not kept()[1]
    assert copy.deepcopy(net)._encoding_budget().held == 0 and pickle.loads(pickle.dumps(net)) is not None
    net.encoding_cache = False
    y, k = kept()
    assert not k and net._encoding_budget().held == 0
    for u, v in zip(grads(y), want):
        assert float((u - v).norm()) <= 2e-5 * float(v.norm())


@pytest.mark.parametrize("steps", [[1280, 1281, 0, 40, 1312], [2600, 33, 5000], [1281] * 3])
def test_patch_adjoint_of_rays_longer_than_the_kept_carries(steps):
    """Rays of more than 1,280 samples, whose transmittances the adjoint's second walk
    forms again from every second, third, ... kept one, against the operator in double.
    2e-4 of the norm: an alpha is a difference of sigmoids that are a few 2^-24 off, over
    up to 5,000 samples, 70 x 4 x 2^-24, times three for what the adjoint makes of it; a
    transmittance taken from another chunk would be off by hundredths."""
    gen = torch.Generator(device="cuda").manual_seed(len(steps))
    H, W, P, B, S, st = 3, 3, 9, len(steps), sum(steps), stream_handle()
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    counts = torch.tensor(steps, device="cuda")
    first = counts.cumsum(0) - counts
    packed = torch.stack([first, counts], 1).to(torch.int32).contiguous()
    ray = torch.repeat_interleave(torch.arange(B, device="cuda"), counts)
    j = (torch.arange(S, device="cuda") - first[ray]).float()
    start = 0.25 - 0.5 * (j / counts[ray])
    start = start[:, None] + 1e-5 * rand(S, P)
    own = torch.rand(S, device="cuda", generator=gen) < 0.1
    own[(first + counts - 1)[counts > 0]] = True            # a ray's last end is its own
    slot = own.cumsum(0) - own.long()
    endp = torch.stack([slot, own.long()], 1).to(torch.int32).contiguous()
    step = (0.5 / counts[ray])[:, None]
    ends = (start - step * (1 + 0.1 * rand(S, P).abs()))[own]
    sdf = torch.cat([start, ends]).contiguous()
    var, ext = torch.tensor([0.3], device="cuda"), rand(S, P, 3)
    tps = torch.arange(S, device="cuda").float()[:, None].expand(S, P).contiguous()
    ro, rd, vinv, gc, gw = rand(B, P, 3), rand(B, P, 3), rand(B, P, 3, 3), rand(B, P, 3), rand(B, P)
    d_sdf, d_ext = torch.full_like(sdf, 7.0), torch.empty_like(ext)
    partials, carry = torch.zeros(B, 4, device="cuda"), torch.empty(B, P, device="cuda")
    call("sn_patch_render_bwd", B, H, W, packed, None, S, endp, sdf, tps, tps + 1, ro, rd, vinv, var, gc, gw, None,
         d_sdf, partials, carry, ext, d_ext, st)

    x = sdf.double().requires_grad_()
    inv_s = torch.exp(10 * var.double())
    nxt = torch.where(own[:, None], x[S + slot.clamp(max=int(own.sum()) - 1)], x[torch.arange(1, S + 1, device="cuda").clamp(max=S - 1)])
    c0, c1 = torch.sigmoid(x[:S] * inv_s), torch.sigmoid(nxt * inv_s)
    alpha = ((c0 - c1 + 1e-5) / (c0 + 1e-5)).clip(0.0, 1.0)
    loss = 0.0
    for b in range(B):
        a = alpha[first[b]:first[b] + counts[b]]
        w = a * torch.cat([torch.ones_like(a[:1]), (1 - a).cumprod(0)[:-1]])
        loss = loss + ((w[..., None] * ext[first[b]:first[b] + counts[b]].double()).sum(0) * gc[b].double()).sum()
        loss = loss + (w.sum(0) * gw[b].double()).sum()
    (want,) = torch.autograd.grad(loss, x)
    assert float((d_sdf.double() - want).norm()) <= 2e-4 * float(want.norm())
