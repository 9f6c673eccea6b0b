"""Performance cases of the soft-shadow library: what its users have it do, over the sizes they do it at.

A case is one call of a program that holds its scene on the GPU: a shadow frame (the context API), a batch of
frames (one launch for all of them), a rasterised view with its shadows and shading, the G-buffer alone, or the
shading pass alone.  Scenes follow the distributions of 4dzb_b200/scenes.py (a height-field receiver, a soup of
small occluder triangles, a rectangular light above), drawn on the GPU from the case's seed.
"""
import importlib
import math

import numpy as np
import torch

DEVICE = "cuda"


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # the smallest calls, where launches and latency count: a preview or probe view
        _frame("frame_tiny", 128, 96, 400, 8, 16),
        # a small interactive view (the repository's "small" workload)
        _frame("frame_small", 256, 256, 1024, 8, 32, sigma=0.15),
        # an odd window size with an animated, back-face culled model and an odd light grid
        _frame("frame_odd", 641, 359, 7001, 5, 32, sigma=0.15, cull=True, xform=True),
        # the headline frame (the "hd" workload): dense occluders, most samples end in umbra
        _frame("frame_hd", 1920, 1080, 200_000, 16, 128),
        # the same view under few occluders: most samples stay in penumbra
        _frame("frame_penumbra", 1920, 1080, 20_000, 16, 128),
        # a wide, rectangular light grid (64-bit row words)
        _frame("frame_rect_light", 1920, 1080, 200_000, 64, 128, nh=48),
        # occluders beside and behind the light too, with the depth plane on
        _frame("frame_depth_plane", 1280, 720, 50_000, 16, 64, zhi=7.0, depth=True),
        # the largest frame (the "large" workload): more triangle/bin pairs than one pass holds
        _frame("frame_large", 3840, 2160, 2_000_000, 32, 256, sigma=0.05, zlo=0.2, zhi=4.0, radius=2.0),
        # offline rendering: independent frames of mixed sizes in one launch
        {"name": "batch_mixed", "kind": "batch", "frames": 16, "samples": 400_000, "T": 70_000},
        # a whole view of an application: G-buffer, shadows, shading
        {"name": "view_hd", "kind": "view", "W": 1920, "H": 1080, "grid": 256, "T": 200_000, "n": 8, "bins": 128},
        # the G-buffer alone, at an odd window size
        {"name": "raster_odd", "kind": "raster", "W": 1367, "H": 769, "grid": 48, "T": 30_000},
        # the shading pass alone, with the one light sample that the application shades with
        {"name": "shade_hd", "kind": "shade", "W": 1920, "H": 1080, "lights": 1},
    ]


def _frame(name, W, H, T, n, bins, nh=0, sigma=0.1, zlo=0.5, zhi=3.0, radius=1.0, cull=False, xform=False,
           depth=False):
    c = {"kind": "frame", "W": W, "H": H, "T": T, "n": n, "nh": nh or n, "bins": bins, "sigma": sigma, "zlo": zlo,
         "zhi": zhi, "radius": radius, "cull": cull, "xform": xform, "depth": depth}
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Shadow frames mostly (their sizes, densities, lights and options drawn together), the other calls now and then."""
    p = rng.random()
    if p < 0.08:
        return {"kind": "batch", "frames": rng.randint(2, 24), "samples": _log(rng, 65_536, 600_000),
                "T": _log(rng, 10_000, 100_000)}
    W, H = _log(rng, 97, 2560), _log(rng, 61, 1440)
    if p < 0.18:
        return {"kind": "view", "W": W, "H": H, "grid": rng.randint(16, 256), "T": _log(rng, 500, 200_000),
                "n": rng.choice([4, 8, 16]), "bins": _bins(W * H)}
    if p < 0.25:
        return {"kind": "raster", "W": W, "H": H, "grid": rng.randint(16, 256), "T": _log(rng, 500, 200_000)}
    if p < 0.30:
        return {"kind": "shade", "W": W, "H": H, "lights": rng.choice([1, 1, 16, 64])}
    n = rng.choice([4, 5, 8, 8, 12, 16, 16, 16, 24, 32])
    nh = rng.choice([0, 0, 0, 0, max(1, n - 3), 40])
    return _frame("", W, H, _log(rng, 300, 300_000), n, _bins(W * H), nh=nh, sigma=rng.choice([0.05, 0.1, 0.15]),
                  zhi=rng.choice([3.0, 3.0, 4.0]), radius=rng.choice([0.25, 0.5, 1.0, 1.0, 2.0]),
                  cull=rng.random() < 0.3, xform=rng.random() < 0.3, depth=rng.random() < 0.15)


def _bins(samples):
    """About 128 samples a bin, the library's own starting point."""
    b = 8
    while b < 256 and b * 2 <= math.sqrt(samples / 128.0) * 1.41421356:
        b *= 2
    return b


# ---- scenes, on the GPU ------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEVICE, dtype=torch.float64)


def _receiver(g, W, H):
    """Positions and normals, float4 row-major: z = 0.3 sin x cos y over [-8, 8]^2, jittered; 0.5 % background."""
    i = torch.arange(W, device=DEVICE, dtype=torch.float64).repeat(H)
    j = torch.arange(H, device=DEVICE, dtype=torch.float64).repeat_interleave(W)
    x = -8.0 + (i + _uniform(g, W * H)) * (16.0 / W)
    y = -8.0 + (j + _uniform(g, W * H)) * (16.0 / H)
    nrm = torch.stack([-0.3 * x.cos() * y.cos(), 0.3 * x.sin() * y.sin(), torch.ones_like(x)], 1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    pos = torch.stack([x, y, 0.3 * x.sin() * y.cos()], 1) + 1e-4 * nrm
    pos4 = torch.ones(W * H, 4, device=DEVICE)
    nrm4 = torch.zeros(W * H, 4, device=DEVICE)
    pos4[:, :3] = pos.float()
    nrm4[:, :3] = nrm.float()
    pos4[_uniform(g, W * H) < 0.005] = float("nan")
    return pos4, nrm4


def _occluders(g, T, sigma, zlo, zhi):
    c = _uniform(g, T, 1, 3) * torch.tensor([12.0, 12.0, zhi - zlo], device=DEVICE, dtype=torch.float64)
    c = c + torch.tensor([-6.0, -6.0, zlo], device=DEVICE, dtype=torch.float64)
    d = torch.randn(T, 3, 3, generator=g, device=DEVICE, dtype=torch.float64) * sigma
    v = torch.ones(3 * T, 4, device=DEVICE)
    v[:, :3] = (c + d).reshape(-1, 3).float()
    return v, torch.arange(3 * T, device=DEVICE, dtype=torch.int32).reshape(T, 3)


def _rotation(degrees):
    a = math.radians(degrees)
    m = np.eye(4, dtype=np.float32)
    m[:2, :2] = [[math.cos(a), -math.sin(a)], [math.sin(a), math.cos(a)]]
    return m


def _light(scenes, radius, n, nh):
    return scenes.Light(right_radius=radius, top_radius=radius, n=n, nh=nh)


def _frame_inputs(case, seed):
    g = _gen(seed)
    pos, nrm = _receiver(g, case["W"], case["H"])
    vtx, idx = _occluders(g, case["T"], case["sigma"], case["zlo"], case["zhi"])
    return pos, nrm, vtx, idx


def _mesh_inputs(case, seed):
    """scenes.mesh_scene on the GPU: a receiver grid and an occluder soup in the MeshManager layout, and a camera."""
    scenes = importlib.import_module("4dzb_b200.scenes")
    grid, T = case["grid"], case["T"]
    base = scenes.mesh_scene(case["W"], case["H"], grid=grid, T=1, n=case.get("n", 8))
    nv = (grid + 1) ** 2
    ov, _ = _occluders(_gen(seed), T, 0.1, 0.5, 3.0)
    tri = ov[:, :3].double().reshape(-1, 3, 3)
    fn = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    fn = fn / fn.norm(dim=1, keepdim=True).clamp_min(1e-30)
    soup = torch.zeros(3 * T, 8, device=DEVICE)
    soup[:, :3] = ov[:, :3]
    soup[:, 5:] = fn.repeat_interleave(3, 0).float()
    vtx = torch.cat([torch.from_numpy(base.vtx[:nv]).to(DEVICE), soup])
    ridx = torch.from_numpy(base.idx[:base.n_receiver].astype(np.int32)).to(DEVICE)
    idx = torch.cat([ridx, torch.arange(3 * T, device=DEVICE, dtype=torch.int32).reshape(T, 3) + nv])
    mat = torch.cat([torch.zeros(len(ridx), device=DEVICE, dtype=torch.int32),
                     torch.ones(T, device=DEVICE, dtype=torch.int32)])
    return base, vtx, idx, mat, torch.from_numpy(base.materials).to(DEVICE), ov


def _batch_case(case, seed):
    """Sizes of the batch's frames: log-uniform around the case's, grids of 8 or 16, light sides of 0.5 to 4."""
    rng = np.random.RandomState(20)   # the sizes belong to the case, the contents to the seed
    out = []
    for k in range(case["frames"]):
        S = case["samples"] * 4.0 ** rng.uniform(-1, 1)
        W = int(round(math.sqrt(S * rng.uniform(1.0, 16.0 / 9.0))))
        H = max(1, int(round(S / W)))
        T = int(round(case["T"] * 4.0 ** rng.uniform(-1, 1)))
        n = int(rng.choice([8, 16]))
        out.append(_frame("", W, H, T, n, _bins(W * H), radius=float(rng.uniform(0.25, 2.0))))
    return out


# ---- the calls ---------------------------------------------------------------

def _context(fdzb, scenes, case, pos, nrm, vtx, idx, masks=True):
    S = case["W"] * case["H"]
    shadow = torch.zeros(S, device=DEVICE)
    mk = torch.zeros(S, fdzb.mask_words(case["n"], case["nh"]), device=DEVICE, dtype=torch.int32) if masks else None
    ctx = fdzb.Context()
    ctx.set_view(case["W"], case["H"])
    ctx.set_bin_num(case["bins"])
    ctx.set_scenes_esp(1e-3)
    ctx.set_backface_cull(case["cull"])
    ctx.add_model(vtx, len(vtx), 16, idx, len(idx), "scene")
    ctx.set_sample_buffers(pos, nrm)
    ctx.set_output_buffer(shadow, mk)
    ctx.set_area_light(_light(scenes, case["radius"], case["n"], case["nh"]))
    if case["depth"]:
        ctx.set_depth_plane(True)
    if case["xform"]:
        ctx.set_model_transform(_rotation(3.0).reshape(-1, order="F"))
    return ctx, shadow, mk


def prepare(case, seed):
    fdzb = importlib.import_module("4dzb_b200")
    scenes = importlib.import_module("4dzb_b200.scenes")
    kind = case["kind"]
    st = {"kind": kind, "fdzb": fdzb, "case": case}
    if kind == "frame":
        inputs = _frame_inputs(case, seed)
        st["ctx"], st["shadow"], st["masks"] = _context(fdzb, scenes, case, *inputs)
    elif kind == "batch":
        frames, st["out"], st["keep"] = [], [], []
        for k, c in enumerate(_batch_case(case, seed)):
            pos, nrm, vtx, idx = _frame_inputs(c, 1000 * int(seed) + k)
            shadow = torch.zeros(len(pos), device=DEVICE)
            masks = torch.zeros(len(pos), fdzb.mask_words(c["n"]), device=DEVICE, dtype=torch.int32)
            frames.append(fdzb.frame_desc(pos, nrm, c["W"], c["H"], vtx, len(vtx), idx, len(idx),
                                          _light(scenes, c["radius"], c["n"], c["n"]), shadow, masks, bins=c["bins"]))
            st["out"].append((shadow, masks))
            st["keep"] += [pos, nrm, vtx, idx]
        st["batch"], st["frames"] = fdzb.Batch(), frames
    elif kind in ("view", "raster"):
        base, vtx, idx, mat, mats, ov = _mesh_inputs(case, seed)
        S = case["W"] * case["H"]
        st["g"] = [torch.zeros(S, 4, device=DEVICE) for _ in range(4)]
        st["depth"] = torch.zeros(S, device=DEVICE)
        st["keep"] = [vtx, idx, mat, mats, ov]
        st["desc"] = fdzb.raster_desc(vtx, len(vtx), idx, len(idx), mats, len(mats), base.model, base.view_proj,
                                      case["W"], case["H"], *st["g"], st["depth"], tri_material=mat)
        st["raster"] = fdzb.Raster()
        if kind == "view":
            st["stream"] = torch.cuda.Stream()
            st["raster"].set_stream(st["stream"].cuda_stream)
            oi = torch.arange(len(ov), device=DEVICE, dtype=torch.int32).reshape(-1, 3)
            st["keep"].append(oi)
            full = dict(case, nh=case["n"], radius=1.0, cull=False, depth=False, xform=False)
            st["ctx"], st["shadow"], _ = _context(fdzb, scenes, full, st["g"][0], st["g"][1], ov, oi, masks=False)
            st["ctx"].set_stream(st["stream"].cuda_stream)
            st["rgba"] = torch.zeros(S, 4, device=DEVICE)
            st["eye"] = base.eye
            st["lights"] = torch.tensor([list(base.light.position)], device=DEVICE)
    else:
        st["shade"] = _shade_inputs(case, seed)
        st["rgba"] = torch.zeros(case["W"] * case["H"], 4, device=DEVICE)
    return st


SHADE_EYE, SHADE_LA, SHADE_LD, SHADE_LS = (0.0, -13.0, 11.0), (0.2, 0.2, 0.2), (0.8, 0.8, 0.8), (0.5, 0.5, 0.5)


def _shade_inputs(case, seed):
    """A G-buffer of the receiver with two materials, its shadows, and light samples over a 2 x 2 light."""
    g = _gen(seed)
    pos, nrm = _receiver(g, case["W"], case["H"])
    S = len(pos)
    mats = torch.tensor([[0.1, 0.1, 0.1, 0.6, 0.6, 0.55, 0.2, 0.2, 0.2, 16.0],
                         [0.1, 0.05, 0.05, 0.7, 0.2, 0.2, 0.5, 0.5, 0.5, 32.0]], device=DEVICE)
    m = mats[(_uniform(g, S) < 0.3).long()]
    shadow = (_uniform(g, S) * 1.5 - 0.25).clamp(0, 1).float()
    pos[:, 3], nrm[:, 3] = m[:, 6], m[:, 7]
    g2 = torch.cat([m[:, 0:3], m[:, 8:9]], 1).contiguous()
    g3 = torch.cat([m[:, 3:6], m[:, 9:10]], 1).contiguous()
    gone = pos[:, 0].isnan()
    shadow[gone] = float("nan")
    lights = torch.cat([_uniform(g, case["lights"], 2) * 2 - 1, torch.full((case["lights"], 1), 6.0, device=DEVICE)], 1)
    return pos, nrm, g2, g3, shadow, lights.float().contiguous()


def run(st):
    kind, fdzb = st["kind"], st["fdzb"]
    if kind == "frame":
        st["ctx"].launch()
        return {"shadow": st["shadow"], "masks": st["masks"]}
    if kind == "batch":
        st["batch"].launch(st["frames"])
        return {"shadow": [s for s, _ in st["out"]], "masks": [m for _, m in st["out"]]}
    if kind == "shade":
        c = st["case"]
        pos, nrm, g2, g3, shadow, lights = st["shade"]
        fdzb.shade(c["W"], c["H"], pos, nrm, g2, g3, shadow, st["rgba"], SHADE_EYE, SHADE_LA, SHADE_LD, SHADE_LS, lights)
        return {"rgba": st["rgba"]}
    st["raster"].draw(st["desc"])
    if kind == "raster":
        st["raster"].sync()
        return {"g": st["g"], "depth": st["depth"]}
    c = st["case"]
    st["ctx"].launch()
    fdzb.shade(c["W"], c["H"], *st["g"], st["shadow"], st["rgba"], st["eye"], SHADE_LA, SHADE_LD, SHADE_LS,
               st["lights"], stream=st["stream"].cuda_stream)
    return {"rgba": st["rgba"], "shadow": st["shadow"], "g": st["g"]}


# ---- what a pass cannot do without -------------------------------------------

def _frame_work(c, masks=True):
    """Samples, vertices and indices read once, shadows and masks written once; each sample projected and, for the
    bits it decides, tested against one triangle at least; each triangle set up."""
    S, N = c["W"] * c["H"], c["n"] * c["nh"]
    out = 4 + (4 * ((N + 31) // 32) if masks else 0)
    return {"bytes": S * (32 + out) + c["T"] * (3 * 12 + 12), "flops": S * (100 + 164 + 31 * c["n"]) + c["T"] * 250}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        return _frame_work(case)
    if kind == "batch":
        ws = [_frame_work(c) for c in _batch_case(case, 0)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    S = case["W"] * case["H"]
    if kind == "shade":
        return {"bytes": S * (64 + 4 + 16) + 12 * case["lights"], "flops": S * (40 + 70 * case["lights"])}
    T = case["T"] + 2 * case["grid"] ** 2
    V = 3 * case["T"] + (case["grid"] + 1) ** 2
    w = {"bytes": T * 16 + V * 24 + S * 68, "flops": V * 70 + T * 60 + S * 90}
    if kind == "view":
        f = _frame_work(dict(case, nh=case["n"]), masks=False)
        w = {"bytes": w["bytes"] + f["bytes"] + S * 84, "flops": w["flops"] + f["flops"] + S * 110}
    return w


# ---- the same results in 64 bits ---------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "frame" and case["W"] * case["H"] * case["T"] * case["n"] * case["nh"] <= 5e10 and not case["depth"]:
        return {"shadow": _exact_shadow(case, seed), "masks": None}
    if kind == "shade":
        return {"rgba": _exact_shade(case, seed)}
    if kind == "raster":
        return _exact_raster(case, seed)
    return None


def _exact_shadow(case, seed):
    """Occluded fraction of the light, every light sample against every triangle: the oriented planes through the
    sample and the triangle's edges, inside the light-plane rectangle that samples and model share."""
    pos, nrm, vtx, idx = _frame_inputs(case, seed)
    P, Nv, V = pos[:, :3].double(), nrm[:, :3].double(), vtx[:, :3].double()
    if case["xform"]:
        m = torch.from_numpy(_rotation(3.0)).to(DEVICE).double()
        V = V @ m[:3, :3].T + m[:3, 3]
    n, nh, R = case["n"], case["nh"], case["radius"]
    # the light looks down -z, up +y: right = (1, 0, 0), top = (0, 1, 0)
    xf, yf = (n - 1) / n, (nh - 1) / nh
    vec = lambda *v: torch.tensor(v, device=DEVICE, dtype=torch.float64)  # noqa: E731
    corner = lambda sx, sy: vec(sx * xf * R, sy * yf * R, 6.0)  # noqa: E731
    ur, corners = corner(1, 1), [corner(1, 1), corner(-1, 1), corner(-1, -1), corner(1, -1)]
    xd, yd = vec(-2 * R / n, 0, 0), vec(0, -2 * R / nh, 0)
    p00 = 1.0 / math.tan(60.0)
    rf = vec(R * xf * p00, R * yf * p00)

    def project(X):
        w = ur[2] - X[:, 2]
        return (X[:, :2] - ur[:2]) * p00 / w[:, None] * 0.5 + 0.5, w

    shadow = torch.zeros(len(P), device=DEVICE, dtype=torch.float64)
    seen = ~P[:, 0].isnan()
    back = seen & torch.stack([((c - P) * Nv).sum(1) <= 0 for c in corners]).all(0)
    shadow[back] = 1.0
    front = seen & ~back
    uvV, wV = project(V)
    uvS, wS = project(P)
    far = torch.maximum(wS[seen].max(), wV.max()) + 0.1
    hiV, hiS = uvV + rf / wV[:, None] - rf / far, uvS + rf / wS[:, None] - rf / far
    B = torch.maximum(uvV.min(0).values, uvS[front].min(0).values)
    E = torch.minimum(hiV.max(0).values, hiS[front].max(0).values)
    valid = (front & (uvS >= B).all(1) & (hiS <= E).all(1) & (uvS <= hiS).all(1)).nonzero()[:, 0]
    t = idx.long()
    v0, v1, v2 = V[t[:, 0]], V[t[:, 1]], V[t[:, 2]]
    if case["cull"]:
        fn = torch.linalg.cross(v0 - v2, v1 - v0)
        keep = ~torch.stack([((c - v) * fn).sum(1) <= 0 for c in corners for v in (v0, v1, v2)]).all(0)
        t, v0, v1, v2 = t[keep], v0[keep], v1[keep], v2[keep]
    lo, hi, zmin = uvV[t].amin(1), hiV[t].amax(1), wV[t].amin(1)
    fn = torch.linalg.cross(v1 - v0, v2 - v1)
    step = max(1, int(2e7) // max(1, len(t)))
    for k in range(0, len(valid), step):
        s = valid[k:k + step]
        Q = P[s]
        ok = (lo[None] <= uvS[s][:, None]).all(2) & (hiS[s][:, None] <= hi[None]).all(2) & (zmin[None] <= wS[s][:, None])
        a, b = ok.nonzero(as_tuple=True)      # (sample, triangle) pairs whose footprints meet
        if not len(a):
            continue
        q, A0, A1, A2 = Q[a], v0[b], v1[b], v2[b]
        side = ((q - A0) * fn[b]).sum(1)
        cr = torch.linalg.cross
        n1, n2, n3 = cr(A1 - A0, q - A1), cr(A2 - A1, q - A2), cr(A0 - A2, q - A0)
        own = (side.abs() < 1e-3) & ((n1 * n2).sum(1) >= 0) & ((n2 * n3).sum(1) >= 0)
        sg = torch.where(side < 0, -1.0, 1.0)
        planes = []
        for x, y in ((A1, A0 - A1), (A2, A1 - A2), (A0, A2 - A0)):
            nn = cr(x - q, y) * sg[:, None]
            planes.append(((nn * xd).sum(1), (nn * yd).sum(1), (nn * (ur - q)).sum(1)))
        hit = torch.zeros(len(s), n * nh, device=DEVICE, dtype=torch.bool)
        for r in range(n):
            rows = [A * r + C for A, _, C in planes]
            for c in range(nh):
                inside = ~own
                for (_, By, _), row in zip(planes, rows):
                    inside = inside & (row + By * c >= 0)
                hit[a[inside], r * nh + c] = True
        shadow[s] = hit.sum(1).double() / (n * nh)
    return shadow


def _exact_shade(case, seed):
    pos, nrm, g2, g3, shadow, lights = [x.double() for x in _shade_inputs(case, seed)]
    unit = lambda v: v / v.norm(dim=1, keepdim=True)  # noqa: E731
    vec = lambda v: torch.tensor(v, dtype=torch.float32, device=DEVICE).double()  # noqa: E731
    wp, N = pos[:, :3], unit(nrm[:, :3])
    ks = torch.stack([pos[:, 3], nrm[:, 3], g2[:, 3]], 1)
    view = unit(vec(SHADE_EYE) - wp)
    out = torch.zeros_like(wp)
    for lp in lights:
        L = unit(lp - wp)
        ldn = (L * N).sum(1, keepdim=True)
        spec = ((2 * ldn * N - L) * view).sum(1, keepdim=True).clamp_min(0) ** g3[:, 3:4]
        out += vec(SHADE_LA) * g2[:, :3] + (vec(SHADE_LD) * g3[:, :3] * ldn.clamp_min(0) + vec(SHADE_LS) * ks * spec) * (
            1 - shadow[:, None])
    rgba = torch.cat([out / len(lights), torch.ones_like(shadow)[:, None]], 1)
    rgba[shadow.isnan()] = 0.0          # pixels without a shadow value are left as they were
    return rgba


def _exact_raster(case, seed):
    """Coverage at pixel centres of vertices snapped to 1/16 pixel, nearest depth, perspective-correct attributes.  The
    camera sees the whole mesh in front of it, so nothing is clipped."""
    base, vtx, idx, mat, mats, _ = _mesh_inputs(case, seed)
    W, H = case["W"], case["H"]
    vp = torch.from_numpy(np.asarray(base.view_proj, np.float32)).to(DEVICE).double()
    wp, wn = vtx[:, :3].double(), vtx[:, 5:8].double()
    clip = torch.cat([wp, torch.ones_like(wp[:, :1])], 1) @ vp.T
    ndc = clip[:, :3] / clip[:, 3:4]
    X = ((ndc[:, 0] * 0.5 + 0.5) * W * 16).round().long()
    Y = ((ndc[:, 1] * 0.5 + 0.5) * H * 16).round().long()
    z, iw = ndc[:, 2] * 0.5 + 0.5, 1.0 / clip[:, 3]
    t = idx.long()
    area = (X[t[:, 1]] - X[t[:, 0]]) * (Y[t[:, 2]] - Y[t[:, 0]]) - (Y[t[:, 1]] - Y[t[:, 0]]) * (X[t[:, 2]] - X[t[:, 0]])
    t = torch.where((area < 0)[:, None], t[:, [0, 2, 1]], t)
    tx, ty = X[t], Y[t]
    x0, x1 = ((tx.amin(1) + 7) >> 4).clamp_min(0), ((tx.amax(1) - 8) >> 4).clamp_max(W - 1)
    y0, y1 = ((ty.amin(1) + 7) >> 4).clamp_min(0), ((ty.amax(1) - 8) >> 4).clamp_max(H - 1)
    wide, high = (x1 - x0 + 1).clamp_min(0), (y1 - y0 + 1).clamp_min(0)
    count = torch.where(area != 0, wide * high, 0)
    best = torch.full((W * H,), float("inf"), device=DEVICE, dtype=torch.float64)
    winner = torch.full((W * H,), len(t), device=DEVICE, dtype=torch.long)
    ends = count.cumsum(0)
    cuts, total = [0], int(ends[-1])
    for k in range(20_000_000, total, 20_000_000):
        cuts.append(int(torch.searchsorted(ends, k)))
    cuts.append(len(t))

    def weights(tri, px, py):
        cx, cy, e = px * 16 + 8, py * 16 + 8, []
        for i, j in ((1, 2), (2, 0), (0, 1)):
            ax, ay, bx, by = tx[tri, i], ty[tri, i], tx[tri, j], ty[tri, j]
            e.append(((bx - ax) * (cy - ay) - (by - ay) * (cx - ax), (by < ay) | ((by == ay) & (bx > ax))))
        return e

    for a, b in zip(cuts[:-1], cuts[1:]):
        if b <= a:
            continue
        tri = torch.repeat_interleave(torch.arange(a, b, device=DEVICE), count[a:b])
        if not len(tri):
            continue
        at = torch.arange(len(tri), device=DEVICE) - torch.repeat_interleave(ends[a:b] - count[a:b] - (ends[a] - count[a]),
                                                                              count[a:b])
        px, py = x0[tri] + at % wide[tri], y0[tri] + at // wide[tri]
        inside = torch.ones(len(tri), device=DEVICE, dtype=torch.bool)
        e = weights(tri, px, py)
        for v, owns in e:
            inside &= (v > 0) | ((v == 0) & owns)
        tri, pix = tri[inside], (py * W + px)[inside]
        ws = torch.stack([v[inside] for v, _ in e], 1).double()
        d = (ws / ws.sum(1, keepdim=True) * z[t[tri]]).sum(1)
        fine = (d >= 0) & (d <= 1)
        tri, pix, d = tri[fine], pix[fine], d[fine]
        old = best.clone()
        best.scatter_reduce_(0, pix, d, "amin")
        winner[best < old] = len(t)
        first = d == best[pix]
        winner.scatter_reduce_(0, pix[first], tri[first], "amin")
    hit = (winner < len(t)).nonzero()[:, 0]
    tri = winner[hit]
    ws = torch.stack([v for v, _ in weights(tri, hit % W, hit // W)], 1).double() * iw[t[tri]]
    ws = ws / ws.sum(1, keepdim=True)
    m = mats.double()[mat.long()[tri]]
    g = [torch.full((W * H, 4), float("nan"), device=DEVICE, dtype=torch.float64) for _ in range(4)]
    depth = torch.ones(W * H, device=DEVICE, dtype=torch.float64)
    depth[hit] = best[hit]
    g[0][hit] = torch.cat([(ws[:, :, None] * wp[t[tri]]).sum(1), m[:, 6:7]], 1)
    g[1][hit] = torch.cat([(ws[:, :, None] * wn[t[tri]]).sum(1), m[:, 7:8]], 1)
    g[2][hit] = torch.cat([m[:, 0:3], m[:, 8:9]], 1)
    g[3][hit] = torch.cat([m[:, 3:6], m[:, 9:10]], 1)
    return {"g": g, "depth": depth}
