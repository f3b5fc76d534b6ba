"""Timed cases of the library, each through its public entry points.

listed() names the cases, draw() gives more of the same ranges; prepare()
makes what a program holds before the call (scene handle, ray batch, records,
network weights), run() is one pass, work() the bytes and operations a pass
cannot do without, exact() the results in 64 bits where they have a closed
form.  Scenes are displaced icospheres over a ground quad under a lat-long sky
(or the Cornell box), built from the seed on the GPU and handed to the library
as host records, as a program that loads a scene has them.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from kagayaki_gb300 import ESTIMATOR_COMPAT, ESTIMATOR_UNBIASED, Scene, camera_setup, lib, scenes
from kagayaki_gb300._lib import check
from kagayaki_gb300.structs import DISNEY, LAMBERT, RAY, TRIANGLE, KgkSvgfConfig, make_material

DEV = "cuda"
MAX_DEPTH = 16
RECORD_WORDS = 28  # the 112-byte SVGFBuffer record in 4-byte words


def listed():
    return [
        # a picking or visibility query of an interactive tool: a few thousand host rays, small scene
        {"name": "trace_box_host_4k", "kind": "trace", "meshes": 0, "subdiv": 0, "rays": 4096, "host": True},
        # batch closest-hit queries (baking, parity runs) on a 1.3M-triangle field, device rays
        {"name": "trace_field_4m", "kind": "trace", "meshes": 16, "subdiv": 6, "rays": 1 << 22, "host": False},
        # batch occlusion with a range per ray (ambient occlusion, light visibility), a ragged count
        {"name": "occlusion_field_1m", "kind": "occlusion", "meshes": 16, "subdiv": 5, "rays": 1000003},
        # acceleration structure of one edited object group, then its first queries
        {"name": "build_82k", "kind": "build", "meshes": 4, "subdiv": 5, "rays": 65536},
        # acceleration structure of the 5.2M-triangle scene at load, then its first queries
        {"name": "build_5m", "kind": "build", "meshes": 64, "subdiv": 6, "rays": 65536},
        # the reference's estimator at its own picture size: Cornell box, 256 x 256, 16 samples
        {"name": "box_compat_256", "kind": "compat_frame", "width": 256, "height": 256, "spp": 16},
        # the offline frame: 5.2M Disney triangles, HDR sky, 1080p, 64 samples
        {"name": "field_1080p_64spp", "kind": "frame", "meshes": 64, "subdiv": 6, "width": 1920, "height": 1080,
         "spp": 64, "env": 2048},
        # the interactive loop: two 1-sample frames of a moving camera with the standard filter
        {"name": "orbit_1080p_svgf", "kind": "orbit", "meshes": 64, "subdiv": 6, "width": 1920, "height": 1080,
         "env": 2048},
        # a 4K 1-sample frame through the radiance cache (width 128), textured scene, trained every frame
        {"name": "cached_4k", "kind": "cached_frame", "meshes": 64, "subdiv": 6, "textures": 32, "width": 3840,
         "height": 2160, "net": 128, "train_paths": 1 << 18, "env": 2048},
        # ApplySVGF over the reference's own records, at 1080p on device buffers
        {"name": "svgf_apply_1080p", "kind": "svgf_apply", "width": 1920, "height": 1080, "motion": False},
        # cache predictions for the queries of a 1080p frame (width 64)
        {"name": "cache_infer_2m", "kind": "infer", "net": 64, "n": 1 << 21},
        # cache gradients (forward, backward, weight gradients) of the 4K batch (width 128)
        {"name": "cache_gradients_262k", "kind": "gradients", "net": 128, "n": 1 << 18},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "occlusion", "build", "compat_frame", "frame", "orbit", "cached_frame", "svgf_apply",
                       "infer", "gradients"])
    c = {"kind": kind}
    if kind in ("trace", "occlusion", "build"):
        c["subdiv"] = rng.choice([3, 4, 5, 6])
        c["meshes"] = _log_int(rng, 1, 32)
    if kind == "trace":
        c["host"] = rng.random() < 0.3
        c["rays"] = _log_int(rng, 1 << 12, 1 << 20 if c["host"] else 1 << 22)
    elif kind == "occlusion":
        c["rays"] = _log_int(rng, 1 << 12, 1 << 22)
    elif kind == "build":
        c["rays"] = _log_int(rng, 1 << 10, 1 << 17)
    elif kind == "compat_frame":
        c["width"], c["height"] = _log_int(rng, 40, 640), _log_int(rng, 40, 480)
        c["spp"] = rng.randint(1, 16)
    elif kind in ("frame", "orbit", "cached_frame"):
        c["subdiv"] = rng.choice([4, 5, 6])
        c["meshes"] = _log_int(rng, 4, 32)
        c["width"], c["height"] = _log_int(rng, 320, 1920), _log_int(rng, 200, 1080)
        c["env"] = rng.choice([512, 1024])
        if kind == "frame":
            c["spp"] = _log_int(rng, 1, 32)
        if kind == "cached_frame":
            c["textures"] = rng.randint(1, 8)
            c["net"] = rng.choice([64, 128])
            c["train_paths"] = _log_int(rng, 1 << 13, 1 << 17)
    elif kind == "svgf_apply":
        c["width"], c["height"] = _log_int(rng, 64, 2560), _log_int(rng, 64, 1440)
        c["motion"] = rng.random() < 0.5
    elif kind == "infer":
        c["net"], c["n"] = rng.choice([64, 128]), _log_int(rng, 1 << 12, 1 << 21)
    else:
        c["net"], c["n"] = rng.choice([64, 128]), _log_int(rng, 1 << 12, 1 << 18)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * int(seed) + salt)


@functools.lru_cache(maxsize=4)
def _icosphere(subdiv):
    """Unit icosphere: vertices, faces and the faces around every vertex (a
    padded table, so that vertex normals are summed in a fixed order)."""
    v, f = scenes.icosphere(subdiv)
    order = np.argsort(f.reshape(-1), kind="stable")
    vert = f.reshape(-1)[order]
    first = np.searchsorted(vert, np.arange(len(v)))
    around = np.full((len(v), 6), len(f), np.int64)
    around[vert, np.arange(len(vert)) - first[vert]] = order // 3
    return (torch.from_numpy(v).to(DEV, torch.float32), torch.from_numpy(f.astype(np.int64)).to(DEV),
            torch.from_numpy(around).to(DEV))


def _field(seed, meshes, subdiv, textures=0):
    """Displaced icospheres over a ground quad: TRIANGLE and MATERIAL records
    (Disney; with textures the ground is Lambert and every second sphere takes
    its base colour from a texture)."""
    v, f, around = _icosphere(subdiv)
    u = torch.rand((meshes, 16), generator=_gen(seed, 1), device=DEV).cpu().numpy()
    nf, n = len(f), meshes * len(f) + 2
    out = torch.zeros((n, 39), dtype=torch.float32, device=DEV)
    ints = out.view(torch.int32)
    uv = torch.stack([torch.atan2(v[:, 1], v[:, 0]) / (2 * math.pi) + 0.5,
                      torch.acos(v[:, 2].clamp(-1, 1)) / math.pi], 1)
    if textures:
        mats = [make_material(LAMBERT, (0.7, 0.7, 0.7), tex=0)]
    else:
        mats = [make_material(DISNEY, (0.5, 0.5, 0.5), roughness=0.6, specular=0.5)]
    for i in range(meshes):
        r = 0.75 + 1.25 * u[i, 0]
        center = torch.tensor([20 * u[i, 1] - 10, 20 * u[i, 2] - 10, r + u[i, 3] * (20 - r)], device=DEV,
                              dtype=torch.float32)
        noise = torch.zeros(len(v), device=DEV)
        for k in range(3):
            ph = 6.2831853 * u[i, 4 + k]
            w = v * float(5 * 2 ** k)
            noise += 0.5 ** k * torch.sin(w[:, 0] + ph) * torch.sin(w[:, 1] + 2 * ph) * torch.sin(w[:, 2] + 3 * ph)
        pos = v * (float(r) * (1 + 0.05 * noise))[:, None] + center
        p = pos[f]  # (faces, 3, 3)
        fn = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        near = torch.cat([fn, torch.zeros((1, 3), device=DEV)])[around]
        vn = near[:, 0]
        for k in range(1, 6):
            vn = vn + near[:, k]
        vn = vn / torch.sqrt((vn * vn).sum(1, keepdim=True))
        t = out[i * nf:(i + 1) * nf, :36].view(nf, 9, 4)
        t[:, 0:3, :3] = p
        t[:, 3:6, :3] = vn[f]
        t[:, 6:9, :2] = uv[f]
        q = ints[i * nf:(i + 1) * nf]
        q[:, 36], q[:, 37], q[:, 38] = 1 + i, 1, i
        mats.append(make_material(
            DISNEY, tuple(0.05 + 0.9 * u[i, 7:10]), metallic=1.0 if u[i, 10] < 0.3 else 0.0,
            roughness=0.05 + 0.95 * u[i, 11], specular=0.5, clearcoat=u[i, 12],
            tex=(1 + i // 2) % textures if textures and i % 2 == 0 else -1))
    g = 100.0
    quad = np.array([[-g, -g, 0], [g, -g, 0], [g, g, 0], [-g, g, 0]], np.float32)
    for k, idx in enumerate(([0, 1, 2], [0, 2, 3])):
        t = out[n - 2 + k, :36].view(9, 4)
        t[0:3, :3] = torch.from_numpy(quad[idx]).to(DEV)
        t[3:6, 2] = 1.0
        t[6:9, :2] = torch.from_numpy(quad[idx][:, :2] / 25.0).to(DEV)
        ints[n - 2 + k, 38] = meshes
    return out.cpu().numpy().view(np.uint8).reshape(-1).view(TRIANGLE), np.stack(mats)


def _sky(seed, width):
    """Lat-long RGB sky with a sun lobe (peak 1e4, sigma 1 degree)."""
    u = torch.rand(2, generator=_gen(seed, 2), device=DEV).cpu().numpy()
    height = width // 2
    el, az = math.radians(20 + 40 * u[0]), 2 * math.pi * u[1]
    sun = torch.tensor([math.cos(el) * math.cos(az), math.cos(el) * math.sin(az), math.sin(el)], device=DEV)
    phi = (0.5 - (torch.arange(height, device=DEV) + 0.5) / height) * math.pi
    theta = (0.5 - (torch.arange(width, device=DEV) + 0.5) / width) * 2 * math.pi
    cp = torch.cos(phi)[:, None]
    d = torch.stack([cp * torch.cos(theta), cp * torch.sin(theta), torch.sin(phi)[:, None].expand(height, width)], -1)
    t = torch.sqrt(d[..., 2].clamp(0, 1))[..., None]
    sky = torch.tensor([1.1, 1.05, 1.0], device=DEV) * (1 - t) + torch.tensor([0.25, 0.45, 0.95], device=DEV) * t
    img = torch.where((d[..., 2] >= 0)[..., None], sky, torch.tensor([0.18, 0.16, 0.14], device=DEV))
    ang = torch.acos((d * sun).sum(-1).clamp(-1, 1))
    lobe = 1e4 * torch.exp(-0.5 * (ang / math.radians(1.0)) ** 2)
    return (img + lobe[..., None] * torch.tensor([1.0, 0.95, 0.85], device=DEV)).cpu().numpy()


def _textures(seed, n, size=1024):
    """RGBA8 textures: a checker of two colours under smooth noise."""
    u = torch.rand((n, 8), generator=_gen(seed, 3), device=DEV)
    g = (torch.arange(size, device=DEV) + 0.5) / size
    out = []
    for k in range(n):
        period = 4 + int(28 * u[k, 0])
        c = (torch.floor(g * period)[:, None] + torch.floor(g * period)[None, :]) % 2
        low = torch.rand((1, 1, 32, 32), generator=_gen(seed, 100 + k), device=DEV)
        noise = torch.nn.functional.interpolate(low, (size, size), mode="bilinear", align_corners=False)[0, 0]
        w = (0.5 * c + 0.5 * noise)[..., None]
        rgb = u[k, 1:4] * (1 - w) + u[k, 4:7] * w
        img = torch.full((size, size, 4), 255, dtype=torch.uint8, device=DEV)
        img[..., :3] = (rgb * 255).to(torch.uint8)
        out.append(img.cpu().numpy())
    return out


def _box(seed):
    """The Cornell box with wall and box colours and a camera of the seed."""
    tris, mats, cam = scenes.cornell_box()
    u = torch.rand(16, generator=_gen(seed, 4), device=DEV).cpu().numpy()
    mats = mats.copy()
    for k in range(3):
        mats["diffuse"][k, :3] = 0.05 + 0.8 * u[3 * k:3 * k + 3]
    org = [cam["origin"][a] + 0.5 * (u[10 + a] - 0.5) for a in range(3)]
    return tris, mats, (org, cam["dist"], cam["rot"])


def _orbit(seed, frame, height, radius=25.0, z=6.0, target=8.0):
    ang = (61.803 * seed) % 360.0 + 6.0 * frame
    a = math.radians(ang)
    pitch = math.degrees(math.atan2(z - target, radius))
    return camera_setup((radius * math.cos(a), radius * math.sin(a), z), 28.0, (90.0 - pitch, 0.0, ang + 90.0), height)


def _rays(seed, n, lo, hi):
    """Origins uniform in the box, directions uniform on the sphere: kgk_ray
    records (10 words) on the GPU."""
    g = _gen(seed, 5)
    r = torch.zeros((n, 10), device=DEV)
    d = torch.randn((n, 3), generator=g, device=DEV)
    r[:, 0:3] = d / torch.sqrt((d * d).sum(1, keepdim=True))
    lo, hi = torch.tensor(lo, device=DEV), torch.tensor(hi, device=DEV)
    r[:, 4:7] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=DEV)
    return r


FIELD_BOX = ((-12.0, -12.0, 0.05), (12.0, 12.0, 20.0))
CORNELL_BOX = ((-4.99, 0.01, -4.99), (4.99, 9.99, 4.99))


def _queries(seed, n):
    """Raw cache queries: position in [0, 1]^3, unit normal and view, roughness, albedo."""
    g = _gen(seed, 6)
    q = torch.rand((n, 13), generator=g, device=DEV)
    for a in (3, 6):
        d = torch.randn((n, 3), generator=g, device=DEV)
        q[:, a:a + 3] = d / torch.sqrt((d * d).sum(1, keepdim=True))
    return q


def _weights(seed, net):
    """He-uniform weights, layer by layer (out, in) row-major."""
    g = _gen(seed, 7)
    ws = []
    for fan_in, fan_out in [(64, net)] + 4 * [(net, net)] + [(net, 3)]:
        ws.append((2 * torch.rand((fan_out, fan_in), generator=g, device=DEV) - 1) * math.sqrt(6.0 / fan_in))
    return ws


def _targets(seed, n):
    """Radiance samples of a path tracer: positive, long-tailed."""
    return -torch.log1p(-torch.rand((n, 3), generator=_gen(seed, 8), device=DEV))


def _svgf_inputs(seed, W, H, motion):
    """A 1-sample frame of spheres on a plane under a sky, as the renderer
    leaves it: noisy radiance (H, W, 4), this frame's records and the previous
    frame's (H, W, 28 words).  With motion the records carry the previous
    position of their pixel, else -1 as the reference's camera leaves them."""
    g = _gen(seed, 9)
    u = torch.rand((12, 8), generator=g, device=DEV).cpu().numpy()
    y, x = torch.meshgrid(torch.arange(H, device=DEV), torch.arange(W, device=DEV), indexing="ij")
    d = torch.stack([(x - W / 2) / H, torch.ones((H, W), device=DEV) * 1.2, (H / 2 - y) / H], -1).float()
    d = d / torch.sqrt((d * d).sum(-1, keepdim=True))
    org = torch.tensor([0.0, -8.0, 3.0], device=DEV)
    t = torch.where(d[..., 2] < -1e-3, -org[2] / d[..., 2].clamp(max=-1e-3), torch.full((H, W), 1e30, device=DEV))
    t = torch.where(t > 60.0, torch.full_like(t, 1e30), t)
    obj = torch.where(t < 1e29, 0, -1)
    nrm = torch.tensor([0.0, 0.0, 1.0], device=DEV).expand(H, W, 3).clone()
    alb = torch.tensor([0.5, 0.5, 0.5], device=DEV).expand(H, W, 3).clone()
    emi = torch.zeros((H, W, 3), device=DEV)
    for i in range(len(u)):
        r = 0.5 + 1.5 * float(u[i, 0])
        c = torch.tensor([8 * u[i, 1] - 4, 10 * u[i, 2], r + 3 * u[i, 3]], device=DEV, dtype=torch.float32)
        oc = org - c
        b = (d * oc).sum(-1)
        disc = b * b - (oc * oc).sum() + r * r
        ts = -b - torch.sqrt(disc.clamp(min=0))
        hit = (disc > 0) & (ts > 0) & (ts < t)
        t = torch.where(hit, ts, t)
        obj = torch.where(hit, 1 + i, obj)
        n = (org + d * ts[..., None] - c) / r
        nrm = torch.where(hit[..., None], n, nrm)
        alb = torch.where(hit[..., None], torch.tensor(0.05 + 0.9 * u[i, 4:7], device=DEV, dtype=torch.float32), alb)
        if i == 0:
            emi = torch.where(hit[..., None], torch.tensor([4.0, 3.0, 2.0], device=DEV), emi)
        else:
            emi = torch.where(hit[..., None], torch.zeros(3, device=DEV), emi)
    seen = obj >= 0
    sun = torch.tensor([0.4, -0.6, 0.69], device=DEV)
    light = 0.3 + 2.0 * (nrm * sun).sum(-1).clamp(min=0)
    sample = -torch.log1p(-torch.rand((H, W, 3), generator=g, device=DEV))
    sample = torch.where(torch.rand((H, W, 1), generator=g, device=DEV) < 0.25, torch.zeros_like(sample), sample)
    rad = torch.where(seen[..., None], alb * light[..., None] * sample + emi + 1e-4,
                      torch.tensor([0.4, 0.6, 0.9], device=DEV))
    noisy = torch.zeros((H, W, 4), device=DEV)
    noisy[..., :3] = rad

    def records():
        r = torch.zeros((H, W, RECORD_WORDS), device=DEV)
        i = r.view(torch.int32)
        r[..., 0:3] = torch.where(seen[..., None], alb, torch.zeros_like(alb))
        r[..., 4:7] = torch.where(seen[..., None], emi, torch.zeros_like(emi))
        r[..., 8:11] = torch.where(seen[..., None], nrm, torch.zeros_like(nrm))
        i[..., 16] = obj
        i[..., 17] = obj
        i[..., 18:20] = -1
        r[..., 20:22] = -1.0
        r[..., 23:25] = -1.0
        r[..., 26] = torch.where(seen, t, torch.zeros_like(t))
        i[..., 27] = 1  # willApplyATrousFilter, no temporal accumulation
        return r, i

    cur, ci = records()
    prev, pi = records()
    if motion:
        dx, dy = int(8 * u[0, 7]) - 4, int(6 * u[1, 7]) - 3
        px, py = x - dx, y - dy
        ok = seen & (px >= 0) & (px < W - 1) & (py >= 0) & (py < H - 1)
        ok &= torch.rand((H, W), generator=g, device=DEV) > 0.02
        ci[..., 18] = torch.where(ok, px, -1)
        ci[..., 19] = torch.where(ok, py, -1)
        frac = torch.rand((H, W, 2), generator=g, device=DEV)
        cur[..., 20] = torch.where(ok, px + frac[..., 0], -1.0)
        cur[..., 21] = torch.where(ok, py + frac[..., 1], -1.0)
        prev[..., 12:15] = alb * light[..., None] + emi
        m1 = light * (0.8 + 0.4 * torch.rand((H, W), generator=g, device=DEV))
        prev[..., 23] = m1
        prev[..., 24] = m1 * m1 * (1.2 + torch.rand((H, W), generator=g, device=DEV))
        pi[..., 22] = torch.randint(1, 9, (H, W), generator=g, device=DEV, dtype=torch.int32)
        pi[..., 27] = torch.where(seen, 0x101, 1)
    return noisy, cur, prev


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _triangles(c):
    return 36 if c["meshes"] == 0 else c["meshes"] * 20 * 4 ** c["subdiv"] + 2


def prepare(case, seed):
    c = dict(case)
    k = c["kind"]
    s = {"case": c}
    if k in ("trace", "occlusion", "build"):
        if c["meshes"]:
            tris, mats = _field(seed, c["meshes"], c["subdiv"])
            lo, hi = FIELD_BOX
        else:
            tris, mats, _ = _box(seed)
            lo, hi = CORNELL_BOX
        s["scene"] = Scene(tris, mats)
        if k != "build":
            s["scene"].build_bvh()
        rays = _rays(seed, c["rays"], lo, hi)
        if c.get("host"):
            s["rays"] = rays.cpu().numpy().view(np.uint8).reshape(-1).view(RAY)
        else:
            s["rays"] = rays
            s["ids"] = torch.empty(c["rays"], dtype=torch.int32, device=DEV)
            s["t"] = torch.empty(c["rays"], device=DEV)
        if k == "occlusion":
            s["tmax"] = 0.5 + 10 * torch.rand(c["rays"], generator=_gen(seed, 10), device=DEV)
            s["occ"] = torch.empty(c["rays"], dtype=torch.uint8, device=DEV)
    elif k == "compat_frame":
        tris, mats, cam = _box(seed)
        s["scene"] = Scene(tris, mats)
        s["scene"].build_bvh()
        s["cam"] = camera_setup(*cam, c["height"])
        s["out"] = torch.empty((c["height"], c["width"], 4), device=DEV)
    elif k in ("frame", "orbit", "cached_frame"):
        ntex = c.get("textures", 0)
        tris, mats = _field(seed, c["meshes"], c["subdiv"], ntex)
        place = [np.zeros((1, 1, 3), np.float32)] * ntex
        s["scene"] = Scene(tris, mats, textures=place, env=_sky(seed, c["env"]))
        if ntex:
            s["scene"].set_textures_rgba8(_textures(seed, ntex))
        s["scene"].build_bvh()
        s["cams"] = [_orbit(seed, f, c["height"]) for f in range(2)]
        s["seed"] = 1 + int(seed)
        s["out"] = [torch.empty((c["height"], c["width"], 4), device=DEV) for _ in range(2 if k == "orbit" else 1)]
        if k == "cached_frame":
            s["scene"].cache_init(width=c["net"], train_paths=c["train_paths"], seed=1 + int(seed))
            s["weights"] = torch.cat([w.reshape(-1) for w in _weights(seed, c["net"])])
    elif k == "svgf_apply":
        s["noisy"], s["rec"], s["prev"] = _svgf_inputs(seed, c["width"], c["height"], c["motion"])
        s["result"], s["cur"] = torch.empty_like(s["noisy"]), torch.empty_like(s["rec"])
        s["filtered"] = torch.empty_like(s["noisy"])
    else:
        tris, mats, _ = _box(seed)
        s["scene"] = Scene(tris, mats)
        s["scene"].cache_init(width=c["net"], seed=1)
        s["params"] = torch.cat([w.reshape(-1) for w in _weights(seed, c["net"])])
        check(lib().kgk_nrc_set_weights(s["scene"]._h, _ptr(s["params"]), s["params"].numel()))
        s["raw"] = _queries(seed, c["n"])
        if k == "infer":
            s["y"] = torch.empty((c["n"], 3), device=DEV)
        else:
            s["target"] = _targets(seed, c["n"])
            s["grad"] = np.empty(s["params"].numel(), np.float32)
            s["loss"] = np.empty(1, np.float32)
    torch.cuda.synchronize()  # the library works on streams of its own
    return s


def _closest(s):
    check(lib().kgk_trace_closest(s["scene"]._h, _ptr(s["rays"]), s["case"]["rays"], _ptr(s["ids"]), _ptr(s["t"]),
                                  None))
    return [s["ids"], s["t"]]


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "trace":
        return list(s["scene"].trace_closest(s["rays"])) if c["host"] else _closest(s)
    if k == "occlusion":
        check(lib().kgk_trace_any(s["scene"]._h, _ptr(s["rays"]), _ptr(s["tmax"]), c["rays"], _ptr(s["occ"]), None))
        return s["occ"]
    if k == "build":
        s["scene"].build_bvh()
        return _closest(s)
    if k == "compat_frame":
        s["scene"].render(s["cam"], c["width"], c["height"], spp=c["spp"], estimator=ESTIMATOR_COMPAT,
                          out=s["out"].data_ptr())
        return s["out"]
    if k == "frame":
        s["scene"].render(s["cams"][0], c["width"], c["height"], spp=c["spp"], max_depth=MAX_DEPTH,
                          estimator=ESTIMATOR_UNBIASED, seed=s["seed"], out=s["out"][0].data_ptr())
        return s["out"][0]
    if k == "orbit":
        cfg = KgkSvgfConfig(mode=1, width=c["width"], height=c["height"], atrous_iterations=5, alpha=0.2,
                            sigma_z=1.0, sigma_n=128.0, sigma_l=4.0)
        for f in range(2):
            s["scene"].render(s["cams"][f], c["width"], c["height"], spp=1, max_depth=MAX_DEPTH,
                              estimator=ESTIMATOR_UNBIASED, seed=s["seed"], frame_index=f, write_gbuffer=True,
                              keep_on_device=True)
            cfg.frame_index = f
            s["scene"].svgf_output(cfg, filtered=s["out"][f].data_ptr(), async_=True)
        s["scene"].sync()
        return s["out"]
    if k == "cached_frame":
        check(lib().kgk_nrc_set_weights(s["scene"]._h, _ptr(s["weights"]), s["weights"].numel()))
        s["scene"].render(s["cams"][0], c["width"], c["height"], spp=1, max_depth=MAX_DEPTH,
                          estimator=ESTIMATOR_UNBIASED, seed=s["seed"], use_cache=True, texture_filter=1,
                          out=s["out"][0].data_ptr())
        return s["out"][0]
    if k == "svgf_apply":
        # what the renderer writes anew for every frame
        s["result"].copy_(s["noisy"])
        s["cur"].copy_(s["rec"])
        torch.cuda.current_stream().synchronize()  # the call works on a stream of its own
        check(lib().kgk_svgf_apply(_ptr(s["result"]), _ptr(s["filtered"]), _ptr(s["prev"]), _ptr(s["cur"]),
                                   c["width"], c["height"], 1 if c["motion"] else 0))
        return {"result": s["result"], "filtered": s["filtered"], "moments": s["cur"][..., 23:26],
                "samples": s["cur"].view(torch.int32)[..., 22]}
    if k == "infer":
        check(lib().kgk_nrc_infer(s["scene"]._h, _ptr(s["raw"]), c["n"], _ptr(s["y"])))
        return s["y"]
    check(lib().kgk_nrc_gradients(s["scene"]._h, _ptr(s["raw"]), _ptr(s["target"]), c["n"],
                                  ctypes.c_void_p(s["grad"].ctypes.data), ctypes.c_void_p(s["loss"].ctypes.data)))
    return {"grad": s["grad"], "loss": s["loss"]}


def _macs(net):
    return 64 * net + 4 * net * net + 3 * net


def work(case):
    """A ray reads 40 B and writes 8 B (1 B for occlusion); it passes about
    log8(triangles) wide nodes (8 children x 12 operations) and one triangle
    (30).  A scene's triangles (three corners, 36 B) are read once."""
    c = case
    k = c["kind"]
    if k in ("trace", "occlusion", "build", "frame", "orbit", "cached_frame"):
        n = _triangles(c)
        per_ray = 96 * max(1.0, math.log(n, 8)) + 30
    if k == "trace":
        return {"bytes": 48 * c["rays"] + 36 * n, "flops": c["rays"] * per_ray}
    if k == "occlusion":
        return {"bytes": 45 * c["rays"] + 36 * n, "flops": c["rays"] * per_ray}
    if k == "build":
        # corners in, triangle records (48 B) and nodes (80 B, one per five triangles) out; a box per level
        return {"bytes": (36 + 48 + 16) * n + 48 * c["rays"], "flops": n * 12 * math.log2(n) + c["rays"] * per_ray}
    if k == "compat_frame":
        px = c["width"] * c["height"]
        return {"bytes": 16 * px, "flops": px * c["spp"] * 5 * 300}
    if k in ("frame", "orbit", "cached_frame"):
        px = c["width"] * c["height"]
        paths = px * (c["spp"] if k == "frame" else 2 if k == "orbit" else 1)
        bytes_ = 36 * n + 12 * c["env"] * c["env"] // 2 + 16 * px * (2 if k == "orbit" else 1)
        flops = paths * 2 * per_ray
        if k == "orbit":
            flops += 2 * px * 6 * 25 * 20
        if k == "cached_frame":
            flops += 2 * _macs(c["net"]) * (0.5 * px + 3 * 4 * c["train_paths"])
        return {"bytes": bytes_, "flops": flops}
    if k == "svgf_apply":
        px = c["width"] * c["height"]
        return {"bytes": px * (3 * 112 + 3 * 16), "flops": px * 25 * 25 * 25}
    bytes_ = 4 * 13 * c["n"] + 12 * c["n"] + 4 * _macs(c["net"])
    return {"bytes": bytes_ + (4 * _macs(c["net"]) if k == "gradients" else 0),
            "flops": 2 * _macs(c["net"]) * c["n"] * (1 if k == "infer" else 3)}


# ---------------------------------------------------------------------------
# results in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    c = dict(case)
    if c["kind"] == "trace" and c["meshes"] == 0:
        return _exact_trace(c, seed)
    if c["kind"] == "svgf_apply":
        return _exact_svgf(*_svgf_inputs(seed, c["width"], c["height"], c["motion"]), 1 if c["motion"] else 0)
    if c["kind"] == "infer":
        w = [x.double() for x in _weights(seed, c["net"])]
        raw = _queries(seed, c["n"])
        return torch.cat([_mlp(w, raw[i:i + 65536].double())[0] for i in range(0, c["n"], 65536)])
    if c["kind"] == "gradients":
        return _exact_gradients(c, seed)
    return None


def _exact_trace(c, seed):
    """Closest hits of the box's 36 triangles, every pair tested in 64 bits."""
    tris, _, _ = _box(seed)
    v = torch.from_numpy(tris["verts"][:, :3, :3].astype(np.float64)).to(DEV)
    r = _rays(seed, c["rays"], *CORNELL_BOX).double()
    d, o = r[:, None, 0:3], r[:, None, 4:7]
    e1, e2 = (v[:, 1] - v[:, 0])[None], (v[:, 2] - v[:, 0])[None]
    h = torch.linalg.cross(d.expand(-1, len(v), 3), e2.expand(len(r), -1, 3))
    inv = 1.0 / (h * e1).sum(-1)
    so = o - v[None, :, 0]
    a = (so * h).sum(-1) * inv
    q = torch.linalg.cross(so, e1.expand(len(r), -1, 3))
    b = (d * q).sum(-1) * inv
    t = (e2 * q).sum(-1) * inv
    t = torch.where((a >= 0) & (b >= 0) & (a + b <= 1) & (t >= 1e-5), t, torch.full_like(t, float(np.float32(1e38))))
    return [None, t.min(1).values]


def _mlp(w, raw):
    """The network's outputs and activations: 64 features (sines and cosines
    of six octaves per position axis, normal and view with theirs, roughness,
    albedo, six ones), five ReLU layers, three linear outputs."""
    f = []
    for ax in range(3):
        for k in range(6):
            x = math.pi * 2.0 ** k * raw[:, ax]
            f += [torch.sin(x), torch.cos(x)]
    f += [raw[:, j] for j in range(3, 9)]
    for j in range(3, 9):
        f += [torch.sin(math.pi * raw[:, j]), torch.cos(math.pi * raw[:, j])]
    f += [raw[:, j] for j in range(9, 13)]
    f += [torch.ones_like(raw[:, 0])] * 6
    acts = [torch.stack(f, 1)]
    for l in range(5):
        acts.append(torch.relu(acts[-1] @ w[l].T))
    return acts[-1] @ w[5].T, acts


def _exact_gradients(c, seed):
    """Mean relative-L2 loss ((y - t)^2 / (y^2 + 0.01), the denominator held)
    and its gradient."""
    w = [x.double() for x in _weights(seed, c["net"])]
    raw, target = _queries(seed, c["n"]), _targets(seed, c["n"])
    g = [torch.zeros_like(x) for x in w]
    loss = torch.zeros(1, dtype=torch.float64, device=DEV)
    for i in range(0, c["n"], 65536):
        y, acts = _mlp(w, raw[i:i + 65536].double())
        diff = y - target[i:i + 65536].double()
        den = y * y + 0.01
        loss += (diff * diff / den).sum() / (3.0 * c["n"])
        dz = 2.0 * diff / den / (3.0 * c["n"])
        for l in range(5, -1, -1):
            g[l] += dz.T @ acts[l]
            if l:
                dz = (dz @ w[l]) * (acts[l] > 0)
    return {"grad": torch.cat([x.reshape(-1) for x in g]), "loss": loss}


def _shift(a, dx, dy, fill):
    """b[y, x] = a[y + dy, x + dx], `fill` where that lies outside."""
    H, W = a.shape[:2]
    b = torch.full_like(a, fill)
    if abs(dx) < W and abs(dy) < H:
        b[max(0, -dy):H - max(0, dy), max(0, -dx):W - max(0, dx)] = \
            a[max(0, dy):H - max(0, -dy), max(0, dx):W - max(0, -dx)]
    return b


def _exact_svgf(noisy, cur, prev, frame):
    """ApplySVGF with a full-image barrier at each of its barriers, in 64
    bits: temporal accumulation, moments and their 7 x 7 edge-stopped
    estimate, the 3 x 3 blur of the variance, five rounds of five 5 x 5
    edge-stopping passes (steps 1 to 16) blended 0.2 : 0.8 with their input."""
    f32 = lambda v: float(np.float32(v))  # noqa: E731  (the constants are floats)
    S = f32(1e-4)
    lum = lambda v: (v * torch.tensor([f32(0.2126), f32(0.7152), f32(0.0722)], device=DEV,  # noqa: E731
                                      dtype=torch.float64)).sum(-1)
    H, W = noisy.shape[:2]
    R = noisy[..., :3].double()
    R = torch.where(torch.isfinite((R * R).sum(-1, keepdim=True)), R, torch.zeros_like(R))
    ci, pi = cur.view(torch.int32), prev.view(torch.int32)
    alb, nrm, depth = cur[..., 0:3].double(), cur[..., 8:11].double(), cur[..., 26].double()
    emi = cur[..., 4:7].double()
    obj, mat = ci[..., 16].long(), ci[..., 17].long()
    px, py = ci[..., 18].long(), ci[..., 19].long()
    samples = ci[..., 22].long()
    if frame == 0:
        p_hist, p_flag = torch.zeros_like(R), torch.zeros_like(obj, dtype=torch.bool)
        p_mat, p_n = torch.full_like(obj, -1), torch.zeros_like(obj)
        p_m1 = torch.full_like(depth, -1.0)
        p_m2 = p_m1.clone()
    else:
        p_hist, p_flag, p_mat = prev[..., 12:15].double(), (pi[..., 27] & 0xff00) != 0, pi[..., 17].long()
        p_n, p_m1, p_m2 = pi[..., 22].long(), prev[..., 23].double(), prev[..., 24].double()
    m1o, m2o = cur[..., 23].double(), cur[..., 24].double()
    first = lum(R / alb)
    m1o = torch.where(p_m1 == -1.0, first, m1o)
    m2o = torch.where(p_m1 == -1.0, first * first, m2o)
    # temporal accumulation
    fs, ft = cur[..., 20].double() - px, cur[..., 21].double() - py
    hsum, hw = torch.zeros_like(R), torch.zeros_like(depth)
    for ox, oy, w in ((0, 0, (1 - fs) * (1 - ft)), (1, 0, fs * (1 - ft)), (0, 1, (1 - fs) * ft), (1, 1, fs * ft)):
        qx, qy = px + ox, py + oy
        inside = (qx >= 0) & (qx < W) & (qy >= 0) & (qy < H)
        q = (qy.clamp(0, H - 1), qx.clamp(0, W - 1))
        ok = inside & (p_mat[q] == mat) & p_flag[q]
        hsum += torch.where(ok[..., None], p_hist[q] * w[..., None], torch.zeros_like(R))
        hw += torch.where(ok, w, torch.zeros_like(w))
    use = ((emi * emi).sum(-1) == 0) & (hw != 0)
    R = torch.where(use[..., None], R * f32(0.2) + hsum / torch.where(use, hw, torch.ones_like(hw))[..., None] * f32(0.8), R)
    # moments
    l = lum(R / (alb + S))
    M1, M2 = l, l * l
    prv = (py.clamp(0, H - 1), px.clamp(0, W - 1))
    lin = W * py + px
    spatial = (px == -1) | (lin < 0) | (lin >= W * H) | (p_n[prv] < 3)
    sx = torch.where(torch.arange(W, device=DEV) < W // 2, 1, -1)[None, :].expand(H, W)
    sy = torch.where(torch.arange(H, device=DEV) < H // 2, 1, -1)[:, None].expand(H, W)
    yy, xx = torch.meshgrid(torch.arange(H, device=DEV), torch.arange(W, device=DEV), indexing="ij")
    grad = lambda dep: ((dep[yy, xx + sx] - dep) / sx, (dep[yy + sy, xx] - dep) / sy)  # noqa: E731
    gx, gy = grad(depth)
    n_new = p_n[prv] + 1
    cw = torch.where(n_new < 5, 1.0 / n_new.double().clamp(min=1), torch.full_like(depth, f32(1.0 / 5.0)))
    m1o = torch.where(spatial, m1o, (1 - cw) * p_m1[prv] + cw * M1)
    m2o = torch.where(spatial, m2o, (1 - cw) * p_m2[prv] + cw * M2)
    samples = torch.where(spatial, samples, n_new)
    M1, M2 = torch.where(spatial, M1, m1o), torch.where(spatial, M2, m2o)

    def depth_w(d, nd, dx, dy):
        return torch.exp(-torch.abs(d - nd) / (torch.abs(dx * gx + dy * gy) + S))

    K7 = [f32(v) for v in (0.00598, 0.060626, 0.241843, 0.383103, 0.241843, 0.060626, 0.00598)]
    s1, s2, sw = torch.zeros_like(depth), torch.zeros_like(depth), torch.zeros_like(depth)
    for kx in range(-3, 4):
        for ky in range(-3, 4):
            h = K7[kx + 3] * K7[ky + 3]
            if kx == 0 and ky == 0:
                s1, s2, sw = s1 + h * M1, s2 + h * M2, sw + h
                continue
            ok = (_shift(obj, kx, ky, -1) != -1) & (_shift(mat, kx, ky, -1) == mat)
            wn = (nrm * _shift(nrm, kx, ky, 0)).sum(-1).clamp(min=0) ** 128
            w = torch.where(ok, h * depth_w(depth, _shift(depth, kx, ky, 0), kx, ky) * wn, torch.zeros_like(depth))
            s1, s2, sw = s1 + w * _shift(M1, kx, ky, 0), s2 + w * _shift(M2, kx, ky, 0), sw + w
    F = torch.zeros_like(R)
    reset = (obj == -1) | (spatial & (sw == 0))
    keep = ~reset
    est = keep & spatial
    m1o, m2o = torch.where(est, s1 / sw, m1o), torch.where(est, s2 / sw, m2o)
    samples = torch.where(est, torch.where(px == -1, torch.ones_like(samples), n_new), samples)
    F = torch.where(reset[..., None], R, F)
    filt = keep & ((ci[..., 27] & 0xff) != 0)
    zero, neg = torch.zeros_like(depth), torch.full_like(depth, -1.0)
    obj, mat = torch.where(reset, -1, obj), torch.where(reset, -1, mat)
    depth, m1o, m2o = torch.where(reset, zero, depth), torch.where(reset, neg, m1o), torch.where(reset, neg, m2o)
    alb, nrm = torch.where(keep[..., None], alb, 0 * alb), torch.where(keep[..., None], nrm, 0 * nrm)
    hist = torch.where(keep[..., None], cur[..., 12:15].double(), 0 * alb)
    samples = torch.where(reset, 0, samples)
    var = torch.where(reset, zero, cur[..., 25].double())
    var = torch.where(obj != -1, (m2o - m1o * m1o).clamp(0, 1000), var)
    # 3 x 3 blur of the variance
    KG = (0.25, 0.5, 0.25)
    gs, gw = zero.clone(), zero.clone()
    for kx in range(-1, 2):
        for ky in range(-1, 2):
            w = torch.where(_shift(obj, kx, ky, -1) != -1, KG[kx + 1] * KG[ky + 1], 0.0).double()
            gs, gw = gs + w * _shift(var, kx, ky, 0), gw + w
    flat, none = (gs == 0) & (gw != 0), gw == 0
    F = torch.where(flat[..., None], R, F)
    filt = filt & ~flat & ~none
    m1o, m2o = torch.where(none, neg, m1o), torch.where(none, neg, m2o)
    samples = torch.where(none, 0, samples)
    blurred = torch.where(flat | none, zero, gs / torch.where(gw == 0, torch.ones_like(gw), gw))
    var = torch.where(flat | none, var, blurred)
    sd = torch.sqrt(blurred)
    gx, gy = grad(depth)
    KW = torch.tensor([1, 4, 6, 4, 1], dtype=torch.float64)
    for _ in range(5):
        for stage in range(5):
            step = 1 << stage
            dm = R / (alb + S)
            l = lum(dm)
            srad, svar, swt = 0 * R, 0 * depth, 0 * depth
            for ki in range(25):
                ox, oy = (ki % 5 - 2) * step, (ki // 5 - 2) * step
                h = float(KW[ki % 5] * KW[ki // 5] / 256)
                if ki == 12:
                    srad, svar, swt = srad + dm * h, svar + h * h * var, swt + h
                    continue
                nl = _shift(l, ox, oy, 0)
                ok = _shift(obj, ox, oy, -1) != -1
                ok &= _shift(mat, ox, oy, -1) == mat
                ok &= ~(((l > 0.5) & (nl > 5 * l)) | ((l > 0.1) & (nl > 50 * l)) | ((l > S) & (nl > 100 * l)))
                w = h * depth_w(depth, _shift(depth, ox, oy, 0), xx + ox, yy + oy)
                w = w * (nrm * _shift(nrm, ox, oy, 0)).sum(-1).clamp(min=0) ** 128
                wl = torch.exp(-torch.abs(l - nl) / (4 * sd + S))
                w = torch.where(ok, torch.where(filt, w * wl, w), zero)
                srad, svar, swt = srad + _shift(dm, ox, oy, 0) * w[..., None], svar + w * w * _shift(var, ox, oy, 0), swt + w
            skip = (obj == -1) | (swt < f32(1e-6)) | (swt * swt < f32(1e-6))
            out = (srad / swt[..., None] * alb) * f32(0.2) + R * (1 - f32(0.2))
            F = torch.where(((obj != -1) & skip)[..., None], R, torch.where(skip[..., None], F, out))
            if stage == 0:
                hist = torch.where(skip[..., None], hist, out)
            R = torch.where(skip[..., None], R, out)
            var = torch.where(skip | ~filt, var, f32(0.2) * var + (1 - f32(0.2)) * svar / (swt * swt))
    full = lambda v: torch.cat([v, torch.zeros_like(v[..., :1])], -1)  # noqa: E731
    return {"result": full(hist), "filtered": full(F), "moments": torch.stack([m1o, m2o, var], -1), "samples": None}
