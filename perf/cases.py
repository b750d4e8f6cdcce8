"""Performance cases of the TSDF -> mesh path, each through the public Python entry points.

listed() gives the cases, draw() more of the same ranges, prepare() what a program has in hand before the call, run() one pass, work() the
bytes and operations a pass cannot do without, exact() the floating outputs in binary64 as plain torch evaluates them.

Volumes stand for what a fusion run leaves: spheres and boxes in a 3 m cube, free space at the upper bound of the truncated distance, voxels
behind the surfaces and out of every view unobserved (lower bound, weight 0), noise of a tenth of a voxel near the surface.  The stress volume
is a union of 200 spheres with three octaves of noise.  The shapes come from a case's "scene"; the seed gives every measured distance an error
of its own (a factor around 1, so that meshes of one case have one size), the weights, the frames and the poses.
"""
import math

import numpy as np
import torch

import marching_cube_gb300 as mcg
from marching_cube_gb300 import synthetic

EXTENT = 3.0          # metres, side of the fused cube
TRUNC_VOXELS = 5.12   # 0.03 m at 512 voxels
MAX_TSDF = 32766

# The marching-cubes case table: for each of the 256 sign patterns its triangles, three edges each, one hexadecimal digit an edge.
_TABLE = (
    "- 083 019 183981 12a 08312a 92a029 2832a8a98 3b2 0b28b0 19023b 1b219b98b 3a1ba3 0a108a8ba 3903b9ba9 98aa8b "
    "478 430734 019847 419471731 12a847 34730412a 92a902847 2a9297273794 8473b2 b47b24204 90184723b 47b94b9b2921 "
    "3a13ba784 1ba14b1047b4 47890b9bab03 47b4b99ba 954 954083 054150 854835315 12a954 30812a495 52a542402 "
    "2a5325354348 95423b 0b208b495 05401523b 21525828b485 a3ba13954 4950818a18ba 54050b5bab03 54858aa8b 978579 "
    "930953573 078017157 153357 978957a12 a12950530573 802825857a52 2a5253357 7957893b2 95797292027b 23b018178157 "
    "b21b17715 958857a13a3b 5705097b010aba0 ba0b03a50807570 ba57b5 a65 0835a6 9015a6 1831985a6 165261 165126308 "
    "965906026 598582526328 23ba65 b08b20a65 01923b5a6 5a61929b298b 63b653513 08b0b50515b6 3b6036065059 65969bb98 "
    "5a6478 43047365a 1905a6847 a65197173794 612651478 125526304347 847905065026 739794329596269 3b2784a65 "
    "5a647242027b 01947823b5a6 9219b294b7b45a6 8473b53515b6 51b5b610b7b404b 059065036b63847 65969b4797b9 a4964a "
    "4a649a083 a01a60640 83181686461a 149124264 308129249264 024426 832824426 a49a64b23 08228b49a4a6 3b201606461a "
    "64161a48121b8b1 964936913b63 8b1810b61914641 3b6360064 648b68 7a678a89a 0730a709a67a a671a7178180 a67a71173 "
    "126168189867 269291679093739 780706602 732672 23ba68a89867 20727b09767a9a7 1801781a767a23b b21b17a61671 "
    "896867916b63136 091b67 7807063b0b60 7b6 76b 308b76 019b76 819831b76 a126b7 12a3086b7 2902a96b7 6b72a3a83a98 "
    "723627 708760620 276237019 162186198876 a76a17137 a7617a187108 03707a0a96a7 76a7a88a9 684b86 36b306046 "
    "86b846901 946963931b36 6846b82a1 12a30b06b046 4b846b0292a9 a93a32943b36463 823842462 042462 190234246438 "
    "194142246 8138618466a1 a10a06604 4634386a3039a93 a946a4 49576b 083495b76 50154076b b76834354315 954a1276b "
    "6b712a083495 76b54a42a402 348354325a52b76 723762549 954086062687 362376150540 628687218485158 954a16176137 "
    "16a176107870954 40a4a503a6a737a 76a7a854a48a 6956b9b89 36b063056095 0b805b01556b 6b3635531 12a95b9b8b56 "
    "0b306b09656912a b85b56805a52025 6b36352a3a53 589528562382 956960062 158180568382628 156216 13616a386569896 "
    "a10a06950560 03856a a56 b5a75b b5ab75830 5b75ab190 a75ab7981831 b12b71751 08312717572b 9759279022b7 "
    "75272b592328982 25a235375 820852875a25 9015a35373a2 982921872a25752 135375 087071175 903935537 987597 "
    "5845a8ab8 5045b05abb30 01984a8aba45 ab4a45b34941314 2512852b8458 04b0b345b2b151b 0250592b5458b85 9452b3 "
    "25a352345384 5a2524420 3a235a385458019 5a2524192942 845853351 045105 845853905035 945 4b749b9ab 0834979b79ab "
    "1ab1b414074b 3143481a474bab4 4b79b492b912 9749b791b2b1083 b74b42240 b74b42834324 29a279237749 "
    "9a7974a27870207 37a3a274a1a040a 1a2874 491417713 491417081871 403743 487 9a8ab8 30939bb9a 01a0a88ab 31ab3a "
    "12b1b99b8 30939b1292b9 02b80b 32b 23828aa89 9a2092 23828a0181a8 1a2 138918 091 038 - "
).split()
_CORNER = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_EDGE = ((0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7))


# ---------------------------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest extraction a program asks for, with everything the reference's run() writes: latency and launches count
        {"name": "run_128", "kind": "run", "scene": 1, "nx": 128, "ny": 128, "nz": 128},
        # the mesh of a fused 512^3 volume, the size the project is quoted on: triangle soup and normals
        {"name": "extract_512", "kind": "extract", "scene": 1, "nx": 512, "ny": 512, "nz": 512},
        # the largest volume: 1024^3 with the surface nearly everywhere, 18 M triangles
        {"name": "extract_1024", "kind": "stress", "scene": 1, "n": 1024},
        # many small objects at once, uneven and mostly odd sizes, into an arena a server keeps
        {"name": "batch_64", "kind": "batch", "scene": 1, "volumes": 64, "lo": 32, "hi": 256},
        # shared-vertex mesh of a volume with odd sides
        {"name": "indexed_odd", "kind": "indexed", "scene": 1, "nx": 385, "ny": 257, "nz": 321, "float": False},
        # optimisation of a float volume with odd sides: mesh positions and their gradient
        {"name": "mesh_grad_odd", "kind": "mesh_grad", "scene": 1, "nx": 201, "ny": 175, "nz": 233},
        # one live depth frame into a 512^3 volume: maps, then integration weighted by the normals
        {"name": "fuse_512", "kind": "fuse", "n": 512, "w": 640, "h": 480, "normals": True, "dynamic": False},
        # a training step through the whole differentiable path: ten frames, 256^3, mesh positions, gradient at every depth pixel
        {"name": "train_256", "kind": "train", "n": 256, "frames": 10, "w": 320, "h": 240},
        # the model's depth and normals as the camera sees them, for tracking the next frame
        {"name": "raycast_512", "kind": "raycast", "n": 512, "w": 640, "h": 480},
        # tracking one frame against the frame before: depth pyramid, maps, three levels of ICP
        {"name": "track_640", "kind": "track", "w": 640, "h": 480, "bilinear": False},
        # saving a fused volume and reading it back: run-length image to the host, image to the device
        {"name": "rle_512", "kind": "rle", "scene": 1, "nx": 512, "ny": 512, "nz": 512, "lossless": False},
        # a text dump of a volume to a mesh file, end to end: load, extract, binary PLY
        {"name": "text_to_ply_192", "kind": "text", "scene": 1, "n": 192},
    ]


def _size(rng, lo, hi):
    """A size, spread over the logarithm of its range; odd ones and multiples of 4 come alike often."""
    s = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, s if rng.random() < 0.5 else (s + 3) // 4 * 4))


def draw(rng):
    kind = rng.choice(("run", "extract", "stress", "batch", "indexed", "mesh_grad", "fuse", "train", "raycast", "track", "rle", "text"))
    scene = rng.randrange(1000)
    w = rng.choice((160, 212, 320, 424, 512, 640))
    h = w * 3 // 4
    if kind == "run":
        return {"kind": kind, "scene": scene, "nx": _size(rng, 48, 384), "ny": _size(rng, 48, 384), "nz": _size(rng, 48, 384)}
    if kind == "extract":
        return {"kind": kind, "scene": scene, "nx": _size(rng, 96, 768), "ny": _size(rng, 96, 768), "nz": _size(rng, 96, 768)}
    if kind == "stress":
        return {"kind": kind, "scene": scene, "n": _size(rng, 384, 1024)}
    if kind == "batch":
        lo = _size(rng, 16, 64)
        return {"kind": kind, "scene": scene, "volumes": _size(rng, 4, 64), "lo": lo, "hi": _size(rng, 2 * lo, 256)}
    if kind == "indexed":
        return {"kind": kind, "scene": scene, "nx": _size(rng, 64, 512), "ny": _size(rng, 64, 512), "nz": _size(rng, 64, 512), "float": rng.random() < 0.3}
    if kind == "mesh_grad":
        return {"kind": kind, "scene": scene, "nx": _size(rng, 64, 320), "ny": _size(rng, 64, 320), "nz": _size(rng, 64, 320)}
    if kind == "fuse":
        return {"kind": kind, "n": _size(rng, 96, 640), "w": w, "h": h, "normals": rng.random() < 0.7, "dynamic": rng.random() < 0.3}
    if kind == "train":
        return {"kind": kind, "n": _size(rng, 96, 288), "frames": rng.randint(3, 12), "w": w // 2, "h": h // 2}
    if kind == "raycast":
        return {"kind": kind, "n": _size(rng, 128, 640), "w": w, "h": h}
    if kind == "track":
        return {"kind": kind, "w": w, "h": h, "bilinear": rng.random() < 0.4}
    if kind == "rle":
        return {"kind": kind, "scene": scene, "nx": _size(rng, 96, 576), "ny": _size(rng, 96, 576), "nz": _size(rng, 96, 576), "lossless": rng.random() < 0.3}
    return {"kind": kind, "scene": scene, "n": _size(rng, 64, 208)}


# ---------------------------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------------------------
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _axes(nx, ny, nz, step, z0=0):
    a = lambda lo, hi: (torch.arange(lo, hi, device=_dev(), dtype=torch.float32) + 0.5) * step  # noqa: E731
    return a(0, nx)[None, None, :], a(0, ny)[None, :, None], a(z0, z0 + nz)[:, None, None]


def _measured(f, g):
    """Truncated distances (as a share of the bound) with an error of their own: the sign stays."""
    return (f * torch.randn(f.shape, generator=g, device=_dev()).mul_(0.1).add_(1.0).clamp_(0.5, 1.5)).clamp_(-1, 1)


def _stored(f, scale=32767):
    """As 16-bit integers: what is negative stays so."""
    t = torch.trunc(f * scale)
    return torch.where(f < 0, t.clamp(max=-1), t).to(torch.int16)


def _sphere(nx, ny, nz, scene, seed):
    """Analytic sphere, radius 0.31 of the smallest side, truncation 5 voxels, weights 1..128."""
    x, y, z = _axes(nx, ny, nz, 1.0)
    c = np.random.default_rng(scene).uniform(-0.5, 0.5, 3)
    sd = torch.sqrt((x - nx / 2 - c[0]) ** 2 + (y - ny / 2 - c[1]) ** 2 + (z - nz / 2 - c[2]) ** 2) - 0.3125 * min(nx, ny, nz)
    g = _gen(seed)
    t = _stored(_measured(sd / 5.0, g))
    w = torch.randint(1, 129, t.shape, generator=g, device=_dev(), dtype=torch.int16)
    return torch.stack([t, w], dim=-1)


def _fused(nx, ny, nz, shapes, seed, as_float=False):
    """What fusing a scene leaves: see the top of the file."""
    step = EXTENT / max(nx, ny, nz)
    trunc = TRUNC_VOXELS * step
    scene = synthetic.FusionScene(shapes)
    side = np.array([nx, ny, nz]) * step / EXTENT
    rough, g = _gen(shapes), _gen(seed)
    out = torch.empty((nz, ny, nx, 2), dtype=torch.float32 if as_float else torch.int16, device=_dev())
    slab = max(1, (1 << 25) // (nx * ny))
    for z0 in range(0, nz, slab):
        z1 = min(nz, z0 + slab)
        x, y, z = _axes(nx, ny, z1 - z0, step, z0)
        sd = torch.full((z1 - z0, ny, nx), 10.0, device=_dev())
        for c, r in zip(scene.sph_c * side, scene.sph_r * side.min()):
            d = (x - float(c[0])) ** 2 + (y - float(c[1])) ** 2
            torch.minimum(sd, (d + (z - float(c[2])) ** 2).sqrt_().sub_(float(r)), out=sd)
        for c, h in zip(scene.box_c * side, scene.box_h * side.min()):
            q = [(a - float(c[i])).abs() - float(h[i]) for i, a in enumerate((x, y, z))]
            away = (q[0].clamp(min=0) ** 2 + q[1].clamp(min=0) ** 2 + q[2].clamp(min=0) ** 2).sqrt_()
            torch.minimum(sd, away.add_(torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp_(max=0)), out=sd)
        sd += torch.randn(sd.shape, generator=rough, device=_dev()).mul_(0.1 * step)
        m = EXTENT / 2 * side
        seen = (x - float(m[0])) ** 2 + (y - float(m[1])) ** 2 + (z - float(m[2])) ** 2 < (1.75 * side.min()) ** 2
        seen = seen & (sd >= -trunc)
        f = _measured(sd / trunc, g)
        w = torch.randint(1, 60000, sd.shape, generator=g, device=_dev(), dtype=torch.int32)
        if as_float:
            out[z0:z1, ..., 0] = torch.where(seen, f, -1.0)
            out[z0:z1, ..., 1] = torch.where(seen, w.to(torch.float32) / 1200.0, 0.0)
        else:
            out[z0:z1, ..., 0] = torch.where(seen, _stored(f, MAX_TSDF), -MAX_TSDF)
            out[z0:z1, ..., 1] = torch.where(seen, torch.where(w >= 32768, w - 65536, w), 0).to(torch.int16)
    return out


def _stress(n, scene, seed):
    """Union of 200 spheres (radii 2 to 8 % of the side) plus three octaves of smooth noise, weights 1..128."""
    rng = np.random.default_rng(scene)
    c, r = rng.uniform(0.05, 0.95, (200, 3)) * n, rng.uniform(0.02, 0.08, 200) * n
    smooth, g = _gen(scene), _gen(seed)
    grids = [torch.randn((1, 1) + (n // p + 2,) * 3, generator=smooth, device=_dev()) for p in (32, 16, 8)]
    out = torch.empty((n, n, n, 2), dtype=torch.int16, device=_dev())
    slab = 32
    for z0 in range(0, n, slab):
        z1 = min(n, z0 + slab)
        x, y, z = _axes(n, n, z1 - z0, 1.0, z0)
        sd = torch.full((z1 - z0, n, n), 6.0, device=_dev())
        for k in np.flatnonzero((c[:, 2] + r + 6 >= z0) & (c[:, 2] - r - 6 <= z1)):
            d = (x - float(c[k, 0])) ** 2 + (y - float(c[k, 1])) ** 2
            torch.minimum(sd, (d + (z - float(c[k, 2])) ** 2).sqrt_().sub_(float(r[k])), out=sd)
        for grid, period, amp in zip(grids, (32, 16, 8), (0.115, 0.057, 0.029)):
            cells = grid[:, :, z0 // period:(z1 + period - 1) // period + 1]
            big = torch.nn.functional.interpolate(cells, size=(z1 - z0 + period, n, n), mode="trilinear", align_corners=True)
            sd += big[0, 0, :z1 - z0] * amp
        out[z0:z1, ..., 0] = _stored(_measured(sd / 5.0, g))
        out[z0:z1, ..., 1] = torch.randint(1, 129, sd.shape, generator=g, device=_dev(), dtype=torch.int16)
    return out


def _batch_sizes(case):
    rng = np.random.default_rng(case["scene"])
    return np.round(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), (case["volumes"], 3)))).astype(int).tolist()


def _objects(nx, ny, nz, scene, seed):
    """1 to 8 spheres and boxes, truncation 5 voxels, weights 1..128."""
    rng = np.random.default_rng(scene)
    x, y, z = _axes(nx, ny, nz, 1.0)
    side = np.array([nx, ny, nz])
    sd = torch.full((nz, ny, nx), 1e9, device=_dev())
    for _ in range(int(rng.integers(1, 9))):
        c = rng.uniform(0.2, 0.8, 3) * side
        if rng.random() < 0.5:
            d = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) - rng.uniform(0.1, 0.35) * side.min()
        else:
            h = rng.uniform(0.05, 0.3, 3) * side
            q = [(x - c[0]).abs() - h[0], (y - c[1]).abs() - h[1], (z - c[2]).abs() - h[2]]
            d = (q[0].clamp(min=0) ** 2 + q[1].clamp(min=0) ** 2 + q[2].clamp(min=0) ** 2).sqrt()
            d = d + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0)
        sd = torch.minimum(sd, d)
    g = _gen(seed)
    t = _stored(_measured(sd / 5.0, g))
    w = torch.randint(1, 129, t.shape, generator=g, device=_dev(), dtype=torch.int16)
    return torch.stack([t, w], dim=-1)


def _camera(w, h):
    f = 525.0 * w / 640.0
    return f, (w - 1) / 2.0, (h - 1) / 2.0


def _maps(depth, k0):
    """Depth pyramid of a frame and the vertex and normal map of every level, as the fusion loop builds them."""
    levels, d, k = [], depth, k0
    for i in range(3):
        if i:
            d, mask = mcg.pyramid_down(d, mcg.float_data_to_mask(d))
            d = mcg.float_mask_to_data(mask, d)
            k = mcg.intrinsic_pyramid_down(k)
        v = mcg.meter_to_vertex(d, k)
        levels.append((v, mcg.vertex_to_normal(v)))
    return levels


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "run":
        s["voxel"] = mcg.Voxel(_sphere(case["nx"], case["ny"], case["nz"], case["scene"], seed), 0.05, 0.05, 0.01)
        s["mc"] = mcg.MarchingCubes()
    elif kind == "extract":
        s["cell"] = EXTENT / max(case["nx"], case["ny"], case["nz"])
        s["volume"] = _fused(case["nx"], case["ny"], case["nz"], case["scene"], seed)
    elif kind == "stress":
        s["cell"] = 0.01
        s["volume"] = _stress(case["n"], case["scene"], seed)
    elif kind == "batch":
        s["volumes"] = [_objects(*d, case["scene"] * 1000 + i, seed * 1000 + i) for i, d in enumerate(_batch_sizes(case))]
        s["cells"] = [0.01] * len(s["volumes"])
        # the arena is sized from a first extraction, with room to spare
        caps = [m.num_vertices + m.num_vertices // 8 + 64 for m in mcg.extract_batched(s["volumes"], s["cells"], normals=False)]
        s["soup"] = torch.zeros((sum(caps), mcg.VERTEX_VOXEL_BYTES), dtype=torch.uint8, device=_dev())
        s["normals"] = torch.zeros((sum(caps), 3), dtype=torch.float32, device=_dev())
        s["caps"] = caps
        at = np.cumsum([0] + caps).tolist()
        s["outputs"] = [{"soup": s["soup"][a:b], "normals": s["normals"][a:b]} for a, b in zip(at, at[1:])]
    elif kind == "indexed":
        s["cell"] = EXTENT / max(case["nx"], case["ny"], case["nz"])
        s["volume"] = _fused(case["nx"], case["ny"], case["nz"], case["scene"], seed, case["float"])
    elif kind == "mesh_grad":
        s["cell"] = EXTENT / max(case["nx"], case["ny"], case["nz"])
        s["volume"] = _fused(case["nx"], case["ny"], case["nz"], case["scene"], seed, True).requires_grad_(True)
    elif kind == "fuse":
        n, w, h = case["n"], case["w"], case["h"]
        f, cx, cy = _camera(w, h)
        step = EXTENT / n
        scene = synthetic.FusionScene(seed)
        R, t = scene.pose(seed % 60, 60)
        s["depth"] = synthetic.mm_to_u16_bits(scene.depth_frame(R, t, w, h, f, f, cx, cy, seed=seed, device=_dev()))
        s["k"], s["e"] = mcg.intrinsic(f, f, cx, cy), mcg.extrinsic(R, t)
        s["voxel"] = mcg.Voxel(_fused(n, n, n, seed, seed), TRUNC_VOXELS * step, TRUNC_VOXELS * step, step)
    elif kind == "train":
        scene = synthetic.BlendedSpheres(seed)
        w, h = case["w"], case["h"]
        f = 262.5 * w / 320.0
        depth, poses = scene.frames(case["frames"], w=w, h=h, fx=f, fy=f, device=_dev())
        s["depth"] = depth.to(torch.float32).contiguous().requires_grad_(True)
        s["k"] = mcg.intrinsic(f, f, (w - 1) / 2.0, (h - 1) / 2.0)
        s["poses"] = torch.stack([mcg.extrinsic_tensor(R, t) for R, t in poses]).contiguous()
    elif kind == "raycast":
        n, w, h = case["n"], case["w"], case["h"]
        f, cx, cy = _camera(w, h)
        scene = synthetic.FusionScene(seed)
        R, t = scene.pose(seed % 60, 60)
        s["k"], s["e"] = mcg.intrinsic(f, f, cx, cy), mcg.extrinsic(R, t)
        s["voxel"] = mcg.Voxel(_fused(n, n, n, seed, seed), TRUNC_VOXELS * EXTENT / n, TRUNC_VOXELS * EXTENT / n, EXTENT / n)
    elif kind == "track":
        w, h = case["w"], case["h"]
        f, cx, cy = _camera(w, h)
        scene = synthetic.BlendedSpheres(seed)
        at = seed % 200
        frames = [scene.depth_frame(*scene.pose(at + i, 200), w=w, h=h, fx=f, fy=f, cx=cx, cy=cy, device=_dev()).float().contiguous()
                  for i in (0, 1)]
        s["k"] = mcg.intrinsic(f, f, cx, cy)
        s["before"], s["depth"] = _maps(frames[0], s["k"]), frames[1]
        s["start"] = mcg.extrinsic(np.eye(3), np.zeros(3))
        s["inlier"] = torch.zeros((h, w), dtype=torch.uint8, device=_dev())
    elif kind == "rle":
        step = EXTENT / max(case["nx"], case["ny"], case["nz"])
        s["voxel"] = mcg.Voxel(_fused(case["nx"], case["ny"], case["nz"], case["scene"], seed), TRUNC_VOXELS * step, TRUNC_VOXELS * step, step)
        # a buffer for the image that is kept from save to save: a record is at most 6 bytes a voxel, in earnest far less
        s["out"] = np.zeros((6 if case["lossless"] else 2) * case["nx"] * case["ny"] * case["nz"] + 4096 * case["nz"], np.uint8)
    else:
        n = case["n"]
        s["text"] = synthetic.text_dump(_fused(n, n, n, case["scene"], seed), mcg.TEXT_ORIGIN).cpu().numpy()
        s["mc"] = mcg.MarchingCubes()
    return s


# ---------------------------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        m = s["mc"].run(s["voxel"])
        return {"soup": m.soup, "normals": m.normals, "vi2vox": m.vi2vox, "ver_voxel": m.ver_voxel}
    if kind in ("extract", "stress"):
        m = mcg.extract(s["volume"], s["cell"])
        return {"soup": m.soup, "normals": m.normals}
    if kind == "batch":
        mcg.extract_batched_into(s["volumes"], s["cells"], s["outputs"], s["caps"])
        return {"soup": s["soup"], "normals": s["normals"]}
    if kind == "indexed":
        m = mcg.extract_indexed(s["volume"], s["cell"])
        return {"positions": m.positions, "normals": m.normals, "triangles": m.triangles}
    if kind == "mesh_grad":
        p = mcg.mesh_positions(s["volume"], s["cell"])
        # the gradient of half the squared distance to the middle of the cube
        g, = torch.autograd.grad(p, s["volume"], p.detach() - EXTENT / 2)
        return {"positions": p.detach(), "gradient": g}
    if kind == "fuse":
        meter, vertex, normal = mcg.depth_to_maps(s["depth"], s["k"], depth_max=4.0)
        mcg.volumetric_integration(s["voxel"], s["k"], s["e"], meter, normal if case["normals"] else None, case["dynamic"])
        return {"meter": meter, "vertex": vertex, "normal": normal, "volume": s["voxel"].data}
    if kind == "train":
        n = case["n"]
        volume = mcg.integrate_frames(s["depth"], s["poses"], (n, n, n), 4.0 / n, 4.0 / n, 1.0 / n, s["k"])
        p = mcg.mesh_positions(volume, 1.0 / n)
        loss = 0.5 * ((p - 0.5) ** 2).sum()
        g, = torch.autograd.grad(loss, s["depth"])
        return {"volume": volume.detach(), "loss": loss.detach(), "gradient": g}
    if kind == "raycast":
        depth, normal = mcg.raycast(s["voxel"], s["k"], s["e"], case["w"], case["h"])
        return {"depth": depth, "normal": normal}
    if kind == "track":
        now = _maps(s["depth"], s["k"])
        ok, pose, iterations = mcg.icp_pyramid(s["k"], s["start"], s["before"], now, bilinear=case["bilinear"], inlier=s["inlier"])
        return {"ok": ok, "iterations": list(iterations), "pose": np.array(list(pose.r) + list(pose.t), np.float32), "inlier": s["inlier"],
                "maps": now}
    if kind == "rle":
        image = mcg.rle_encode(s["voxel"], case["lossless"], out=s["out"])
        return {"image": s["out"], "bytes": len(image), "volume": mcg.rle_decode(image).data}
    voxel = mcg.load_text_records(s["text"], case["n"])
    return {"volume": voxel.data, "ply": np.frombuffer(mcg.mesh_ply(s["mc"].run(voxel)), np.uint8)}


# ---------------------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------------------------
def _triangles(case):
    """About how many triangles the case's surface has (from its area in voxel faces)."""
    kind = case["kind"]
    if kind == "stress":
        return 17 * case["n"] ** 2
    if kind == "batch":
        return sum(int(4.05 * (x * y * z) ** (2 / 3)) for x, y, z in _batch_sizes(case))
    if kind == "train":
        return int(2.5 * case["n"] ** 2)
    if kind == "text":
        return int(5.2 * case["n"] ** 2)
    face = min(case["nx"], case["ny"], case["nz"]) ** 2
    return int((3.7 if kind == "run" else 5.2) * face)


def work(case):
    kind = case["kind"]
    if "nx" in case:
        voxels = case["nx"] * case["ny"] * case["nz"]
    elif "n" in case:
        voxels = case["n"] ** 3
    pixels = case.get("w", 0) * case.get("h", 0)
    if kind == "run":  # the volume; soup, normals and voxels of the vertices; the cleared per-voxel map
        t = _triangles(case)
        return {"bytes": 4 * voxels + 3 * t * (28 + 12 + 12) + 2 * voxels, "flops": 3 * t * 90}
    if kind in ("extract", "stress"):
        t = _triangles(case)
        return {"bytes": 4 * voxels + 3 * t * (28 + 12), "flops": 3 * t * 90}
    if kind == "batch":
        t = _triangles(case)
        return {"bytes": 4 * sum(x * y * z for x, y, z in _batch_sizes(case)) + 3 * t * (28 + 12), "flops": 3 * t * 90}
    if kind == "indexed":  # half as many shared vertices as triangles
        t = _triangles(case)
        return {"bytes": (8 if case["float"] else 4) * voxels + t // 2 * 24 + 12 * t, "flops": t // 2 * 90}
    if kind == "mesh_grad":  # volume in, positions out, gradient of both channels out
        t = _triangles(case)
        return {"bytes": 8 * voxels + 3 * t * 12 + 8 * voxels, "flops": 3 * t * 60}
    if kind == "fuse":  # frame in, maps out, the voxels before and at the surface (1 %) read and written
        return {"bytes": pixels * (2 + 28) + 8 * voxels // 100, "flops": 40 * voxels // 100}
    if kind == "train":  # frames in, their gradients out, the volume and the positions out
        t = _triangles(case)
        return {"bytes": 8 * pixels * case["frames"] + 8 * voxels + 36 * t, "flops": 40 * voxels * case["frames"]}
    if kind == "raycast":  # the voxels around the surface that the rays meet, and the maps
        return {"bytes": pixels * 16 + 4 * 8 * case["n"] ** 2, "flops": pixels * 60 * 40}
    if kind == "track":  # the frame, both frames' maps on three levels, the inliers
        return {"bytes": pixels * 4 + pixels * 24 * 21 // 16 * 2 + pixels, "flops": pixels * 21 // 16 * 150 * 3}
    if kind == "rle":  # volume in, image out and in, volume out
        return {"bytes": 2 * 4 * voxels + 2 * voxels * (5 if case["lossless"] else 1) // 5, "flops": 0}
    return {"bytes": 20 * voxels + 4 * voxels + 3 * _triangles(case) * 28, "flops": 0}


# ---------------------------------------------------------------------------------------------------------------------------------------
# the floating outputs in binary64
# ---------------------------------------------------------------------------------------------------------------------------------------
def _soup(volume, cell, normals=False, grad=None):
    """Soup positions (n, 3) in the order of the library (bricks of 32 x 8 x 8 cubes in z, y, x order, cubes in z, y, x order inside), then
    the normals or the gradient of half the squared distance to `grad` with respect to the distances, each None where not asked for."""
    nz, ny, nx, _ = volume.shape
    dev, f64 = volume.device, torch.float64
    tri = torch.full((256, 16), 0, dtype=torch.int64)
    for i, row in enumerate(_TABLE):
        if row != "-":
            e = [int(c, 16) for c in row]
            e = [e[3 * (k // 3) + 2 - k % 3] for k in range(len(e))]  # written with the winding reversed
            tri[i, :len(e)] = torch.tensor(e)
    tri, count = tri.to(dev), torch.tensor([0 if r == "-" else len(r) for r in _TABLE], device=dev)
    corner, edge = torch.tensor(_CORNER, device=dev), torch.tensor(_EDGE, device=dev)
    flat = volume.reshape(-1, 2)

    def value(i):
        t = flat[i, 0].to(f64)
        return t if volume.dtype == torch.float32 else t / MAX_TSDF

    gf = torch.zeros(nx * ny * nz, dtype=f64, device=dev) if grad is not None else None
    places, vectors = [], []
    for z0 in range(0, nz - 1, 8):
        z1 = min(nz - 1, z0 + 8)
        part = volume[z0:z1 + 1]
        neg, live = part[..., 0] < 0, part[..., 1] != 0
        index = torch.zeros((z1 - z0, ny - 1, nx - 1), dtype=torch.int64, device=dev)
        valid = torch.ones(index.shape, dtype=torch.bool, device=dev)
        for k, (cx, cy, cz) in enumerate(_CORNER):
            at = (slice(cz, cz + z1 - z0), slice(cy, cy + ny - 1), slice(cx, cx + nx - 1))
            index |= neg[at].to(torch.int64) << k
            valid &= live[at]
        z, y, x = torch.nonzero(valid & (index != 0) & (index != 255), as_tuple=True)
        if not z.numel():
            continue
        brick = (y // 8) * ((nx + 31) // 32) + x // 32
        order = torch.argsort(((brick * 8 + z) * 8 + y % 8) * 32 + x % 32)
        z, y, x = z[order], y[order], x[order]
        case = index[z, y, x]
        n = count[case]
        which = torch.repeat_interleave(torch.arange(n.numel(), device=dev), n)
        slot = torch.arange(which.numel(), device=dev) - (torch.cumsum(n, 0) - n)[which]
        ends = edge[tri[case[which], slot]]
        base = torch.stack([x, y, z + z0], dim=1)[which]
        a, b = base + corner[ends[:, 0]], base + corner[ends[:, 1]]
        ia, ib = ((v[:, 2] * ny + v[:, 1]) * nx + v[:, 0] for v in (a, b))
        fa, fb = value(ia), value(ib)
        pa, pb = (a.to(f64) + 0.5) * cell, (b.to(f64) + 0.5) * cell
        p = pa + (-fa / (fb - fa + 1e-15))[:, None] * (pb - pa)
        places.append(p)
        if grad is not None:
            g = ((p - grad) * (pb - pa)).sum(dim=1) / (fb - fa + 1e-15) ** 2
            gf.index_add_(0, ia, -g * (fb + 1e-15))
            gf.index_add_(0, ib, g * fa)
        if normals:
            vectors.append(_normals(volume, flat, value, p / cell))
    none = torch.zeros((0, 3), dtype=f64, device=dev)
    return torch.cat(places) if places else none, (torch.cat(vectors) if vectors else none) if normals else None, gf


def _normals(volume, flat, value, p):
    """Unit gradient of the trilinear field at p (voxel units); zero where a sample is at a bound or outside the volume."""
    nz, ny, nx, _ = volume.shape
    i = p.floor().to(torch.int64)
    u, v, w = (p - i).unbind(1)
    at = ((i[:, 2] * ny + i[:, 1]) * nx + i[:, 0])[:, None] + torch.tensor(
        [c[0] + c[1] * nx + c[2] * nx * ny for c in _CORNER], device=p.device)
    good = ((at >= 0) & (at < nx * ny * nz)).all(dim=1)
    at = at.clamp(0, nx * ny * nz - 1)
    if volume.dtype == torch.int16:
        good &= (flat[at, 0].to(torch.int32).abs() != MAX_TSDF).all(dim=1)
    s = value(at)
    du, dv, dw = 1 - u, 1 - v, 1 - w
    g = torch.stack([((s[:, 1] - s[:, 0]) * dv + (s[:, 2] - s[:, 3]) * v) * dw + ((s[:, 5] - s[:, 4]) * dv + (s[:, 6] - s[:, 7]) * v) * w,
                     ((s[:, 3] - s[:, 0]) * du + (s[:, 2] - s[:, 1]) * u) * dw + ((s[:, 7] - s[:, 4]) * du + (s[:, 6] - s[:, 5]) * u) * w,
                     ((s[:, 4] - s[:, 0]) * du + (s[:, 5] - s[:, 1]) * u) * dv + ((s[:, 7] - s[:, 3]) * du + (s[:, 6] - s[:, 2]) * u) * v],
                    dim=1)
    norm = g.norm(dim=1, keepdim=True)
    return torch.where(good[:, None], torch.where(norm > 2.0 ** -23, g / norm, g), 0.0)


def _indexed(volume, cell):
    """Positions and normals of the shared vertices: one for each grid edge whose ends differ in sign and that a cube with no unobserved corner
    touches, in the order of the library (bricks, in a brick rows in z, y order, the axes, then x; an edge belongs to its lower voxel's brick)."""
    nz, ny, nx, _ = volume.shape
    flat, f64 = volume.reshape(-1, 2), torch.float64

    def value(i):
        t = flat[i, 0].to(f64)
        return t if volume.dtype == torch.float32 else t / MAX_TSDF

    neg, live = volume[..., 0] < 0, volume[..., 1] != 0
    cubes = torch.ones((nz - 1, ny - 1, nx - 1), dtype=torch.bool, device=volume.device)
    for cx, cy, cz in _CORNER:
        cubes &= live[cz:cz + nz - 1, cy:cy + ny - 1, cx:cx + nx - 1]
    found = []
    for axis in range(3):
        d = 2 - axis  # the tensor's dimension
        lo, hi = neg.narrow(d, 0, neg.shape[d] - 1), neg.narrow(d, 1, neg.shape[d] - 1)
        pad = [0 if k // 2 == axis else 1 for k in range(6)]
        around = torch.nn.functional.pad(cubes, pad)
        for e in range(3):
            if e != d:
                around = around.narrow(e, 0, around.shape[e] - 1) | around.narrow(e, 1, around.shape[e] - 1)
        z, y, x = torch.nonzero((lo != hi) & around, as_tuple=True)
        found.append(torch.stack([x, y, z, torch.full_like(x, axis)], dim=1))
    v = torch.cat(found)
    x, y, z, axis = v.unbind(1)
    bx, by, bz = ((c // b).clamp(max=(n - 1 + b - 1) // b - 1) for c, b, n in ((x, 32, nx), (y, 8, ny), (z, 8, nz)))
    brick = (bz * ((ny + 6) // 8) + by) * ((nx + 30) // 32) + bx
    order = torch.argsort((((brick * 9 + z - 8 * bz) * 9 + y - 8 * by) * 3 + axis) * 64 + x - 32 * bx)
    a, axis = v[order, :3], axis[order]
    step = torch.eye(3, dtype=torch.int64, device=v.device)[axis]
    fa, fb = (value((p[:, 2] * ny + p[:, 1]) * nx + p[:, 0]) for p in (a, a + step))
    p = (a.to(f64) + 0.5 + (-fa / (fb - fa + 1e-15))[:, None] * step) * cell
    return p, _normals(volume, flat, value, p / cell)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "run":
            n = _soup(_sphere(case["nx"], case["ny"], case["nz"], case["scene"], seed), 0.01, normals=True)[1]
            return {"soup": None, "normals": n, "vi2vox": None, "ver_voxel": None}
        if kind == "extract":
            step = EXTENT / max(case["nx"], case["ny"], case["nz"])
            return {"soup": None, "normals": _soup(_fused(case["nx"], case["ny"], case["nz"], case["scene"], seed), step, normals=True)[1]}
        if kind == "stress":
            return {"soup": None, "normals": _soup(_stress(case["n"], case["scene"], seed), 0.01, normals=True)[1]}
        if kind == "batch":
            rows = []
            for i, d in enumerate(_batch_sizes(case)):
                n = _soup(_objects(*d, case["scene"] * 1000 + i, seed * 1000 + i), 0.01, normals=True)[1]
                rows += [n, torch.zeros((n.shape[0] // 8 + 64, 3), dtype=n.dtype, device=n.device)]  # the arena's room to spare
            return {"soup": None, "normals": torch.cat(rows)}
        if kind == "indexed":
            volume = _fused(case["nx"], case["ny"], case["nz"], case["scene"], seed, case["float"])
            p, n = _indexed(volume, EXTENT / max(case["nx"], case["ny"], case["nz"]))
            return {"positions": p, "normals": n, "triangles": None}
        if kind == "mesh_grad":
            volume = _fused(case["nx"], case["ny"], case["nz"], case["scene"], seed, True)
            p, _, g = _soup(volume, EXTENT / max(case["nx"], case["ny"], case["nz"]), grad=EXTENT / 2)
            return {"positions": p, "gradient": torch.stack([g, torch.zeros_like(g)], dim=-1).reshape(volume.shape)}
        if kind == "fuse":
            w, h = case["w"], case["h"]
            f, cx, cy = _camera(w, h)
            scene = synthetic.FusionScene(seed)
            mm = scene.depth_frame(*scene.pose(seed % 60, 60), w, h, f, f, cx, cy, seed=seed, device=_dev())
            m = mm.to(torch.float64) / 1000.0
            m = torch.where(m > 4.0, 0.0, m)
            y, x = torch.meshgrid(torch.arange(h, device=_dev(), dtype=m.dtype), torch.arange(w, device=_dev(), dtype=m.dtype), indexing="ij")
            v = torch.stack([(x - cx) / f * m, (y - cy) / f * m, m], dim=-1)
            n = torch.zeros_like(v)
            c, right, down = v[:-1, :-1], v[:-1, 1:], v[1:, :-1]
            k = torch.linalg.cross(right - c, c - down)
            k = k / k.norm(dim=-1, keepdim=True).clamp(min=1e-300)
            n[:-1, :-1] = torch.where(((c[..., 2] != 0) & (right[..., 2] != 0) & (down[..., 2] != 0))[..., None], k, 0.0)
            return {"meter": m, "vertex": v, "normal": n, "volume": None}
    # A pose that an iteration stops at, a march's stops and a gradient through rounded pixel choices are what binary32 makes them; the
    # codecs and the text are whole numbers.
    return None
