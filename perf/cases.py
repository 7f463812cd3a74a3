"""The work that users of this framework have it do, as cases for timing.

Each case is one call path of the public API over the sizes, options and data that a
viewer, an offline renderer, a render server or a tool brings to it. Meshes are the two
constructions of the framework's own workloads (a bumpy icosphere and a displaced torus),
made on the GPU from the seed; cameras look at the mesh from a seeded direction.

G-buffers, images and hit records come back as the 32-bit words that the framework
writes: they are records of bytes whose results are fixed bit for bit.
"""
import functools
import math

import numpy as np
import torch

from j3d_gb300 import Canvas, Context, Matcap, Mesh, Scene, camera_for_vfov, settings, workloads
from j3d_gb300.learned import Learned
from j3d_gb300.scene import (Batch, Geometry, PointCloud, SceneObject, find_closest, mesh_from_geometry, render_batch,
                             voxelize)

BATCH_SIZES = [(256, 256), (512, 512), (768, 512), (1024, 1024)]
HIDDEN, CLASSES, FEATURES = 128, 4096, 256
ACTIVE = 2048  # classes whose logits count in the gradient case; the rest are switched off by their bias


def listed():
    return [
        # the smallest frame of the batched workload's sizes, rendered on its own: a thumbnail, or a viewer window
        # of a small model, where the launch and the slowest rays count
        frame_case("frame_small", "sphere", 81_920, 256, 256, shadow=True),
        # the headline workload: a 28M-triangle scan on a full-HD canvas with shadows
        frame_case("frame_large", "torus", 28_090_000, 1920, 1080, shadow=True),
        # the viewer with its default settings (edges on, shadows off) on a scene of several coloured objects,
        # in a window of odd size
        frame_case("frame_viewer", "torus", 100_352, 1279, 717, objects=24, mode="edges", colors=True),
        # opening a small model: the BVH build and the first frame
        open_case("open_small", "sphere", 81_920, 512, 384),
        # opening a 28M-triangle scan whose arrays are in hand
        open_case("open_large", "torus", 28_090_000, 1280, 720),
        # opening a mesh file that is in memory: decode, build, first frame
        open_case("open_ply", "torus", 2_000_000, 1024, 768, source="ply"),
        # a batch of ray queries (ambient occlusion, picking, collision): incoherent closest hits
        dict(name="rays", kind="rays", shape="torus", tris=2_000_000, rays=1_000_003, any=False, objects=1),
        # what the render server does with the requests that wait: many meshes, cameras and resolutions at once
        dict(name="batch", kind="batch", meshes=8, cameras=3, t_min=10_000, t_max=2_000_000, shadow=True, graph=False),
        # the voxel grid that the exporter writes
        dict(name="voxels", kind="voxels", shape="torus", tris=500_000, max_dim=256, colors=True),
        # a scanned point cloud drawn over a frame
        dict(name="points", kind="points", points=14_045_000, w=1920, h=1080, colors=True),
        # closest hits of a camera's rays through a trained network (inference)
        dict(name="learned_hits", kind="learned", tris=500_000, w=1280, h=720),
        # one training step's forward and backward passes
        dict(name="learned_grad", kind="grad", tris=500_000, batch=16_384),
    ]


def frame_case(name, shape, tris, w, h, shadow=False, objects=1, mode="plain", colors=False):
    c = dict(kind="frame", shape=shape, tris=tris, w=w, h=h, shadow=shadow, objects=objects, mode=mode, colors=colors)
    return dict(c, name=name) if name else c


def open_case(name, shape, tris, w, h, source="arrays", width=4, builder="ploc"):
    c = dict(kind="open", shape=shape, tris=tris, w=w, h=h, source=source, width=width, builder=builder)
    return dict(c, name=name) if name else c


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo, hi):
        w = log(lo, hi)
        return w, max(16, int(w * rng.uniform(0.5, 1.0)))

    kind = rng.choice(["frame", "frame", "open", "open", "rays", "batch", "voxels", "points", "learned", "grad"])
    if kind == "frame":
        objects = rng.choice([1, 1, log(2, 60)])
        mode = rng.choice(["plain", "plain", "edges", "wireframe", "one_bit"])
        tris = log(5_000, 28_000_000) if objects == 1 else log(5_000, 200_000)
        return frame_case(None, "torus", tris, *size(200, 1920), shadow=rng.random() < 0.6, objects=objects, mode=mode,
                          colors=rng.random() < 0.3 and tris < 3_000_000)
    if kind == "open":
        source = rng.choice(["arrays", "arrays", "ply", "stl"])
        width, builder = rng.choice([(4, "ploc"), (4, "ploc"), (4, "lbvh"), (2, "ploc"), (8, "ploc")])
        tris = log(5_000, 20_000_000) if source == "arrays" else log(5_000, 2_000_000)
        return open_case(None, "torus", tris, *size(200, 1280), source=source, width=width, builder=builder)
    if kind == "rays":
        return dict(kind="rays", shape="torus", tris=log(5_000, 8_000_000), rays=log(100, 4_000_000),
                    any=rng.random() < 0.4, objects=rng.choice([1, 1, log(2, 60)]))
    if kind == "batch":
        return dict(kind="batch", meshes=rng.randint(2, 10), cameras=rng.randint(1, 3), t_min=10_000,
                    t_max=log(50_000, 2_000_000), shadow=rng.random() < 0.7, graph=rng.random() < 0.5)
    if kind == "voxels":
        return dict(kind="voxels", shape="torus", tris=log(5_000, 2_000_000), max_dim=log(32, 512),
                    colors=rng.random() < 0.5)
    if kind == "points":
        w, h = size(200, 1920)
        return dict(kind="points", points=log(10_000, 14_000_000), w=w, h=h, colors=rng.random() < 0.6)
    if kind == "learned":
        w, h = size(200, 1280)
        return dict(kind="learned", tris=log(100_000, 2_000_000), w=w, h=h)
    return dict(kind="grad", tris=500_000, batch=128 * rng.randint(2, 128))


# --------------------------------------------------------------------------- inputs

_context = None


def context():
    """One context for the program, as its users keep one."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def ready(*tensors):
    """The tensors once torch has written them: the library works on a stream of its own."""
    torch.cuda.synchronize()
    return tensors if len(tensors) > 1 else tensors[0]


def torus(tris, seed):
    """Displaced torus on the GPU, about `tris` triangles: R = 1, r = 0.35 plus 0.02 times 16 seeded sinusoids."""
    nu, nv = workloads.torus_grid_for(tris)
    r = np.random.RandomState(seed)
    amp, phase = r.uniform(0, 1, 16), r.uniform(0, 2 * np.pi, 16)
    mu, mv = r.randint(1, 25, 16), r.randint(1, 13, 16)
    i = torch.arange(nu, device="cuda", dtype=torch.float64)[:, None] * (2 * math.pi / nu)
    j = torch.arange(nv, device="cuda", dtype=torch.float64)[None, :] * (2 * math.pi / nv)
    rad = torch.full((nu, nv), 0.35, device="cuda", dtype=torch.float64)
    for a, p, m, n in zip(amp, phase, mu, mv):
        rad += 0.02 * float(a) * torch.sin(int(m) * i + int(n) * j + float(p))
    ring = 1.0 + rad * torch.cos(j)
    V = torch.stack([ring * torch.cos(i), rad * torch.sin(j), ring * torch.sin(i)], -1).reshape(-1, 3).float()
    a = torch.arange(nu, device="cuda")[:, None]
    b = torch.arange(nv, device="cuda")[None, :]
    a1, b1 = (a + 1) % nu, (b + 1) % nv
    p00, p10, p01, p11 = a * nv + b, a1 * nv + b, a * nv + b1, a1 * nv + b1
    T = torch.stack([p00, p10, p11, p00, p11, p01], -1).reshape(-1, 3).int()
    return ready(V.contiguous(), T.contiguous())


@functools.lru_cache(maxsize=None)
def unit_icosphere(level):
    t = (1 + 5 ** 0.5) / 2
    V = np.array([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t], [0, 1, -t],
                  [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]], np.float64)
    T = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                  [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5], [2, 4, 11],
                  [6, 2, 10], [8, 6, 7], [9, 8, 1]], np.int64)
    for _ in range(level):
        e = np.sort(np.concatenate([T[:, [0, 1]], T[:, [1, 2]], T[:, [2, 0]]]), axis=1)
        u, inv = np.unique(e[:, 0] * len(V) + e[:, 1], return_inverse=True)
        mid = (V[u // len(V)] + V[u % len(V)]) / 2
        ab, bc, ca = (inv.reshape(-1) + len(V)).reshape(3, -1)
        a, b, c = T.T
        T = np.concatenate([np.stack(x, 1) for x in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))])
        V = np.concatenate([V, mid])
    return V / np.linalg.norm(V, axis=1, keepdims=True), T.astype(np.int32)


def sphere(tris, seed):
    """Icosphere with its radius moved by 0.05 times 8 seeded sinusoids of the direction."""
    D, T = unit_icosphere(int(round(math.log(tris / 20, 4))))
    r = np.random.RandomState(seed)
    rad = np.ones(len(D))
    for _ in range(8):
        u = r.normal(size=3)
        rad += 0.05 * r.uniform(0, 1) * np.sin(r.uniform(2, 12) * (D @ (u / np.linalg.norm(u))) + r.uniform(0, 2 * np.pi))
    V = torch.from_numpy((D * rad[:, None]).astype(np.float32)).cuda()
    return ready(V, torch.from_numpy(T).cuda())


def surface(case, seed):
    return sphere(case["tris"], seed) if case.get("shape") == "sphere" else torus(case["tris"], seed)


def colors_of(V):
    return ready((0.5 + 0.5 * torch.sin(7 * V)).contiguous())


def rigid(rng, spread):
    """A random rotation and a translation within the spread, column-major."""
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    M = np.eye(4)
    M[:3, :3] = [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                 [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                 [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]
    M[:3, 3] = rng.uniform(-spread, spread, 3)
    return M.T.reshape(16).astype(np.float32)


def objects_of(case, seed):
    """The case's objects: one mesh as it is, or instances of up to four meshes under rigid transforms. Returns
    [(mesh, cs)] and the radius range of cameras that see them all."""
    ctx, n = context(), case["objects"]
    if n == 1:
        V, T = surface(case, seed)
        m = Mesh(ctx, V, T)
        if case.get("colors"):
            m.set_vertex_colors(colors_of(V))
        return [(m, None)], (2.5, 4.0)
    rng = np.random.RandomState(seed + 17)
    meshes = []
    for k in range(min(4, n)):
        V, T = torus(max(200, case["tris"] >> k), seed + k)
        m = Mesh(ctx, V, T)
        if case.get("colors"):
            m.set_vertex_colors(colors_of(V))
        meshes.append(m)
    spread = 1.5 * n ** (1 / 3)
    return [(meshes[k % len(meshes)], rigid(rng, spread)) for k in range(n)], (2.2 * spread, 3.0 * spread)


class DeviceArray:
    """A device address as an array that torch can wrap without a copy."""

    def __init__(self, address, shape):
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": "<i4", "version": 3}


def canvas_words(canvas):
    """The canvas's G-buffer and image on the device, as 32-bit words."""
    pixels, image, _ = canvas.device_buffers()
    h, w = canvas.height, canvas.width
    return {"pixels": torch.as_tensor(DeviceArray(pixels, (h, w, 8)), device="cuda"),
            "image": torch.as_tensor(DeviceArray(image, (h, w)), device="cuda")}


def new_canvas(w, h, mode="plain", shadow=False):
    cv = Canvas(context(), w, h)
    cv.set_camera(camera_for_vfov(60.0))
    cv.set_background_color()
    cv.update_settings(settings(shadow=shadow, edges=mode == "edges", wireframe=mode == "wireframe",
                                one_bit=mode == "one_bit"))
    return cv


def new_scene(objects, pose):
    sc = Scene()
    for k, (mesh, cs) in enumerate(objects):
        sc.add_object(mesh, cs, 1 + k)
    sc.prepare_scene()
    sc.unzoom()
    sc.set_pose(pose)
    return sc


def pose_of(seed, radii):
    return workloads.cameras(1, seed + 1000, *radii)[0]


def ply_bytes(V, T):
    head = ("ply\nformat binary_little_endian 1.0\nelement vertex %d\nproperty float x\nproperty float y\nproperty float z\n"
            "element face %d\nproperty list uchar int vertex_indices\nend_header\n" % (len(V), len(T))).encode()
    faces = torch.empty((len(T), 13), dtype=torch.uint8, device=T.device)
    faces[:, 0] = 3
    faces[:, 1:] = T.contiguous().view(torch.uint8).reshape(-1, 12)
    return head + V.cpu().numpy().tobytes() + faces.cpu().numpy().tobytes()


def stl_bytes(V, T):
    recs = torch.zeros((len(T), 50), dtype=torch.uint8, device=T.device)
    recs[:, 12:48] = V[T.long()].reshape(-1, 9).contiguous().view(torch.uint8).reshape(-1, 36)
    return b"\0" * 80 + np.uint32(len(T)).tobytes() + recs.cpu().numpy().tobytes()


def ray_records(origin, direction, near=0.0):
    n = len(origin)
    r = torch.zeros((n, 10), device="cuda")
    r[:, 0:3], r[:, 3] = origin, 1.0
    r[:, 4:7] = direction
    r[:, 8], r[:, 9] = near, torch.finfo(torch.float32).max
    return r


def camera_rays(w, h, pose):
    """Rays through the pixel centres of a 60 degree camera."""
    M = torch.from_numpy(np.asarray(pose, np.float32).reshape(4, 4)).cuda()  # rows: the columns of the pose
    f = math.tan(math.radians(30))
    x = ((torch.arange(w, device="cuda") + 0.5) / w * 2 - 1) * f * w / h
    y = ((torch.arange(h, device="cuda") + 0.5) / h * 2 - 1) * f
    d = x[None, :, None] * M[0, :3] + y[:, None, None] * M[1, :3] - M[2, :3]
    return ray_records(M[3, :3].expand(w * h, 3), d.reshape(-1, 3))


# --------------------------------------------------------------------------- prepare

def prepare(case, seed):
    st = {"kind": case["kind"]}
    PREPARE[case["kind"]](case, int(seed) & 0x3FFFFFFF, st)
    torch.cuda.synchronize()
    return st


def prepare_frame(case, seed, st):
    objects, radii = objects_of(case, seed)
    st["scene"] = new_scene(objects, pose_of(seed, radii))
    st["canvas"] = new_canvas(case["w"], case["h"], case["mode"], case["shadow"])
    st["matcap"] = Matcap.make(context(), 0)
    st["out"] = canvas_words(st["canvas"])


def prepare_open(case, seed, st):
    V, T = surface(case, seed)
    if case["source"] == "arrays":
        st["V"], st["T"] = V, T
    else:
        st["data"] = ply_bytes(V, T) if case["source"] == "ply" else stl_bytes(V, T)
    st.update(source=case["source"], width=case["width"], builder=case["builder"], pose=pose_of(seed, (2.5, 4.0)))
    st["canvas"] = new_canvas(case["w"], case["h"])
    st["matcap"] = Matcap.make(context(), 0)
    st["out"] = canvas_words(st["canvas"])


def prepare_rays(case, seed, st):
    objects, radii = objects_of(case, seed)
    st["objects"] = [SceneObject(m, cs, 1 + k) for k, (m, cs) in enumerate(objects)]
    n, g = case["rays"], torch.Generator(device="cuda").manual_seed(seed)
    o = torch.randn((n, 3), device="cuda", generator=g)
    o = o / o.norm(dim=1, keepdim=True) * radii[1]
    to = (torch.rand((n, 3), device="cuda", generator=g) - 0.5) * (2.6 if case["objects"] == 1 else radii[1])
    st["rays"] = ray_records(o, to - o)
    st["hits"] = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
    st["any"] = case["any"]


def batch_frames(case):
    """(mesh index, w, h) of every frame: the batched workload's sizes in turn, every fifth one odd."""
    n = case["meshes"] * case["cameras"]
    sizes = [BATCH_SIZES[(3 * i + i // 4) % 4] for i in range(n)]
    return [(i % case["meshes"], w - 3 * (i % 5 == 4), h - 5 * (i % 5 == 4)) for i, (w, h) in enumerate(sizes)]


def batch_tris(case):
    m = case["meshes"]
    return [int(case["t_min"] * (case["t_max"] / case["t_min"]) ** (k / max(1, m - 1))) for k in range(m)]


def prepare_batch(case, seed, st):
    ctx = context()
    meshes = [Mesh(ctx, *torus(t, seed + k)) for k, t in enumerate(batch_tris(case))]
    st["matcap"] = Matcap.make(ctx, 0)
    st["frames"] = [(new_canvas(w, h, shadow=case["shadow"]),
                     new_scene([(meshes[k], None)], pose_of(seed + 31 * i, (2.5, 4.0))), st["matcap"])
                    for i, (k, w, h) in enumerate(batch_frames(case))]
    st["graph"] = Batch(ctx, st["frames"]) if case["graph"] else None
    st["out"] = [canvas_words(cv) for cv, _, _ in st["frames"]]


def prepare_voxels(case, seed, st):
    V, T = surface(case, seed)
    lo, hi = V.amin(0).double(), V.amax(0).double()
    # every seed's mesh in one box, so that its grid has one shape
    V = ready(((V - lo) / (hi - lo) * torch.tensor([2.7, 0.757, 2.7], device="cuda", dtype=torch.float64)).float())
    st["mesh"] = Mesh(context(), V, T)
    if case["colors"]:
        st["mesh"].set_vertex_colors(colors_of(V))
    st["max_dim"] = case["max_dim"]


def prepare_points(case, seed, st):
    ctx, g = context(), torch.Generator(device="cuda").manual_seed(seed)
    a, b = (torch.rand((2, case["points"]), device="cuda", generator=g) * (2 * math.pi)).unbind(0)
    r = 0.4 + 0.02 * torch.randn(case["points"], device="cuda", generator=g)
    ring = 1 + r * torch.cos(b)
    P = torch.stack([ring * torch.cos(a), r * torch.sin(b), ring * torch.sin(a)], -1).contiguous()
    C = torch.randint(0, 1 << 24, (case["points"],), device="cuda", generator=g, dtype=torch.int32) if case["colors"] else None
    torch.cuda.synchronize()
    st["scene"] = new_scene([(Mesh(ctx, *torus(100_000, seed)), None)], pose_of(seed, (2.5, 4.0)))
    st["scene"].add_pointcloud(PointCloud(ctx, P, C))
    st["canvas"] = new_canvas(case["w"], case["h"])
    st["matcap"] = Matcap.make(ctx, 0)
    st["out"] = canvas_words(st["canvas"])


def prepare_learned(case, seed, st):
    ctx = context()
    st["mesh"] = Mesh(ctx, *torus(case["tris"], seed))
    st["net"] = Learned(ctx, st["mesh"], seed=seed)
    st["net"].train(262_144)
    st["rays"] = camera_rays(case["w"], case["h"], pose_of(seed, (2.5, 4.0)))
    st["hits"] = torch.zeros((len(st["rays"]), 6), dtype=torch.int32, device="cuda")


def gradient_inputs(case, seed):
    """Parameters (scaled normal weights, small biases, the classes past ACTIVE switched off by their bias),
    features and labels of a training batch."""
    r = np.random.RandomState(seed)
    parts, n_in = [], FEATURES
    for k in range(5):
        n_out = HIDDEN if k < 4 else CLASSES
        parts.append(r.standard_normal((n_in, n_out)).astype(np.float32).ravel() * np.float32((2 / n_in) ** 0.5))
        bias = r.standard_normal(n_out).astype(np.float32) * np.float32(0.1)
        if k == 4:
            bias[ACTIVE:] = -1e4
        parts.append(bias)
        n_in = n_out
    X = np.zeros((case["batch"], FEATURES), np.float32)
    X[:, :192] = r.uniform(-1, 1, (case["batch"], 192)).astype(np.float32)
    y = r.randint(0, ACTIVE, case["batch"]).astype(np.int32)
    y[r.uniform(size=case["batch"]) < 0.4] = -1  # rays that miss
    return np.concatenate(parts), X, y


def prepare_grad(case, seed, st):
    ctx = context()
    st["mesh"] = Mesh(ctx, *torus(case["tris"], seed))
    st["net"] = Learned(ctx, st["mesh"], seed=seed)
    if st["net"].n_clusters < ACTIVE:
        raise RuntimeError("the mesh has too few clusters")
    params, st["X"], st["y"] = gradient_inputs(case, seed)
    st["net"].set_params(params)


PREPARE = {"frame": prepare_frame, "open": prepare_open, "rays": prepare_rays, "batch": prepare_batch,
           "voxels": prepare_voxels, "points": prepare_points, "learned": prepare_learned, "grad": prepare_grad}


# --------------------------------------------------------------------------- run

def run(st):
    kind = st["kind"]
    if kind == "frame":
        st["canvas"].render_frame(st["scene"], st["matcap"])
        return st["out"]
    if kind == "open":
        if st["source"] == "arrays":
            mesh = Mesh(context(), st["V"], st["T"], build=st["builder"], width=st["width"])
        else:
            g = Geometry.read_memory(context(), st["data"], st["source"])
            mesh = mesh_from_geometry(context(), g, build=st["builder"], width=st["width"])
            g.close()
        st["scene"] = new_scene([(mesh, None)], st["pose"])  # the one of an earlier pass goes away
        st["canvas"].render_frame(st["scene"], st["matcap"])
        return st["out"]
    if kind == "rays":
        find_closest(context(), st["objects"], st["rays"], st["hits"], any_hit=st["any"])
        # an occlusion query answers whether something was hit; which triangle it met first is not part of the answer
        return st["hits"][:, 0] if st["any"] else st["hits"]
    if kind == "batch":
        if st["graph"]:
            st["graph"].launch()
        else:
            render_batch(context(), st["frames"])
        return st["out"]
    if kind == "voxels":
        return voxelize(context(), st["mesh"], st["max_dim"])
    if kind == "points":
        st["canvas"].render_frame(st["scene"], st["matcap"])
        st["canvas"].render_pointclouds(st["scene"])
        return st["out"]
    if kind == "learned":
        return st["net"].find_closest(st["rays"], st["hits"])
    loss, grads = st["net"].loss_grad(st["X"], st["y"])
    return {"loss": loss, "grads": grads}


# --------------------------------------------------------------------------- work

def ray_flops(tris):
    """A ray's way through a 4-wide tree: a node visit a level (four boxes of 12 operations) and two triangle tests."""
    return 48 * math.log(max(tris, 4), 4) + 2 * 60


def frame_work(pixels, tris, shadow):
    """The triangles (36 bytes) that the pixels' rays can meet, the background, the records and the image."""
    rays = pixels * (1.5 if shadow else 1)
    return pixels * (32 + 4 + 4) + 36 * min(tris, rays), rays * ray_flops(tris)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        b, f = frame_work(case["w"] * case["h"], case["tris"], case["shadow"])
    elif kind == "open":
        # vertices and indices in; nodes (about a fifth of a 128-byte node a triangle), leaf triangles and normals out
        t = case["tris"]
        b, f = frame_work(case["w"] * case["h"], t, False)
        file = {"arrays": 0, "ply": 19, "stl": 50}[case["source"]]
        b, f = b + t * (18 + file + 28 + 48 + 16), f + t * 100.0
    elif kind == "rays":
        b, f = case["rays"] * (40 + 24) + 36 * min(case["tris"], case["rays"]), case["rays"] * ray_flops(case["tris"])
    elif kind == "batch":
        tris = batch_tris(case)
        each = [frame_work(w * h, tris[k], case["shadow"]) for k, w, h in batch_frames(case)]
        b, f = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "voxels":
        d = case["max_dim"]
        rays = d * d + 2 * d * d * 0.28
        b, f = 0.28 * d ** 3 + 36 * min(case["tris"], 3 * rays), rays * ray_flops(case["tris"]) * 2
    elif kind == "points":
        b, f = frame_work(case["w"] * case["h"], 100_000, False)
        b, f = b + 12 * case["points"] + 8 * case["w"] * case["h"], f + 70.0 * case["points"]
    elif kind == "learned":
        n = case["w"] * case["h"]
        b, f = n * (40 + 24) + 2 * 610_816, n * (2.0 * 606_208 + ray_flops(case["tris"]))
    else:
        n = case["batch"]
        b, f = n * (4 * FEATURES + 4) + 8 * 610_816, n * 6.0 * 606_208
    return {"bytes": float(b), "flops": float(f)}


# --------------------------------------------------------------------------- exact

def exact(case, seed):
    """The loss and the gradients in 64 bits; the other cases return records of bytes, which have no other value."""
    if case["kind"] != "grad":
        return None
    params, X, y = gradient_inputs(case, int(seed) & 0x3FFFFFFF)
    p = torch.from_numpy(params).cuda().double().requires_grad_()
    h, at, n_in = torch.from_numpy(X).cuda().double(), 0, FEATURES
    for k in range(5):
        n_out = HIDDEN if k < 4 else CLASSES
        W = p[at:at + n_in * n_out].reshape(n_in, n_out)
        b = p[at + n_in * n_out:at + n_in * n_out + n_out]
        at, n_in = at + n_in * n_out + n_out, n_out
        h = h @ W + b
        if k < 4:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    loss = torch.nn.functional.cross_entropy(h, torch.from_numpy(y).cuda().long(), ignore_index=-1)
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad}
