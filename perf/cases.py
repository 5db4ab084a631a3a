"""What the coupling library is timed on: the calls that a solver makes of it, from one cylinder to 512^3 cells.

A case is a dict of plain values with a "kind":
  interact     SolidCloud.interact on device fields (the fraction method, forcing and CUDA graphs as the case says)
  step         one time step of a solver whose fields live on the GPU: interact, apply_forcing, evolve, fix_internal,
               and the new solid states read back
  host         interact_host64 / interact_host on page-locked host fields (an OpenFOAM solver's own storage)
  polymesh     interact on an explicit polyMesh (graded 2-D, or hexahedra with moved points in 3-D)
  mlp_forward  the learned fraction's network on feature records
  mlp_grad     loss and gradient of one training batch of it
prepare() makes the inputs from the seed alone; exact() gives what run() returns in 64 bits, from the published
definitions of the fraction (apex / pyramid volume, midpoint lattice), the direct forcing and the rigid-body update, in
plain torch.  The learned fraction of a coupling pass has no exact(): which cells its network answers is decided by its
own stencil.
"""
import math

import numpy as np
import torch

from sdfibm_gb300 import abi, host, learned
from sdfibm_gb300.cloud import SolidCloud

METHODS = {"refgeo": abi.FRACTION_REFGEO, "subsample": abi.FRACTION_SUBSAMPLE, "learned": abi.FRACTION_LEARNED}
F64 = torch.float64
TWO_D = ("Circle", "Ellipse", "Rectangle", "Plane")


def listed():
    return [
        # the smallest use: flow past one fixed cylinder (2-D, 400 x 200), default options, forces read every step
        dict(name="cylinder2d_step", kind="step", nx=400, ny=200, nz=1, twod=True, h=0.1, solids=1, shapes="Circle",
             r=5.0, sigma=0.0, walls=False, fixed=True, gravity=0.0, collide="off", u_mean=1.0, u_std=0.05, dt=5e-3,
             graphs=False, ft=True),
        # 100 circles settling in a walled box (2-D, 1024^2), contacts, captured steps
        dict(name="sedimentation2d_step", kind="step", nx=1024, ny=1024, nz=1, twod=True, h=1.0 / 1024, solids=100,
             shapes="Circle", r=30.72, sigma=0.0, walls=True, fixed=False, gravity=-10.0, collide="reference",
             u_mean=0.0, u_std=0.1, dt=1e-4, graphs=True, ft=False),
        # a polydisperse suspension with contacts on a mesh with unequal sides: the time step of a GPU-resident solver
        dict(name="suspension_step", kind="step", nx=256, ny=288, nz=224, twod=False, h=1.0 / 256, solids=1800,
             shapes="Sphere,Ellipsoid,Box", r=2.5, sigma=0.4, walls=False, fixed=False, gravity=0.0, collide="spheres",
             u_mean=0.0, u_std=0.1, dt=1e-3, graphs=True, ft=False),
        # the coupling alone with the default options (the reference's fraction, FP64 forcing, forces read back)
        dict(name="poly3d_256_refgeo", kind="interact", nx=256, ny=256, nz=256, twod=False, h=1.0 / 256, solids=4096,
             shapes="Sphere,Ellipsoid", r=2.56, sigma=0.4, method="refgeo", n=10, exact_forcing=True, graphs=False,
             ft=True),
        # the same with the lattice fraction, 10 samples per axis
        dict(name="poly3d_256_subsample", kind="interact", nx=256, ny=256, nz=256, twod=False, h=1.0 / 256,
             solids=4096, shapes="Sphere,Ellipsoid", r=2.56, sigma=0.4, method="subsample", n=10, exact_forcing=True,
             graphs=False, ft=True),
        # the benchmark's workload: 512^3, 16384 solids, FP32 forcing, captured; the reference's fraction ...
        dict(name="poly3d_512_refgeo", kind="interact", nx=512, ny=512, nz=512, twod=False, h=1.0 / 512, solids=16384,
             shapes="Sphere,Ellipsoid,Box", r=2.048, sigma=0.5, method="refgeo", n=10, exact_forcing=False,
             graphs=True, ft=False),
        # ... and the learned one
        dict(name="poly3d_512_learned", kind="interact", nx=512, ny=512, nz=512, twod=False, h=1.0 / 512,
             solids=16384, shapes="Sphere,Ellipsoid,Box", r=2.048, sigma=0.5, method="learned", n=16,
             exact_forcing=False, graphs=True, ft=False),
        # an OpenFOAM-resident caller: FP64 fields in page-locked host memory, the reference's fraction
        dict(name="host64_refgeo", kind="host", nx=192, ny=208, nz=176, twod=False, h=1.0 / 200, solids=750,
             shapes="Sphere,Ellipsoid,Box", r=2.5, sigma=0.4, method="refgeo", n=10, exact_forcing=True, fp64=True),
        # flow past a cylinder on a graded mesh (re200's 280 x 280 cells)
        dict(name="polymesh_cylinder", kind="polymesh", nx=280, ny=280, nz=1, twod=True, h=0.05, solids=1,
             shapes="Circle", r=20.0, sigma=0.0, grade=4.0, jiggle=0.0),
        # particles on a mesh of general hexahedra
        dict(name="polymesh_hex", kind="polymesh", nx=56, ny=52, nz=48, twod=False, h=1.0 / 50, solids=40,
             shapes="Sphere,Ellipsoid,Box", r=3.0, sigma=0.3, grade=1.0, jiggle=0.25),
        # the network on the cut cells of a large step
        dict(name="mlp_forward", kind="mlp_forward", cells=1 << 22),
        # one batch of the shipped training run
        dict(name="mlp_grad", kind="mlp_grad", cells=32768),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    """A case of the listed ranges: sizes over their logarithm, odd ones among them."""
    kind = rng.choice(["interact", "interact", "interact", "step", "step", "host", "polymesh", "polymesh",
                       "mlp_forward", "mlp_grad"])
    if kind == "mlp_forward":
        return dict(kind=kind, cells=int(_log(rng, 1000, 1 << 22)))
    if kind == "mlp_grad":
        return dict(kind=kind, cells=int(_log(rng, 1000, 1 << 18)))
    twod = kind == "step" and rng.random() < 0.5 or kind == "polymesh" and rng.random() < 0.4
    if kind == "polymesh":
        if twod:
            side = _log(rng, 80, 300)
            r, count, shapes = side * rng.uniform(0.03, 0.08), rng.randint(1, 4), "Circle"
            dims = [int(side * rng.uniform(0.8, 1.2)), int(side * rng.uniform(0.8, 1.2)), 1]
        else:
            side = _log(rng, 20, 56)
            r, count, shapes = rng.uniform(2.0, 4.0), 1 + int((side / 9.0) ** 3 * rng.uniform(0.1, 0.25)), \
                rng.choice(["Sphere", "Sphere,Ellipsoid,Box"])
            dims = [int(side * rng.uniform(0.8, 1.15)) for _ in range(3)]
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], twod=bool(twod), h=round(rng.uniform(0.01, 0.1), 3),
                    solids=count, shapes=shapes, r=round(r, 2), sigma=0.0 if twod else 0.3,
                    grade=rng.choice([1.0, 4.0, 20.0]) if twod else 1.0, jiggle=0.0 if twod else 0.25)
    if twod:
        side = _log(rng, 200, 1100)
        dims = [int(side * rng.uniform(0.8, 1.25)), int(side * rng.uniform(0.8, 1.25)), 1]
        r = side * rng.uniform(0.012, 0.03)
        # circles and their gaps cover a tenth to a quarter of the box
        count = max(1, int(rng.uniform(0.1, 0.25) * dims[0] * dims[1] / (math.pi * r * r)))
        walls = rng.random() < 0.5
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=1, twod=True, h=1.0 / dims[0], solids=count,
                    shapes="Circle", r=round(r, 2), sigma=0.0, walls=walls, fixed=False,
                    gravity=-10.0 if walls else 0.0, collide="reference" if walls else "spheres", u_mean=0.0,
                    u_std=0.1, dt=1e-4, graphs=rng.random() < 0.5, ft=rng.random() < 0.5)
    side = _log(rng, 48, {"interact": 448, "step": 256, "host": 192}[kind])
    dims = [max(17, int(side * rng.uniform(0.8, 1.12))) for _ in range(3)]
    r, sigma = round(rng.uniform(1.6, 4.0), 2), round(rng.uniform(0.1, 0.5), 2)
    shapes = rng.choice(["Sphere", "Sphere,Ellipsoid", "Sphere,Ellipsoid,Box"])
    # up to one solid per cube of 10 r, as dense as the listed workloads
    count = min(16384, max(1, int(rng.uniform(0.2, 1.0) * dims[0] * dims[1] * dims[2] / (10 * r) ** 3)))
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], twod=False, h=1.0 / dims[0], solids=count, shapes=shapes,
             r=r, sigma=sigma)
    if kind == "step":
        c.update(walls=False, fixed=False, gravity=0.0, collide=rng.choice(["off", "spheres"]), u_mean=0.0, u_std=0.1,
                 dt=1e-3, graphs=rng.random() < 0.5, ft=rng.random() < 0.5)
        return c
    method = rng.choice(["refgeo", "subsample"] if kind == "host" else ["refgeo", "subsample", "learned"])
    c.update(method=method, n=16 if method == "learned" else rng.choice([4, 6, 8, 10, 12]),
             exact_forcing=method != "learned" and rng.random() < 0.7)
    if kind == "host":
        c["fp64"] = rng.random() < 0.7
    else:
        c["graphs"] = rng.random() < 0.5
        c["ft"] = bool(c["exact_forcing"])  # with FP32 forcing the forces stay on the device
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------
class Solids:
    """Plain arrays of the solids of a case: shape name, sizes [S, 3], pose and motion."""

    def __init__(self, case, seed, box):
        rng = np.random.default_rng([int(seed), 11])
        kinds = case["shapes"].split(",")
        S = case["solids"]
        h, twod = case["h"], case["twod"]
        r = case["r"] * h * np.exp(case["sigma"] * rng.standard_normal(S))
        a, b = rng.uniform(1.0, 3.0, S), rng.uniform(1.0, 3.0, S)
        kind = np.array([kinds[i % len(kinds)] for i in range(S)])
        size = np.stack([r, np.where(kind == "Sphere", r, r * a), np.where(kind == "Sphere", r, r * b)], axis=1)
        if twod:
            size[:, 1:] = r[:, None]
        bound = np.where(kind == "Box", np.linalg.norm(size, axis=1), size.max(axis=1))
        # no solid larger than a fifth of the box, as the long tail of a lognormal draw on a small mesh would be
        scale = np.minimum(1.0, 0.2 * (box[1] - box[0])[:2 if twod else 3].min() / bound)
        if not twod:
            # none of 17 to 26 cells: a program may hold several contexts at once (they are timed side by side), and
            # those with flood-fill bitmaps of 48 to 96 KB share one reservation of shared memory per process
            scale = np.where((bound * scale > 17 * h) & (bound * scale < 26 * h), 17 * h / bound, scale)
        size, bound = size * scale[:, None], bound * scale
        pos = _place(rng, bound, box, twod, seed)
        if case.get("fixed") or (case["kind"] == "polymesh" and twod and S == 1):
            pos[0, :2] = 0.5 * (box[0] + box[1])[:2] - (10.0 * h if case.get("fixed") else 0.0) + rng.uniform(-h, h, 2)
        if twod:
            t = rng.uniform(0, math.pi, S)
            quat = np.stack([np.cos(t / 2), 0 * t, 0 * t, np.sin(t / 2)], axis=1)
        else:
            quat = rng.standard_normal((S, 4))
            quat /= np.linalg.norm(quat, axis=1)[:, None]
        vel, omega = rng.normal(0, 0.05, (S, 3)), rng.normal(0, 0.5, (S, 3))
        mask = np.ones((S, 6))
        if twod:
            vel[:, 2] = 0.0
            omega[:, :2] = 0.0
            mask[:] = [1, 1, 0, 0, 0, 1]
        if case.get("fixed"):
            vel[:], omega[:], mask[:] = 0.0, 0.0, 0.0
        if case.get("walls"):  # four planes around the box, normals into the fluid, listed first
            lo, hi = box
            mid = 0.5 * (lo + hi)
            wp = np.array([[lo[0], mid[1], 0], [hi[0], mid[1], 0], [mid[0], lo[1], 0], [mid[0], hi[1], 0]])
            ang = np.radians([-90.0, 90.0, 0.0, 180.0])
            wq = np.stack([np.cos(ang / 2), 0 * ang, 0 * ang, np.sin(ang / 2)], axis=1)
            z = np.zeros((4, 3))
            kind = np.concatenate([["Plane"] * 4, kind])
            size, pos, quat = np.concatenate([z, size]), np.concatenate([wp, pos]), np.concatenate([wq, quat])
            vel, omega, mask = np.concatenate([z, vel]), np.concatenate([z, omega]), \
                np.concatenate([np.zeros((4, 6)), mask])
        self.kind, self.size, self.pos, self.quat, self.vel, self.omega, self.mask = kind, size, pos, quat, vel, \
            omega, mask
        self.free = not twod and not case.get("fixed")
        self.rho = 1.5


def _place(rng, bound, box, twod, seed):
    """Random placement without overlap of the bounding spheres, the largest first, in rounds on the GPU; a solid that
    finds no room in 60 rounds stays where its last draw put it (and may touch another)."""
    S = len(bound)
    lo, hi = torch.tensor(box[0], device="cuda", dtype=F64), torch.tensor(box[1], device="cuda", dtype=F64)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    order = np.argsort(-bound, kind="stable")
    R = torch.tensor(bound[order], device="cuda", dtype=F64)
    P = torch.zeros((S, 3), device="cuda", dtype=F64)
    for b0 in range(0, S, 1024):
        rows = torch.arange(b0, min(S, b0 + 1024), device="cuda")
        for attempt in range(60):
            r = R[rows, None]
            p = lo + r + torch.rand((len(rows), 3), generator=g, device="cuda", dtype=F64) * (hi - lo - 2 * r)
            if twod:
                p[:, 2] = 0.0
            P[rows] = p
            done = torch.ones(b0 + 1024, dtype=torch.bool, device="cuda")[:min(S, b0 + 1024)]
            done[rows] = False
            near = torch.cdist(p, P[:len(done)], compute_mode="donot_use_mm_for_euclid_dist") < r + R[None, :len(done)]
            earlier = done[None, :] | (torch.arange(len(done), device="cuda")[None, :] < rows[:, None])
            rows = rows[(near & earlier).any(dim=1)]
            if len(rows) == 0:
                break
    out = np.zeros((S, 3))
    out[order] = P.cpu().numpy()
    return out


def _box(case):
    n = np.array([case["nx"], case["ny"], case["nz"]])
    if case["twod"]:
        lo = np.array([0.0, 0.0, -0.5])
        hz = 1.0
    else:
        lo, hz = np.zeros(3), case["h"]
    h = np.array([case["h"], case["h"], hz])
    return lo, lo + n * h, h


def _velocity(case, seed, ncells):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 104729 + 5)
    U = torch.randn((3, ncells), generator=g, device="cuda", dtype=torch.float32) * case.get("u_std", 0.1)
    U[0] += case.get("u_mean", 0.0)
    return U


_SHAPE_ARGS = {"Circle": ("radius",), "Sphere": ("radius",), "Ellipse": ("radiusa", "radiusb"),
               "Rectangle": ("radiusa", "radiusb"), "Ellipsoid": ("radiusa", "radiusb", "radiusc"),
               "Box": ("radiusa", "radiusb", "radiusc"), "Plane": ()}


def _descriptors(s):
    out = []
    motions = {}
    for i in range(len(s.kind)):
        shape = host.make_shape(s.kind[i], **dict(zip(_SHAPE_ARGS[s.kind[i]], s.size[i])))
        word = "b" + "".join("%d" % v for v in s.mask[i])
        if word not in motions:
            motions[word] = None if s.free else host.mask_motion(word)
        d = host.make_solid(i, shape, s.rho, s.pos[i], vel=s.vel[i], omega=s.omega[i], motion=motions[word])
        d.quat[:] = s.quat[i].tolist()
        out.append(d)
    return out


_stream = []  # the program's stream


def _options(case):
    o = dict(rho_f=1.0, exact_forcing=1, fraction_method=METHODS[case.get("method", "refgeo")],
             subsample_n=case.get("n", 10), graphs=int(case.get("graphs", False)))
    if "exact_forcing" in case:
        o["exact_forcing"] = int(case["exact_forcing"])
    if case["kind"] == "step":
        o["gravity"] = (0.0, case["gravity"], 0.0)
        o["collision_mode"] = {"off": abi.COLLISION_OFF, "reference": abi.COLLISION_REFERENCE,
                               "spheres": abi.COLLISION_SPHERES}[case["collide"]]
    return abi.options(**o)


def _dataset(case, seed):
    """Labelled cut cells as the training run draws them."""
    return learned.make_dataset(torch, case["cells"], 1000 + int(seed))[:2]


def _parameters(case, seed):
    """The shipped network, or for a gradient a network at the start of its training."""
    return torch.from_numpy(learned.load_model()[0] if case["kind"] == "mlp_forward" else
                            learned.init_params(int(seed))).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("mlp"):
        feat, label = _dataset(case, seed)
        return dict(case=case, feat=feat, label=label, params=_parameters(case, seed))
    if kind == "polymesh":
        mesh = _polymesh(case, seed)
        s = Solids(case, seed, _poly_box(mesh))
        cloud = SolidCloud.from_polymesh(mesh["points"], mesh["face_off"], mesh["faces"].reshape(-1), mesh["owner"],
                                         mesh["neighbour"], _descriptors(s), _options(case), twod=case["twod"])
        return dict(case=case, cloud=cloud, U=_velocity(case, seed, cloud.ncells), fields=cloud.new_fields(), dt=1e-3)
    lo, hi, h = _box(case)
    s = Solids(case, seed, (lo, hi))
    mesh = abi.mesh_desc((case["nx"], case["ny"], case["nz"]), lo, h, twod=int(case["twod"]))
    stream = None
    if case.get("graphs"):
        if not _stream:
            _stream.append(torch.cuda.Stream())
        stream = _stream[0]
    cloud = SolidCloud(mesh, _descriptors(s), _options(case), stream=stream)
    if case.get("method") == "learned":
        params, tau, rho_min, _ = learned.load_model()
        cloud.set_fraction_model(params, tau, rho_min)
    st = dict(case=case, cloud=cloud, stream=stream, dt=case.get("dt", 1e-3), t=0.0)
    U = _velocity(case, seed, cloud.ncells)
    if kind == "host":
        ft, ct = (torch.float64, torch.float64) if case["fp64"] else (torch.float32, torch.int32)
        N = cloud.ncells
        shapes = dict(As=((N,), ft), Fs=((N, 3) if case["fp64"] else (3, N), ft), Ts=((N,), ft), Ct=((N,), ct))
        st["keep"] = {k: torch.zeros(sh, dtype=t, pin_memory=True) for k, (sh, t) in shapes.items()}
        Uh = (U.t().contiguous() if case["fp64"] else U).to(ft)
        st["keep"]["U"] = torch.empty(Uh.shape, dtype=ft, pin_memory=True).copy_(Uh)
        st["U"] = st["keep"]["U"].numpy()
        st["fields"] = {k: st["keep"][k].numpy() for k in shapes}
        return st
    st["U"], st["fields"] = U, cloud.new_fields()
    if kind == "step":
        st["states"] = (abi.SolidState * len(s.kind))()
    torch.cuda.synchronize()  # the fields were written on torch's stream
    return st


# ---- one pass ----------------------------------------------------------------------------------------------------
def _states(buf):
    """The solid states as an array [S, 43]: the record's doubles, without the two first-step flags behind them."""
    a = np.frombuffer(buf, dtype=np.float64).reshape(len(buf), -1)
    return a[:, :-1]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "mlp_forward":
        return learned.forward(torch, st["params"], st["feat"])
    if kind == "mlp_grad":
        return learned.loss_grad(torch, st["params"], st["feat"], st["label"])
    cloud, f, dt = st["cloud"], st["fields"], st["dt"]
    if kind == "host":
        call = cloud.interact_host64 if case["fp64"] else cloud.interact_host
        return dict(f, FT=call(0.0, dt, st["U"], f))
    if kind == "polymesh":
        return dict(f, FT=cloud.interact(0.0, dt, st["U"], f))
    FT = cloud.interact(st["t"], dt, st["U"], f, want_ft=case["ft"])
    out = dict(f)
    if kind == "step":
        cloud.apply_forcing(dt, f, st["U"])
        cloud.evolve(st["t"], dt)
        cloud.fix_internal(f["Ct"], st["U"])
        cloud._check(cloud._L.sdfibm_cuda_get_solids(cloud._h, st["states"], len(st["states"])))
        st["t"] += dt
        out["U"], out["states"] = st["U"], _states(st["states"])
    if case["ft"]:
        out["FT"] = FT
    return out


# ---- work --------------------------------------------------------------------------------------------------------
def _touched(case):
    """Expected (touched, cut) cells: a body of volume V and surface A in cell units touches about V + 0.75 A cells and
    cuts about 1.5 A (2-D: V + 0.64 A and 1.27 A)."""
    rng = np.random.default_rng(0)
    S = case["solids"]
    r = case["r"] * np.exp(case["sigma"] * rng.standard_normal(S))
    a, b = rng.uniform(1.0, 3.0, S), rng.uniform(1.0, 3.0, S)
    kinds = case["shapes"].split(",")
    touched = cut = 0.0
    for q, k in enumerate(kinds):
        x, y, z = r[q::len(kinds)], (r * a)[q::len(kinds)], (r * b)[q::len(kinds)]
        if k == "Circle":
            V, A, w, c = math.pi * x * x, 2 * math.pi * x, 0.64, 1.27
        else:
            if k == "Sphere":
                V, A = 4 / 3 * math.pi * x ** 3, 4 * math.pi * x ** 2
            elif k == "Ellipsoid":
                e = 1.6075
                V = 4 / 3 * math.pi * x * y * z
                A = 4 * math.pi * (((x * y) ** e + (x * z) ** e + (y * z) ** e) / 3) ** (1 / e)
            else:
                V, A = 8 * x * y * z, 8 * (x * y + y * z + x * z)
            w, c = 0.75, 1.5
        touched += float(np.sum(V + w * A))
        cut += float(np.sum(c * A))
    if case.get("walls"):
        touched += 2 * (case["nx"] + case["ny"])
        cut += 2 * (case["nx"] + case["ny"])
    N = case["nx"] * case["ny"] * case["nz"]
    return min(touched, N), min(cut, N)


def work(case):
    kind = case["kind"]
    if kind.startswith("mlp"):
        n = case["cells"]
        flops = 2 * (16 * 64 + 64 * 64 + 64)
        # features and prior in; the fraction out, or the labels in and the gradient out
        return dict(bytes=72 * n + 4 * abi.MLP_NPARAM, flops=(flops if kind == "mlp_forward" else 3 * flops) * n)
    touched, cut = _touched(case)
    S = case["solids"] + (4 if case.get("walls") else 0)
    # U read, As / Fs / Ts / Ct written at the touched cells; a state read and a force written per solid
    per = 72 if case.get("fp64") else 36
    b = per * touched + 392 * S
    fraction = {"refgeo": 300.0, "subsample": 20.0 * case.get("n", 10) ** 2, "learned": 125 * 10 + 72 * 40 + 10400.0}
    f = 40 * touched + fraction[case.get("method", "refgeo")] * cut
    if kind == "step":
        b += 24 * touched + 12 * max(0.0, touched - cut) + 688 * S  # U updated and pinned, the states written
        f += 9 * touched + 20 * 400 * S
    return dict(bytes=b, flops=f)


# ---- the same in 64 bits -----------------------------------------------------------------------------------------
SMALL = 1e-6   # the reference's guard in the apex denominator
TOL = 1e-8     # its filter of signed distances


def _rotations(quat):
    w, x, y, z = quat.unbind(-1)
    R = torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                     w * w - x * x + y * y - z * z, 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                     w * w - x * x - y * y + z * z], dim=-1)
    return R.reshape(quat.shape[:-1] + (3, 3))


class Exact:
    def __init__(self, s):
        t = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda", dtype=F64)
        self.kind, self.size, self.pos, self.quat = s.kind, t(s.size), t(s.pos), t(s.quat)
        self.vel, self.omega, self.mask = t(s.vel), t(s.omega), t(s.mask)
        self.R = _rotations(self.quat)
        self.code = torch.tensor([_CODES.index(k) for k in s.kind], device="cuda")

    def local(self, sid, p):
        """Points p [n, ..., 3] in the frame of solid sid [n]."""
        shape = (len(sid),) + (1,) * (p.dim() - 2) + (3,)
        d = p - self.pos[sid].reshape(shape)
        R = self.R[sid].reshape((len(sid),) + (1,) * (p.dim() - 2) + (3, 3))
        return (R.transpose(-1, -2) @ d[..., None])[..., 0]

    def each(self, sid, q, fn):
        """fn(kind, sizes, points) over the shapes present, points [n, ..., 3]."""
        out = None
        for c in torch.unique(self.code[sid]).tolist():
            at = self.code[sid] == c
            a = self.size[sid[at]].reshape((-1,) + (1,) * (q.dim() - 2) + (3,))
            v = fn(_CODES[c], a, q[at])
            if out is None:
                out = torch.zeros(q.shape[:-1], dtype=v.dtype, device=q.device)
            out[at] = v
        return out if out is not None else torch.zeros(q.shape[:-1], dtype=torch.bool, device=q.device)

    def inside(self, sid, q):
        def fn(k, a, p):
            if k == "Plane":
                return p[..., 1] < 0
            if k in ("Rectangle", "Box"):
                return (p.abs() < a)[..., :2 if k == "Rectangle" else 3].all(-1)
            v = (p / a) ** 2
            return (v[..., :2] if k in TWO_D else v).sum(-1) < 1
        return self.each(sid, q, fn)

    def distance(self, sid, q):
        def fn(k, a, p):
            if k == "Plane":
                return p[..., 1]
            if k in ("Rectangle", "Box"):
                d = (p.abs() - a)[..., :2 if k == "Rectangle" else 3]
                phi = d.clamp(min=0).norm(dim=-1) + d.amax(-1).clamp(max=0)
            elif k in ("Circle", "Sphere"):
                phi = (p[..., :2] if k == "Circle" else p).norm(dim=-1) - a[..., 0]
            else:
                v = (p / a)[..., :2 if k == "Ellipse" else 3]
                w = (p / a ** 2)[..., :2 if k == "Ellipse" else 3]
                phi = 0.5 * ((v * v).sum(-1) - 1) / w.norm(dim=-1)
            return torch.where(phi.abs() < TOL, torch.full_like(phi, -TOL), phi)
        return self.each(sid, q, fn)


_CODES = ("Circle", "Sphere", "Ellipse", "Rectangle", "Ellipsoid", "Box", "Plane")


def _apex(P, phi):
    """The apex of points P [n, k, 3] with distances phi [n, k]: on the segment from the first point to the first later
    one across the surface."""
    other = phi[:, :1] * phi[:, 1:] <= 0
    row = torch.arange(len(P), device=P.device)
    j = torch.where(other.any(1), other.to(torch.uint8).argmax(1) + 1, P.shape[1] - 1)
    B, pb = P[row, j], phi[row, j]
    pa = phi[:, 0]
    return P[:, 0] - (pa.abs() / (SMALL + pa.abs() + pb.abs()))[:, None] * (P[:, 0] - B)


def _face_geometry(Q):
    """Centres and area vectors of quadrilaterals Q [n, 4, 3]: triangles about the mean point."""
    m = Q.mean(1)
    nxt = Q.roll(-1, 1)
    N = torch.linalg.cross(nxt - Q, m[:, None] - Q)
    A = N.norm(dim=-1)
    C = ((Q + nxt + m[:, None]) / 3 * A[..., None]).sum(1) / A.sum(1)[:, None]
    return C, 0.5 * N.sum(1)


def _apex_volume(P, phi, slots, twod):
    """Solid volume of hexahedra: points P [n, 8, 3] (ascending labels), distances phi [n, 8], the point slots of
    their six faces [n, 6, 4]."""
    apex = _apex(P, phi)
    if twod:
        apex[:, 2] = 0.0
    vol = torch.zeros(len(P), dtype=F64, device=P.device)
    rows = torch.arange(len(P), device=P.device)[:, None]
    for f in range(6):
        Q, ph = P[rows, slots[:, f]], phi[rows, slots[:, f]]
        C, Sf = _face_geometry(Q)
        fa = _apex(Q, ph)
        pa, pb = ph, ph.roll(-1, 1)
        frac = torch.where((pa > 0) & (pb > 0), 0.0, torch.where((pa <= 0) & (pb <= 0), 1.0, torch.where(
            pa > 0, -pb / (pa - pb), -pa / (pb - pa)))).to(F64)
        area = (0.5 * torch.linalg.cross(Q.roll(-1, 1) - Q, fa[:, None] - Q).norm(dim=-1) * frac).sum(1)
        eps = area / Sf.norm(dim=-1)
        eps = torch.where((ph > 0).all(1), 0.0, torch.where((ph <= 0).all(1), 1.0, eps))
        vol += eps * ((apex - C) * Sf).sum(1).abs() / 3
    return vol


# point slots of the faces of a cell of the uniform mesh: 0 (i,j,k) 1 (i+1,j,k) 2 (i,j+1,k) 3 (i+1,j+1,k), 4..7 at k+1
_HIGH = [[1, 3, 7, 5], [2, 6, 7, 3], [4, 5, 7, 6]]
_LOW_IN, _LOW_WALL = [[0, 2, 6, 4], [0, 4, 5, 1], [0, 1, 3, 2]], [[0, 4, 6, 2], [0, 1, 5, 4], [0, 2, 3, 1]]


def _uniform_pairs(case, ex):
    """(solid, i, j, k, alpha) of every touched cell, in pieces."""
    lo, hi, h = _box(case)
    n = np.array([case["nx"], case["ny"], case["nz"]])
    pos, size = ex.pos.cpu().numpy(), ex.size.cpu().numpy()
    reach = np.where(ex.kind == "Plane", 1e9, np.linalg.norm(size, axis=1))[:, None] + 2 * h
    b0 = np.clip(np.floor((pos - reach - lo) / h), 0, n - 1).astype(np.int64)
    b1 = np.clip(np.ceil((pos + reach - lo) / h), 1, n).astype(np.int64)
    if case["twod"]:
        b0[:, 2], b1[:, 2] = 0, n[2]
    ext = b1 - b0
    cells = ext.prod(axis=1)
    T = lambda a, t=torch.int64: torch.tensor(a, device="cuda", dtype=t)
    o, hh = T(lo, F64), T(h, F64)
    corner = torch.tensor([[q & 1, (q >> 1) & 1, q >> 2] for q in range(8)], device="cuda")
    s0 = 0
    while s0 < len(cells):
        s1, tot = s0, 0
        while s1 < len(cells) and (s1 == s0 or tot + cells[s1] <= 3_000_000):
            tot += cells[s1]
            s1 += 1
        sid = torch.repeat_interleave(torch.arange(s0, s1, device="cuda"), T(cells[s0:s1]))
        start = T(np.concatenate([[0], np.cumsum(cells[s0:s1])[:-1]]))
        e = torch.arange(int(tot), device="cuda") - start[sid - s0]
        E, B = T(ext)[sid], T(b0)[sid]
        ijk = torch.stack([e % E[:, 0], (e // E[:, 0]) % E[:, 1], e // (E[:, 0] * E[:, 1])], dim=1) + B
        del e, E, B
        s0 = s1
        cnt = torch.zeros(len(sid), dtype=torch.int8, device="cuda")
        for q in range(8):
            cnt += ex.inside(sid, ex.local(sid, o + (ijk + corner[q]) * hh))
        keep = cnt > 0
        sid, ijk, cnt = sid[keep], ijk[keep], cnt[keep]
        alpha = torch.ones(len(sid), dtype=F64, device="cuda")
        cut = torch.nonzero(cnt < 8)[:, 0]
        for c in cut.split(200_000):
            alpha[c] = _lattice(case, ex, sid[c], ijk[c], o, hh) if case.get("method") == "subsample" else \
                _uniform_apex(case, ex, sid[c], ijk[c], o, hh, corner)
        yield sid, ijk, alpha


def _uniform_apex(case, ex, sid, ijk, o, hh, corner):
    P = o + (ijk[:, None] + corner) * hh
    phi = ex.distance(sid, ex.local(sid, P))
    slots = torch.tensor(_HIGH + _LOW_IN, device="cuda")[None].repeat(len(sid), 1, 1)
    for a in range(3):
        wall = torch.tensor(_LOW_WALL[a], device="cuda")
        slots[:, 3 + a] = torch.where((ijk[:, a] == 0)[:, None], wall, slots[:, 3 + a])
    return _apex_volume(P, phi, slots, case["twod"]) / float(hh.prod())


def _lattice(case, ex, sid, ijk, o, hh):
    n = case["n"]
    t = (2 * torch.arange(n, device="cuda", dtype=F64) + 1) / (2 * n)
    xy = torch.stack(torch.meshgrid(t, t, indexing="ij"), dim=-1).reshape(-1, 2)
    count = torch.zeros(len(sid), dtype=torch.int64, device="cuda")
    for z in [torch.tensor(0.5, device="cuda", dtype=F64)] if case["twod"] else t:
        off = torch.cat([xy, z.expand(len(xy), 1)], dim=1)
        for part in torch.arange(len(sid), device="cuda").split(40_000):
            p = o + (ijk[part][:, None] + off) * hh
            count[part] += ex.inside(sid[part], ex.local(sid[part], p)).sum(1)
    return count.to(F64) / (n * n * (1 if case["twod"] else n))


def _couple(ex, N, pieces, U, dt, S):
    """Fields and forces of (solid, cell, alpha, centre, volume) pieces."""
    As = torch.zeros(N, dtype=F64, device="cuda")
    Fs = torch.zeros((3, N), dtype=F64, device="cuda")
    FT = torch.zeros((S, 6), dtype=F64, device="cuda")
    for sid, cell, alpha, C, V in pieces:
        d = C - ex.pos[sid]
        us = ex.vel[sid] + torch.linalg.cross(ex.omega[sid], d)
        f = alpha[:, None] * (U[:, cell].t().to(F64) - us)
        As.index_add_(0, cell, alpha)
        Fs.index_add_(1, cell, (f / dt).t())
        FT.index_add_(0, sid, torch.cat([f, torch.linalg.cross(d, f)], dim=1) * (V / dt if torch.is_tensor(V) else
                                                                               torch.tensor(V / dt)))
    return dict(As=As.clamp(max=1.0), Ts=As, Fs=Fs, FT=FT)


def _uniform_pieces(case, ex):
    lo, hi, h = _box(case)
    o, hh = torch.tensor(lo, device="cuda"), torch.tensor(h, device="cuda")
    for sid, ijk, alpha in _uniform_pairs(case, ex):
        cell = ijk[:, 0] + case["nx"] * (ijk[:, 1] + case["ny"] * ijk[:, 2])
        yield sid, cell, alpha, o + (ijk + 0.5) * hh, float(np.prod(h))


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("mlp"):
        return _exact_network(case, seed)
    if case.get("method") == "learned":
        return None
    if kind == "polymesh":
        mesh = _polymesh(case, seed)
        ex = Exact(Solids(case, seed, _poly_box(mesh)))
        N = case["nx"] * case["ny"] * case["nz"]
        out = _couple(ex, N, _poly_pieces(case, mesh, ex), _velocity(case, seed, N), 1e-3, len(ex.kind))
        return dict(out, Ct=None)
    lo, hi, h = _box(case)
    s = Solids(case, seed, (lo, hi))
    ex = Exact(s)
    N = case["nx"] * case["ny"] * case["nz"]
    U = _velocity(case, seed, N)
    dt = case.get("dt", 1e-3)
    out = dict(_couple(ex, N, _uniform_pieces(case, ex), U, dt, len(s.kind)), Ct=None)
    if kind == "host":
        if case["fp64"]:
            out["Fs"] = out["Fs"].t()
        return {k: None if v is None else v.cpu().numpy() for k, v in out.items()}
    FT = out["FT"]
    if kind == "interact":
        if not case["ft"]:
            out["FT"] = None
        return out
    out["FT"] = FT if case["ft"] else None
    U = U.to(F64) - out["Fs"] * dt
    out["states"] = _evolve(case, s, ex, FT, dt, (lo, hi))
    # the cells whose last solid holds them whole move with it (fixInternal)
    owner = torch.full((N,), -1, dtype=torch.int64, device="cuda")
    whole = []
    for sid, cell, alpha, C, V in _uniform_pieces(case, ex):
        inside = _all_inside(case, ex, sid, cell)
        code = 2 * sid + inside
        owner.scatter_reduce_(0, cell, code, "amax")
        whole.append((cell[inside], sid[inside], C[inside]))
    st = out["states"]
    pos, vel, omega = st[:, 0:3], st[:, 7:10], st[:, 10:13]
    for cell, sid, C in whole:
        last = owner[cell] == 2 * sid + 1
        cell, sid, C = cell[last], sid[last], C[last]
        U[:, cell] = (vel[sid] + torch.linalg.cross(omega[sid], C - pos[sid])).t()
    out["U"] = U
    return out


def _all_inside(case, ex, sid, cell):
    lo, hi, h = _box(case)
    o, hh = torch.tensor(lo, device="cuda"), torch.tensor(h, device="cuda")
    ijk = torch.stack([cell % case["nx"], (cell // case["nx"]) % case["ny"], cell // (case["nx"] * case["ny"])], dim=1)
    out = torch.ones(len(sid), dtype=torch.bool, device="cuda")
    for q in range(8):
        c = torch.tensor([q & 1, (q >> 1) & 1, q >> 2], device="cuda")
        out &= ex.inside(sid, ex.local(sid, o + (ijk + c) * hh))
    return out


def _evolve(case, s, ex, FT, dt, box):
    """The states after one evolve from the construction state with fluid force FT (rho_f = 1): 20 sub-steps (one for a
    single solid) of force, contact and move; columns as the library's state record holds them."""
    S = len(s.kind)
    nsub = 1 if S == 1 else 20
    ds = dt / nsub
    a, b, c = ex.size.unbind(1)
    pi = math.pi
    V, I = torch.zeros(S, dtype=F64, device="cuda"), torch.ones((S, 3), dtype=F64, device="cuda")
    for k in set(s.kind.tolist()) - {"Plane"}:
        at = torch.tensor(s.kind == k, device="cuda")
        x, y, z = a[at], b[at], c[at]
        if k == "Circle":
            v = pi * x * x
            m = (0.5 * v * x * x)[:, None].expand(-1, 3)
        elif k == "Sphere":
            v = 4 / 3 * pi * x ** 3
            m = (0.4 * v * x * x)[:, None].expand(-1, 3)
        else:
            v, e = (4 / 3 * pi * x * y * z, 0.2) if k == "Ellipsoid" else (8 * x * y * z, 1 / 3)
            m = e * v[:, None] * torch.stack([y * y + z * z, x * x + z * z, x * x + y * y], dim=1)
        V[at], I[at] = v, m
    plane = torch.tensor(s.kind == "Plane", device="cuda")
    rB = torch.where(plane, 0.0, ex.size.amax(1))
    mass = V * s.rho
    minv = torch.where(plane, 0.0, 1 / torch.where(plane, 1.0, mass))
    Iinv = 1 / (I * s.rho)
    g = torch.tensor([0.0, case["gravity"], 0.0], device="cuda", dtype=F64)
    pos, quat, vel, om = ex.pos.clone(), ex.quat.clone(), ex.vel.clone(), ex.omega.clone()
    masked = torch.full((S,), not s.free, device="cuda")
    lo, hi = (torch.tensor(v, device="cuda", dtype=F64) for v in box)
    for _ in range(nsub):
        force = FT[:, :3] + (mass * (s.rho - 1.0) / s.rho)[:, None] * g
        torque = FT[:, 3:]
        if case["collide"] != "off":
            d = 2 * float(rB.max())
            dims = torch.ceil((hi - lo) / d).to(torch.int64)
            key3 = torch.floor((pos - lo) / d).to(torch.int64)
            key = key3[:, 0] * dims[1] * dims[2] + key3[:, 1] * dims[2] + key3[:, 2]
            on = (key >= 0) & (key < dims.prod())
            cell = torch.stack([key // (dims[1] * dims[2]), (key // dims[2]) % dims[1], key % dims[2]], dim=1)
            ball = torch.nonzero(~plane)[:, 0]
            for rows in ball.split(1024):
                D = pos[ball][None] - pos[rows][:, None]
                dist = D.norm(dim=-1)
                depth = rB[rows][:, None] + rB[ball][None] - dist
                hit = (depth >= 0) & (rows[:, None] != ball[None]) & on[rows][:, None] & on[ball][None] & \
                    ((cell[rows][:, None] - cell[ball][None]).abs() <= 1).all(-1)
                w = torch.where(hit, 1e4 * depth / torch.where(hit, dist, 1.0), 0.0)
                force = force.index_add(0, rows, -(w[..., None] * D).sum(1))
            for p in torch.nonzero(plane)[:, 0].tolist():
                n = ex.R[p][:, 1]
                depth = rB[ball] - (pos[ball] - pos[p]) @ n
                hit = (depth >= 0) & on[ball] & on[p] & ((cell[ball] - cell[p]).abs() <= 1).all(-1)
                fc = torch.where(hit, 1e4 * depth, 0.0)[:, None] * n
                force = force.index_add(0, ball, fc)
                force[p] -= fc.sum(0)
        R = _rotations(quat)
        v1 = vel + force * minv[:, None] * ds
        W = R @ (Iinv[:, :, None] * R.transpose(1, 2))
        o1 = om + (W @ torque[..., None])[..., 0] * ds
        v1 = torch.where(masked[:, None], v1 * ex.mask[:, :3], v1)
        o1 = torch.where(masked[:, None], o1 * ex.mask[:, 3:], o1)
        pos = pos + 0.5 * (v1 + vel) * ds
        hv = 0.25 * (o1 + om)
        qw, qv = quat[:, :1], quat[:, 1:]
        dq = torch.cat([-(hv * qv).sum(1, keepdim=True), qw * hv + torch.linalg.cross(hv, qv)], dim=1)
        quat = quat + dq * ds
        quat = quat / quat.norm(dim=1, keepdim=True)
        vel, om = v1, o1
    z = torch.zeros((S, 12), dtype=F64, device="cuda")
    return torch.cat([pos, quat, vel, om, force, torque, FT, FT, z], dim=1)


def _exact_network(case, seed):
    feat, label = _dataset(case, seed)
    p = _parameters(case, seed).to(F64)
    if case["kind"] == "mlp_grad":
        p.requires_grad_(True)
    W1, b1, W2, b2, w3, b3 = torch.split(p, [1024, 64, 4096, 64, 64, 1])

    def net(x):
        h = torch.nn.functional.silu(x[:16].t() @ W1.reshape(64, 16).t() + b1)
        h = torch.nn.functional.silu(h @ W2.reshape(64, 64).t() + b2)
        return torch.sigmoid(x[16] + h @ w3 + b3)
    if case["kind"] == "mlp_forward":
        return torch.cat([net(x.to(F64)) for x in feat.split(1 << 20, dim=1)])
    loss = ((net(feat.to(F64)) - label.to(F64)) ** 2).mean()
    loss.backward()
    return float(loss), p.grad.cpu().numpy()


# ---- polyMesh ----------------------------------------------------------------------------------------------------
def _lines(n, lo, h, grade):
    """Mesh lines of one direction: the middle third uniform, the outer ones growing outwards by `grade` in all (the
    multi-block grading of a flow past a body)."""
    if grade == 1.0 or n < 9:
        return lo + h * np.arange(n + 1)
    m = n // 3
    w = np.concatenate([np.geomspace(grade, 1.0, m), np.ones(n - 2 * m), np.geomspace(1.0, grade, m)])
    x = np.concatenate([[0.0], np.cumsum(w)])
    return lo + x * h


def _polymesh(case, seed):
    """OpenFOAM lists of a structured block: points i fastest, internal faces by owner then neighbour with the owner's
    outward vertex order, then the boundary faces."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    xs = [_lines(nx, 0.0, case["h"], case["grade"]), _lines(ny, 0.0, case["h"], case["grade"]),
          np.array([-0.5, 0.5]) if case["twod"] else _lines(nz, 0.0, case["h"], 1.0)]
    Z, Y, X = np.meshgrid(xs[2], xs[1], xs[0], indexing="ij")
    pts = np.stack([X, Y, Z], axis=-1).reshape(-1, 3)
    if case["jiggle"]:
        inner = np.zeros((nz + 1, ny + 1, nx + 1), bool)
        inner[1:-1, 1:-1, 1:-1] = True
        rng = np.random.default_rng([int(seed), 23])
        pts += rng.uniform(-1, 1, pts.shape) * case["jiggle"] * case["h"] * inner.reshape(-1, 1)
    k, j, i = (a.reshape(-1) for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    v = lambda a, b, c: (i + a) + (nx + 1) * ((j + b) + (ny + 1) * (k + c))
    H = [v(0, 0, 0), v(1, 0, 0), v(1, 1, 0), v(0, 1, 0), v(0, 0, 1), v(1, 0, 1), v(1, 1, 1), v(0, 1, 1)]
    face = lambda a, b, c, d: np.stack([H[a], H[b], H[c], H[d]], axis=1)
    cell = np.arange(nx * ny * nz)
    up = np.stack([face(1, 2, 6, 5), face(3, 7, 6, 2), face(4, 5, 6, 7)], axis=1)      # x-max, y-max, z-max
    there = np.stack([i + 1 < nx, j + 1 < ny, k + 1 < nz], axis=1)
    nb = np.stack([cell + 1, cell + nx, cell + nx * ny], axis=1)
    own = np.repeat(cell[:, None], 3, axis=1)
    faces, owner, neighbour = [up[there]], [own[there]], nb[there]
    for at, f in ((i == 0, face(0, 4, 7, 3)), (i == nx - 1, up[:, 0]), (j == 0, face(0, 1, 5, 4)),
                  (j == ny - 1, up[:, 1]), (k == 0, face(0, 3, 2, 1)), (k == nz - 1, up[:, 2])):
        faces.append(f[at])
        owner.append(cell[at])
    faces = np.concatenate(faces).astype(np.int32)
    return dict(points=pts, faces=faces, face_off=np.arange(0, 4 * len(faces) + 1, 4, dtype=np.int32),
                owner=np.concatenate(owner).astype(np.int32), neighbour=neighbour.astype(np.int32))


def _poly_box(mesh):
    return mesh["points"].min(axis=0), mesh["points"].max(axis=0)


def _poly_pieces(case, mesh, ex):
    T = lambda a, t=torch.int64: torch.tensor(np.asarray(a), device="cuda", dtype=t)
    pts, faces, owner, nb = T(mesh["points"], F64), T(mesh["faces"]), T(mesh["owner"]), T(mesh["neighbour"])
    N = case["nx"] * case["ny"] * case["nz"]
    C, Sf = _face_geometry(pts[faces])
    # cell -> its six faces, its eight points in ascending order, the slots of each face's points among them
    who, which = torch.cat([owner, nb]), torch.cat([torch.arange(len(owner), device="cuda"),
                                                    torch.arange(len(nb), device="cuda")])
    cf = which[torch.argsort(who, stable=True)].reshape(N, 6)
    labels = faces[cf].reshape(N, 24).sort(dim=1)[0].reshape(N, 8, 3)[:, :, 0]
    slots = (faces[cf][..., None] == labels[:, None, None, :]).to(torch.uint8).argmax(-1)
    # centres and volumes: pyramids about the mean of the face centres
    mean = C[cf].mean(1)
    h3 = ((C[cf] - mean[:, None]) * Sf[cf]).sum(-1).abs()
    V = h3.sum(1) / 3
    cc = ((0.75 * C[cf] + 0.25 * mean[:, None]) * h3[..., None]).sum(1) / h3.sum(1)[:, None]
    for s in range(len(ex.kind)):
        one = lambda n: torch.full((n,), s, dtype=torch.int64, device="cuda")
        ins = ex.inside(one(1), ex.local(one(1), pts[None]))[0]
        cnt = ins[labels].sum(1)
        cell = torch.nonzero(cnt > 0)[:, 0]
        alpha = torch.ones(len(cell), dtype=F64, device="cuda")
        cut = torch.nonzero(cnt[cell] < 8)[:, 0]
        P = pts[labels[cell[cut]]]
        phi = ex.distance(one(len(cut)), ex.local(one(len(cut)), P))
        alpha[cut] = _apex_volume(P, phi, slots[cell[cut]], case["twod"]) / V[cell[cut]]
        yield one(len(cell)), cell, alpha, cc[cell], V[cell][:, None]
