"""What a user of this framework has it do, as timed cases with their 64-bit answers.

Every case goes through the public entry points (the ``EulerCase``, ``NSICase``,
``EulerBatch`` and ``WarmStart`` drivers, and the C ABI under them) on the
procedural meshes of ``graphite_b200.meshgen``:

* ``euler``      a steady Euler solve as the replayed loop, from the free stream or from a saved
                 state, with the final fields, the residual history and the wall force;
* ``polar``      the same mesh at several angles of attack, one solve after another;
* ``percall``    the reference's own loop: one call per stage and iteration, the residual read every
                 time, values and gradients copied to the host at the end;
* ``batch``      many (mesh, Mach, angle) instances advanced together, autotuned;
* ``nsi``        the incompressible model's replayed loop;
* ``train``      training of the warm start's network on a set of fields;
* ``predict``    a predicted initial state for one case;
* ``transport``  a scalar transport model assembled from the generic operators;
* ``reduce``     the sum of an array in device memory;
* ``load``       loading a mesh file (connectivity, numbering, metrics, device layout).

Meshes depend on the sizes of a case alone and are kept as files in the
temporary directory; states, Mach numbers, angles and weights come from the seed.
"""
from __future__ import annotations

import ctypes as C
import json
import math
import os
import tempfile

import numpy as np
import torch

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase
from graphite_b200.warmstart import WarmStart

# the free stream of the reference's examples: p = 1, T = 1 / 1.4 (R = 1), so that the speed of sound is 1
P_INF, T_INF = 1.0, 1.0 / 1.4
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # A small 3-D tet channel, the size that fits a few SMs: launches and latency count.
        dict(name="channel_28800_tets", path="euler", mesh="channel", a=60, b=20, c=4, cells="tet", iters=400,
             start="uniform", transposed=True, density=False, cfl=0.8),
        # The production run: a swept wing of 1.1 million prisms.
        dict(name="wing_1116k", path="euler", mesh="wing", a=160, b=48, c=40, d=32, iters=30, start="uniform",
             transposed=True, density=False, cfl=0.8),
        # A polar on a one-layer airfoil mesh: solve after solve with other conditions on one mesh.
        dict(name="airfoil_120k_polar", path="polar", mesh="airfoil", a=400, b=150, iters=150, angles=3, cfl=0.5),
        # The reference's main loop, stage by stage, on a mid-size wing.
        dict(name="wing_141k_percall", path="percall", mesh="wing", a=80, b=24, c=20, d=16, iters=50,
             transposed=True, cfl=0.8),
        # The parameter sweep: 64 instances on three meshes of uneven sizes.
        dict(name="sweep_64_instances", path="batch", sizes="250x100,400x150,600x250", counts="24,24,16", iters=60,
             cfl=0.5),
        # A handful of conditions on small meshes, where a batch is launch-bound.
        dict(name="batch_10_small", path="batch", sizes="64x36,90x41", counts="6,4", iters=100, cfl=0.5),
        # Incompressible flow past a cylinder on 100k hexes.
        dict(name="cylinder_100k", path="nsi", mesh="cylinder", a=400, b=250, ratio=1.03, iters=300, limited=False,
             corrected=True, cfl=0.8),
        # Six epochs of the warm start's training on 24 fields of the 120k airfoil mesh.
        dict(name="train_24_fields", path="train", mesh="airfoil", a=400, b=150, fields=24, epochs=6, tiles=8),
        # The trained network's initial state for one case.
        dict(name="predict_120k", path="predict", mesh="airfoil", a=400, b=150),
        # A user's own model on a mesh of hexes, prisms and pyramids.
        dict(name="transport_mixed", path="transport", mesh="channel", a=96, b=32, c=8, cells="mixed", iters=50,
             second=True),
        # The reduction alone, on device memory.
        dict(name="reduce_5M", path="reduce", n=5_000_017),
        # Reading a mid-size mesh file.
        dict(name="load_wing_141k", path="load", mesh="wing", a=80, b=24, c=20, d=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_channel(rng):
    nx = _log_int(rng, 9, 120)
    return dict(mesh="channel", a=nx, b=_log_int(rng, 5, 40), c=rng.randint(2, 9),
                cells=rng.choice(["tet", "hex", "prism", "pyramid", "mixed", "layered"]))


def _draw_airfoil(rng, top=300):
    return dict(mesh="airfoil", a=2 * _log_int(rng, 16, top), b=_log_int(rng, 9, 250))


def _draw_wing(rng):
    return dict(mesh="wing", a=4 * rng.randint(8, 28), b=rng.randint(9, 36), c=rng.randint(7, 30), d=rng.randint(5, 22))


def draw(rng):
    path = rng.choice(["euler", "euler", "polar", "percall", "batch", "batch", "nsi", "nsi", "train", "predict",
                       "transport", "reduce", "load"])
    any_mesh = rng.choice([_draw_channel, _draw_airfoil, _draw_wing])(rng)
    if path == "euler":
        return dict(any_mesh, path=path, iters=rng.randint(20, 80), start="saved" if rng.random() < 0.2 else "uniform",
                    transposed=rng.random() < 0.75, density=rng.random() < 0.25, cfl=0.5)
    if path == "polar":
        return dict(_draw_airfoil(rng, 250), path=path, iters=rng.randint(40, 160), angles=rng.randint(2, 4), cfl=0.5)
    if path == "percall":
        return dict(any_mesh, path=path, iters=rng.randint(10, 60), transposed=rng.random() < 0.75, cfl=0.5)
    if path == "batch":
        k = rng.randint(1, 3)
        sizes = ",".join("%dx%d" % (2 * _log_int(rng, 16, 200), _log_int(rng, 9, 120)) for _ in range(k))
        return dict(path=path, sizes=sizes, counts=",".join(str(rng.randint(1, 12)) for _ in range(k)),
                    iters=rng.randint(30, 100), cfl=0.5)
    if path == "nsi":
        return dict(path=path, mesh="cylinder", a=4 * _log_int(rng, 8, 110), b=_log_int(rng, 12, 260),
                    ratio=rng.choice([1.02, 1.03]), iters=rng.randint(40, 200), limited=rng.random() < 0.3,
                    corrected=rng.random() < 0.8, cfl=0.5)
    if path == "train":
        return dict(_draw_airfoil(rng), path=path, fields=rng.randint(3, 24), epochs=rng.randint(1, 6),
                    tiles=rng.choice([4, 8, 16]))
    if path == "predict":
        return dict(_draw_airfoil(rng), path=path)
    if path == "transport":
        return dict(any_mesh, path=path, iters=rng.randint(10, 60), second=rng.random() < 0.5)
    if path == "reduce":
        return dict(path=path, n=_log_int(rng, 100, 8_000_000))
    return dict(any_mesh, path=path)


# ---------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------
def _dir():
    d = os.path.join(tempfile.gettempdir(), "graphite_b200_meshes_%d" % os.getuid())
    os.makedirs(d, exist_ok=True)
    return d


def _mesh_key(case):
    k = case["mesh"]
    if k == "channel":
        return "channel_%dx%dx%d_%s" % (case["a"], case["b"], case["c"], case["cells"])
    if k == "airfoil":
        return "airfoil_%dx%d" % (case["a"], case["b"])
    if k == "cylinder":
        return "cylinder_%dx%d_%g" % (case["a"], case["b"], case["ratio"])
    return "wing_%dx%dx%dx%d" % (case["a"], case["b"], case["c"], case["d"])


def _generate(case):
    k = case["mesh"]
    if k == "channel":
        return meshgen.channel_bump(case["a"], case["b"], case["c"], cells=case["cells"])
    if k == "airfoil":
        return meshgen.airfoil_2d_prisms(case["a"], case["b"])
    if k == "cylinder":
        return meshgen.cylinder_ogrid(case["a"], case["b"], ratio=case["ratio"])
    return meshgen.swept_wing(case["a"], case["b"], case["c"], case["d"])


def _put(path, write):
    tmp = "%s.%d" % (path, os.getpid())
    write(tmp)
    os.replace(tmp, path)


def _files(case):
    """(mesh file, file of the elements, sizes) of the case's mesh, made at its first use."""
    base = os.path.join(_dir(), _mesh_key(case))
    fvm, npz, sizes = base + ".fvm", base + ".npz", base + ".json"
    if not (os.path.exists(fvm) and os.path.exists(npz) and os.path.exists(sizes)):
        em = _generate(case)
        arrays, n_entries = {"nodes": em.nodes.astype(np.float32)}, 0
        for i, (kind, conn) in enumerate(em.blocks):
            arrays["block%d_%d" % (i, kind)] = conn.astype(np.int32)
            n_entries += conn.shape[0] * len(meshgen.LOCAL_FACES[kind])
        for r, (name, lists) in enumerate(em.markers.items()):
            for i, (kind, faces) in enumerate(lists):
                arrays["marker%d_%d_%d_%s" % (r, i, kind, name)] = faces.astype(np.int32)

        def npz_out(p):
            with open(p, "wb") as f:
                np.savez(f, **arrays)

        _put(npz, npz_out)
        su2 = "%s.%d.su2" % (base, os.getpid())
        em.write_su2(su2)
        _put(fvm, lambda p: capi.check(capi.load().cuMeshFromSu2(su2.encode(), p.encode()), "cuMeshFromSu2"))
        os.unlink(su2)
        n, g = em.n_cells, em.n_ghosts

        def sizes_out(p):
            with open(p, "w") as f:
                json.dump({"N": n, "G": g, "E": n_entries, "F": (n_entries + g) // 2}, f)

        _put(sizes, sizes_out)
    with open(sizes) as f:
        return fvm, npz, json.load(f)


_centres = {}


def _cell_centres(case):
    """Node averages of the cells, float32 [N][3]."""
    key = _mesh_key(case)
    if key not in _centres:
        z = np.load(_files(case)[1])
        nodes = z["nodes"]
        _centres.clear()
        _centres[key] = np.concatenate([nodes[z[k]].mean(axis=1) for k in z.files if k.startswith("block")])
    return _centres[key]


# ---------------------------------------------------------------------------
# flow conditions and states
# ---------------------------------------------------------------------------
def _mach(kind, rng):
    """Free-stream Mach vector: what each kind of mesh is run at."""
    if kind == "channel":
        return (float(rng.uniform(0.3, 0.6)), 0.0, 0.0)
    m, a = (rng.uniform(0.75, 0.86), rng.uniform(1.0, 4.0)) if kind == "wing" else (rng.uniform(0.3, 0.8),
                                                                                rng.uniform(-2.0, 6.0))
    return (float(m * math.cos(math.radians(a))), 0.0, float(m * math.sin(math.radians(a))))


def _euler_bcs(kind, mach):
    far = tuple(mach) + (P_INF, T_INF)
    if kind == "channel":
        return [("farfield", "inlet") + far, ("slip", "lower"), ("farfield", "outlet") + far, ("slip", "sides"),
                ("slip", "upper")]
    return [("farfield", "farfield") + far, ("slip", "symmetry" if kind == "wing" else "sides"), ("slip", "wing")]


def _wall(kind):
    return "lower" if kind == "channel" else "wing"


def _saved_state(case, sizes, mach, rng):
    """A smooth flow field around the free stream (rho, rho u, rho E), float32, cells then ghosts."""
    c = _cell_centres(case)
    n = sizes["N"] + sizes["G"]
    s = np.zeros((n, 3), np.float32)
    s[: sizes["N"]] = c / np.sqrt(1.0 + (c * c).sum(axis=1, keepdims=True))
    k = rng.uniform(1.0, 4.0, (5, 3)).astype(np.float32)
    ph = rng.uniform(0.0, 2 * math.pi, 5).astype(np.float32)
    w = np.sin(s @ k.T + ph)
    rho = 1.4 * (1.0 + 0.06 * w[:, 0])
    u = np.float32(mach) + 0.06 * w[:, 1:4]
    p = P_INF * (1.0 + 0.06 * w[:, 4])
    rhoe = p / 0.4 + 0.5 * rho * (u * u).sum(axis=1)
    return rho.astype(np.float32), (rho[:, None] * u).astype(np.float32), rhoe.astype(np.float32)


def _array(pointer, n, owner, ctype=C.c_float):
    """n values at a ctypes pointer as an array that keeps their owner alive."""
    buf = (ctype * n).from_address(C.cast(pointer, C.c_void_p).value)
    buf.owner = owner
    return np.ctypeslib.as_array(buf)


def _view(owner, field, what="value"):
    """A host mirror of a field (value, gradient or limiter), as it is."""
    b = field.contents._cpu.contents
    k = b.elem_size // 4 * (3 if what == "gradient" else 1)
    v = _array(getattr(b, what), b.size * k, owner)
    return v.reshape(b.size, k) if k > 1 else v


def _batch_spec(case, seed):
    sizes = [dict(mesh="airfoil", a=int(s.split("x")[0]), b=int(s.split("x")[1])) for s in case["sizes"].split(",")]
    counts = [int(k) for k in case["counts"].split(",")]
    rng = np.random.default_rng([3, seed])
    inst = [(m, _mach("airfoil", rng)) for m, k in enumerate(counts) for _ in range(k)]
    return sizes, inst


N_PARAMS = 36864


def _weights(rng):
    """Weights of the network as after some training: W1[128][16], W2, W3[128][128], W4[16][128], padding zero."""
    w = []
    for rows, cols, ur, uc, bound in ((128, 16, 128, 8, 8 ** -0.5), (128, 128, 128, 128, 128 ** -0.5),
                                      (128, 128, 128, 128, 128 ** -0.5), (16, 128, 5, 128, 128 ** -0.5)):
        m = np.zeros((rows, cols))
        m[:ur, :uc] = rng.uniform(-bound, bound, (ur, uc))
        w.append(m.reshape(-1))
    return np.concatenate(w).astype(np.float32)


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def prepare(case, seed):
    path = case["path"]
    rng = np.random.default_rng([1, seed])
    s = {"case": case, "lib": capi.load()}
    if path == "reduce":
        g = torch.Generator(device=DEV).manual_seed(seed)
        s["x"] = torch.rand(case["n"], generator=g, device=DEV) ** 2      # squared residuals: not negative
        s["out"] = torch.zeros(1, dtype=torch.float64, device=DEV)
        return s
    if path == "batch":
        sizes, inst = _batch_spec(case, seed)
        s["cases"] = [EulerCase(_files(m)[0]) for m in sizes]
        s["inst"] = inst
        s["batch"] = b = EulerBatch(s["cases"], [(m, _euler_bcs("airfoil", mach)) for m, mach in inst])
        n = [s["cases"][m].n_cells + s["cases"][m].n_ghosts for m, _ in inst]
        s["at"] = np.concatenate([[0], np.cumsum(n)])
        s["out"] = [torch.empty(k * int(s["at"][-1]), pin_memory=True).numpy() for k in (1, 3, 1)]
        for i, (m, mach) in enumerate(inst):
            b.init_uniform(i, mach, P_INF, T_INF)
        b.autotune(case["cfl"], 3)
        return s
    fvm, _, sizes = _files(case)
    s["sizes"] = sizes
    if path == "load":
        s["fvm"], s["mesh"] = fvm.encode(), None
        s["seed"] = seed
        # another seed is another file: the same mesh in other length units
        k = np.float32(rng.uniform(0.5, 2.0))
        own = os.path.join(_dir(), "%s_%d_%d.fvm" % (_mesh_key(case), seed, os.getpid()))
        with open(fvm, "rb") as f:
            data = bytearray(f.read())
        n = int(np.frombuffer(data, np.uint32, 1)[0])
        x = np.frombuffer(data, np.float32, 3 * n, 4)
        x *= k
        with open(own, "wb") as f:
            f.write(data)
        s["fvm"], s["own"] = own.encode(), _Unlink(own)
        return s
    if path == "nsi":
        s["nsi"] = NSICase(fvm)
        s["nu"] = float(1.0 / rng.uniform(20.0, 60.0))
        a = math.radians(rng.uniform(-5.0, 5.0))
        s["u"] = (math.cos(a), 0.0, math.sin(a))
        s["bcs"] = [("wall", "cylinder"), ("inletoutlet", "farfield") + s["u"] + (0.0,), ("slip", "sides")]
        return s
    s["euler"] = c = EulerCase(fvm)
    if path == "polar":
        s["machs"] = [_mach("airfoil", rng) for _ in range(case["angles"])]
        return s
    mach = s["mach"] = _mach(case["mesh"], rng)
    if path in ("euler", "percall"):
        s["bcs"] = _euler_bcs(case["mesh"], mach)
        if case.get("start") == "saved":
            s["state"] = _saved_state(case, sizes, mach, rng)
            c.init(mach, P_INF, T_INF)
        return s
    if path in ("train", "predict"):
        s["ws"] = ws = WarmStart(c, wall="wing", seed=seed)
        s["weights"] = _weights(rng)
        if path == "predict":
            ws.weights = s["weights"]
            ws.set_scales(rng.uniform(0.02, 0.2, 5))
            return s
        for _ in range(case["fields"]):
            m = _mach("airfoil", rng)
            c.set_state(*_saved_state(case, sizes, m, rng))
            ws.add_field(c, m, P_INF, T_INF)
            torch.cuda.synchronize()           # the host mirrors are filled again
        per_step = 128 * torch.cuda.get_device_properties(0).multi_processor_count * case["tiles"]
        tiles = case["fields"] * ((sizes["N"] + 127) // 128) * case["epochs"]
        s["steps"] = (tiles * 128 + per_step - 1) // per_step
        return s
    # transport
    n = sizes["N"] + sizes["G"]
    u, _, _ = _saved_state(case, sizes, mach, rng)
    s["u0"], s["phi0"] = u, (np.float32((0.8, 0.1, 0.05)) + 0.1 * _saved_state(case, sizes, mach, rng)[1])
    s["phi0"] = np.ascontiguousarray(s["phi0"], np.float32)
    s["u"], s["phi"] = s["lib"].FvmFieldNew(4, n, b"u", 1), s["lib"].FvmFieldNew(12, n, b"phi", 0)
    s["r"] = s["lib"].FvmFieldNew(4, n, b"r", 0)
    s["fields"] = _Fields(s["lib"], [s["u"], s["phi"], s["r"]], c)
    capi.set_field_values(s["phi"], s["phi0"])
    capi.check(s["lib"].gbVarCpuToGpu(c.mesh, s["phi"]), "gbVarCpuToGpu")
    s["nu"], s["dt"], s["n_regions"] = 0.002, 1e-4, len(c.regions)
    s["const"] = (0.8, 0.1, float(rng.uniform(0.0, 0.1)))
    s["terms"] = t = (capi.gbFvmTerm * 2)()
    if case["second"]:
        t[0] = capi.gbFvmTerm(8, -1.0, s["u"], None, capi.vec(s["const"]))      # limited second-order convection
    else:
        t[0] = capi.gbFvmTerm(9, -1.0, s["u"], s["phi"], capi.vec(s["const"]))  # convection by a velocity field
    t[1] = capi.gbFvmTerm(0, s["nu"], s["u"], None, capi.vec(s["const"]))       # diffusion
    return s


class _Unlink:
    def __init__(self, path):
        self.path = path

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


class _Fields:
    """Frees fields before the mesh they are on."""

    def __init__(self, lib, fields, case):
        self.lib, self.fields, self.case = lib, fields, case

    def __del__(self):
        for f in self.fields:
            self.lib.FvmFieldFree(f)


class _Mesh:
    def __init__(self, lib, fvm):
        self.lib, self.mesh = lib, lib.cuMeshFromFile(fvm)
        if not self.mesh:
            raise capi.GraphiteError(capi.last_error())

    def __del__(self):
        self.lib.cuMeshFree(self.mesh)


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(s):
    case, lib = s["case"], s["lib"]
    path = case["path"]
    if path == "reduce":
        capi.check(lib.gbReduceSumNoAlloc(s["x"].data_ptr(), case["n"], s["out"].data_ptr(), None),
                   "gbReduceSumNoAlloc")
        return s["out"]
    if path == "load":
        s["mesh"] = None                       # the mesh of the pass before goes first
        m = s["mesh"] = _Mesh(lib, s["fvm"])
        b = m.mesh.contents._cpu.contents
        n, g, f = b.n_cells, b.n_ghosts, b.n_faces

        def arr(p, k, t=C.c_float):
            return _array(p, k, m, t)

        return {"volumes": arr(b.cell_volumes, n + g), "centers": arr(b.cell_centers, 3 * (n + g)),
                "matrices": arr(b.cell_matrices, 9 * n), "areas": arr(b.face_areas, f),
                "face_centers": arr(b.face_centers, 3 * f), "normals": arr(b.face_normals, 3 * f),
                "cell_faces": arr(b.cell_faces, b.cell_faces_starts[n + g], C.c_int),
                "cell_connects": arr(b.cell_connects, b.cell_faces_starts[n + g], C.c_int)}
    if path == "batch":
        b = s["batch"]
        for i, (m, mach) in enumerate(s["inst"]):
            b.init_uniform(i, mach, P_INF, T_INF)
        done, its, ratios, status, hist = b.run(case["cfl"], case["iters"], tolerance=1e-9, history=True)
        r, u, e = s["out"]
        for i in range(b.n):
            k = int(s["at"][i])
            capi.check(lib.gbBatchGetState(b.h, i, r.ctypes.data + 4 * k, u.ctypes.data + 12 * k,
                                           e.ctypes.data + 4 * k), "gbBatchGetState")
        force = np.stack([b.wall_force(i, "wing") for i in range(b.n)])
        return {"rho": r, "rhou": u, "rhoe": e, "history": hist, "ratios": ratios, "force": force, "iterations": its,
                "status": status}
    if path == "nsi":
        c = s["nsi"]
        c.set_constants(1.0, s["nu"], 2.0, case["corrected"], case["limited"])
        c.init(s["u"], 0.0)
        hist = c.run(s["bcs"], case["cfl"], case["iters"], tolerance=1e-12)
        force = c.wall_force("cylinder")
        lib.VarGpuToCpu(c.velocity)
        lib.VarGpuToCpu(c.pressure)
        return {"velocity": _view(c, c.velocity), "pressure": _view(c, c.pressure), "history": hist, "force": force}
    c = s["euler"]
    if path == "transport":
        capi.set_field_values(s["u"], s["u0"])
        capi.check(lib.gbVarCpuToGpu(c.mesh, s["u"]), "gbVarCpuToGpu")
        for _ in range(case["iters"]):
            for r in range(s["n_regions"]):
                capi.check(lib.gbFieldBcZeroGrad(c.mesh, s["u"], r), "gbFieldBcZeroGrad")
            capi.check(lib.gbFvmGradient(c.mesh, s["u"]), "gbFvmGradient")
            capi.check(lib.gbFvmApplyTerms(c.mesh, 2, s["terms"], s["r"]), "gbFvmApplyTerms")
            capi.check(lib.gbFieldAxpy(c.mesh, s["u"], s["dt"], s["r"]), "gbFieldAxpy")
        lib.VarGpuToCpu(s["u"])
        return _view(s["fields"], s["u"])
    if path == "train":
        ws = s["ws"]
        ws.weights = s["weights"]
        steps, hist = ws.train(case["epochs"], case["tiles"], 1e-3, history=s["steps"])
        return {"weights": ws.weights, "loss": hist}
    if path == "predict":
        s["ws"].predict(c, s["mach"], P_INF, T_INF)
        c.download_mirrors()
        n = c.n_cells
        return {"rho": _view(c, c.rho)[:n], "rhou": _view(c, c.rhou)[:n], "rhoe": _view(c, c.rhoe)[:n]}
    lib.gbSetReferenceMomentumReconstruction(1 if case.get("transposed", True) else 0)
    if path == "polar":
        hists, forces = [], []
        for mach in s["machs"]:
            c.init(mach, P_INF, T_INF)
            hists.append(c.run(_euler_bcs("airfoil", mach), case["cfl"], case["iters"], tolerance=1e-9))
            forces.append(c.wall_force("wing"))
        c.download_mirrors()
        return {"history": np.stack(hists), "force": np.stack(forces), "rho": _view(c, c.rho), "rhou": _view(c, c.rhou),
                "rhoe": _view(c, c.rhoe)}
    if path == "percall":
        c.init(s["mach"], P_INF, T_INF)
        hist = [c.iterate(s["bcs"], case["cfl"]) for _ in range(case["iters"])]
        out = {"history": np.array(hist, np.float32)}
        for name, f in (("rho", c.rho), ("rhou", c.rhou), ("rhoe", c.rhoe)):
            lib.VarAllGpuToCpu(f)
            out[name] = _view(c, f)
            out["grad_" + name], out["lim_" + name] = _view(c, f, "gradient"), _view(c, f, "limiter")
        return out
    if "state" in s:
        for f, v in zip((c.rho, c.rhou, c.rhoe), s["state"]):
            _view(c, f)[...] = v
        c.upload_mirrors()
    else:
        c.init(s["mach"], P_INF, T_INF)
    out = {}
    if case["density"]:
        out["history"], out["density"] = c.run_density(s["bcs"], case["cfl"], case["iters"], tolerance=1e-9)
    else:
        out["history"] = c.run(s["bcs"], case["cfl"], case["iters"], tolerance=1e-9)
    out["force"] = c.wall_force(_wall(case["mesh"]))
    c.download_mirrors()
    return dict(out, rho=_view(c, c.rho), rhou=_view(c, c.rhou), rhoe=_view(c, c.rhoe))


# ---------------------------------------------------------------------------
# work: per iteration the state once in and once out and the mesh once (per cell centroid, volume and the symmetric
# least-squares inverse; per face normal, area and centre; per entry of a cell its face and neighbour)
# ---------------------------------------------------------------------------
def _sweep_work(z, comps, flops):
    return {"bytes": 8 * comps * z["N"] + 4 * (4 + 6) * z["N"] + 28 * z["F"] + 8 * z["E"] + 16 * z["G"],
            "flops": flops * z["E"]}


def work(case):
    path = case["path"]
    if path == "reduce":
        return {"bytes": 4 * case["n"], "flops": case["n"]}
    if path == "batch":
        sizes, inst = _batch_spec(case, 0)
        z = [_files(m)[2] for m in sizes]
        per = {"bytes": 0, "flops": 0}
        for k, n in enumerate(int(x) for x in case["counts"].split(",")):
            per["flops"] += n * 220 * z[k]["E"]
            per["bytes"] += n * 40 * z[k]["N"] + _sweep_work(z[k], 0, 0)["bytes"]
        out = sum(20 * (z[m]["N"] + z[m]["G"]) for m, _ in inst)
        return {"bytes": case["iters"] * per["bytes"] + out, "flops": case["iters"] * per["flops"]}
    z = _files(case)[2]
    n = z["N"] + z["G"]
    if path == "load":
        read = os.path.getsize(_files(case)[0])
        return {"bytes": read + 4 * (16 * n + 9 * z["N"] + 7 * z["F"] + 2 * (z["E"] + z["G"])), "flops": 400 * z["E"]}
    if path in ("euler", "percall"):
        w = _sweep_work(z, 5, 220)
        return {"bytes": case["iters"] * w["bytes"] + 20 * n, "flops": case["iters"] * w["flops"]}
    if path == "polar":
        w = _sweep_work(z, 5, 220)
        return {"bytes": case["angles"] * case["iters"] * w["bytes"] + 20 * n,
                "flops": case["angles"] * case["iters"] * w["flops"]}
    if path == "nsi":
        w = _sweep_work(z, 4, 200)
        return {"bytes": case["iters"] * w["bytes"] + 16 * n, "flops": case["iters"] * w["flops"]}
    if path == "transport":
        w = _sweep_work(z, 1, 50)
        return {"bytes": case["iters"] * w["bytes"] + 4 * n, "flops": case["iters"] * w["flops"]}
    mac = 8 * 128 + 2 * 128 * 128 + 128 * 5                       # multiply-adds of one sample, forward
    if path == "predict":
        return {"bytes": 36 * z["N"] + 2 * N_PARAMS, "flops": 2 * mac * z["N"]}
    samples = case["fields"] * case["epochs"] * z["N"]
    return {"bytes": samples * 36, "flops": 6 * mac * samples}     # forward, data and weight gradients


# ---------------------------------------------------------------------------
# exact: the same in float64, in plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    path = case["path"]
    rng = np.random.default_rng([1, seed])
    if path == "reduce":
        g = torch.Generator(device=DEV).manual_seed(seed)
        x = torch.rand(case["n"], generator=g, device=DEV) ** 2
        return x.double().sum().reshape(1)
    if path == "train":
        return None
    if path == "batch":
        sizes, inst = _batch_spec(case, seed)
        if sum(m["a"] * m["b"] for m in sizes) * len(inst) * case["iters"] > 5e7:
            return None
        flows = [_Geometry(m) for m in sizes]
        out = []
        for m, mach in inst:
            q = _Euler(flows[m], True)
            q.init(mach)
            h = [q.iterate(_euler_bcs("airfoil", mach), case["cfl"])[0] for _ in range(case["iters"])]
            out.append((q.q[:, 0], q.q[:, 1:4].reshape(-1), q.q[:, 4], torch.stack(h), q.force("wing")))
        rho, rhou, rhoe = (torch.cat([o[k] for o in out]) for k in range(3))
        hist = torch.stack([o[3] for o in out])
        return {"rho": rho, "rhou": rhou, "rhoe": rhoe, "history": hist, "ratios": hist[:, -1] / hist[:, 0],
                "force": torch.stack([o[4] for o in out]), "iterations": None, "status": None}
    if path == "load":
        m = _Geometry(case, float(np.float32(rng.uniform(0.5, 2.0))))
        return {"volumes": torch.cat([m.vol, m.gvol]), "centers": m.cc.reshape(-1), "matrices": m.lsq.reshape(-1),
                "areas": None, "face_centers": None, "normals": None, "cell_faces": None, "cell_connects": None}
    geo = _Geometry(case)
    sizes = _files(case)[2]
    if path == "nsi":
        nu = float(np.float32(1.0 / rng.uniform(20.0, 60.0)))
        a = math.radians(rng.uniform(-5.0, 5.0))
        u = tuple(float(np.float32(x)) for x in (math.cos(a), 0.0, math.sin(a)))
        return _nsi64(geo, case, nu, u)
    if path == "polar":
        machs = [_mach("airfoil", rng) for _ in range(case["angles"])]
        hists, forces, q = [], [], _Euler(geo, True)
        for mach in machs:
            q.init(mach)
            hists.append(torch.stack([q.iterate(_euler_bcs("airfoil", mach), case["cfl"])[0]
                                      for _ in range(case["iters"])]))
            forces.append(q.force("wing"))
        return {"history": torch.stack(hists), "force": torch.stack(forces), "rho": q.q[:, 0], "rhou": q.q[:, 1:4],
                "rhoe": q.q[:, 4]}
    mach = _mach(case["mesh"], rng)
    if path in ("euler", "percall"):
        q = _Euler(geo, case["transposed"])
        if case.get("start") == "saved":
            r, u, e = (torch.from_numpy(x).to(DEV).double() for x in _saved_state(case, sizes, mach, rng))
            q.q = torch.cat([r[:, None], u, e[:, None]], 1)
        else:
            q.init(mach)
        bcs = _euler_bcs(case["mesh"], mach)
        h = [q.iterate(bcs, case["cfl"]) for _ in range(case["iters"])]
        out = {"rho": q.q[:, 0], "rhou": q.q[:, 1:4], "rhoe": q.q[:, 4], "history": torch.stack([x[0] for x in h])}
        if path == "euler":
            out["force"] = q.force(_wall(case["mesh"]))
            if case["density"]:
                out["density"] = torch.stack([x[1] for x in h])
            return out
        g = torch.cat([q.g, q.g[geo.gcell]])
        lim = torch.cat([q.lim, q.lim[geo.gcell]])
        return dict(out, grad_rho=g[:, 0], lim_rho=lim[:, 0], grad_rhou=g[:, 1:4].reshape(-1, 9), lim_rhou=lim[:, 1:4],
                    grad_rhoe=g[:, 4], lim_rhoe=lim[:, 4])
    if path == "predict":
        w = torch.from_numpy(_weights(rng)).to(DEV).double()
        scale = torch.from_numpy(rng.uniform(0.02, 0.2, 5).astype(np.float32)).to(DEV).double()
        return _predict64(geo, w, scale, mach)
    u0, _, _ = _saved_state(case, sizes, mach, rng)
    phi0 = np.float32((0.8, 0.1, 0.05)) + 0.1 * _saved_state(case, sizes, mach, rng)[1]
    phi0 = np.ascontiguousarray(phi0, np.float32)
    const = torch.tensor(np.float32((0.8, 0.1, float(rng.uniform(0.0, 0.1))))).to(DEV).double()
    return _transport64(geo, case, torch.from_numpy(u0).to(DEV).double(), torch.from_numpy(phi0).to(DEV).double(), const)


def _f32(x):
    return float(np.float32(x))


def _dot(a, b):
    return (a * b).sum(-1)


class _Geometry:
    """A mesh in float64: entries [N][M] (M the most faces of a cell, absent ones masked out) with their neighbour,
    outward normal, area / volume, offsets of the neighbour and of the face centre."""

    def __init__(self, case, scale=None):
        z = np.load(_files(case)[1])
        x = z["nodes"] if scale is None else z["nodes"] * np.float32(scale)
        x = torch.from_numpy(x).to(DEV).double()
        blocks = [(int(k.rsplit("_", 1)[1]), torch.from_numpy(z[k]).to(DEV).long()) for k in z.files
                  if k.startswith("block")]
        n = self.n = sum(c.shape[0] for _, c in blocks)
        m = max(len(meshgen.LOCAL_FACES[k]) for k, _ in blocks)
        fn = torch.full((n, m, 4), -1, dtype=torch.long, device=DEV)     # nodes of each entry's face
        at = 0
        for kind, conn in blocks:
            for t, lf in enumerate(meshgen.LOCAL_FACES[kind]):
                fn[at:at + conn.shape[0], t, :len(lf)] = conn[:, list(lf)]
            at += conn.shape[0]
        self.mask = mask = fn[:, :, 0] >= 0

        def key(f):                            # the three smallest nodes name a face
            f = torch.where(f < 0, torch.full_like(f, 1 << 20), f).sort(-1)[0]
            return (f[..., 0] << 42) | (f[..., 1] << 21) | f[..., 2]

        flat = mask.reshape(-1).nonzero()[:, 0]
        keys, order = key(fn).reshape(-1)[flat].sort()
        entry = flat[order]
        nb = torch.full((n * m,), -1, dtype=torch.long, device=DEV)
        same = (keys[1:] == keys[:-1]).nonzero()[:, 0]
        nb[entry[same]] = entry[same + 1] // m
        nb[entry[same + 1]] = entry[same] // m
        self.regions, g, gent = {}, 0, []
        for k in (k for k in z.files if k.startswith("marker")):
            f = torch.from_numpy(z[k]).to(DEV).long()
            if f.shape[1] == 3:
                f = torch.cat([f, torch.full_like(f[:, :1], -1)], 1)
            e = entry[torch.searchsorted(keys, key(f))]
            name = k.split("_", 3)[3]
            a, b = self.regions.get(name, (g, g))
            self.regions[name] = (a, g + f.shape[0])
            nb[e] = n + g + torch.arange(f.shape[0], device=DEV)
            g += f.shape[0]
            gent.append(e)
        gent = self.gent = torch.cat(gent)
        self.gcell = gent // m
        self.nb = nb.reshape(n, m)
        # faces: fan around the node average
        has = (fn >= 0)[..., None].double()
        p = x[fn.clamp_min(0)]
        self.points = p.reshape(n * m, 4, 3)
        c = (p * has).sum(2) / has.sum(2).clamp_min(1)
        cnt = has[..., 0].sum(2).long()
        nxt = torch.arange(1, 5, device=DEV).expand(n, m, 4)
        nxt = torch.where(nxt >= cnt[..., None], torch.zeros_like(nxt), nxt)
        p1 = p.gather(2, nxt[..., None].expand(-1, -1, -1, 3))
        cr = torch.cross(c[:, :, None] - p, c[:, :, None] - p1, dim=-1) * has
        h = cr.norm(dim=-1) * 0.5
        area = h.sum(2)
        nsum = cr.sum(2)
        fc = ((p + p1 + c[:, :, None]) * (h / 3.0)[..., None]).sum(2) / area.clamp_min(1e-300)[..., None]
        nrm = nsum / nsum.norm(dim=-1, keepdim=True).clamp_min(1e-300)
        area = area * mask
        c0 = (fc * area[..., None]).sum(1) / area.sum(1)[:, None]
        d = fc - c0[:, None]
        w = d.norm(dim=-1) * area
        c1 = ((c0[:, None] + d * 0.75) * w[..., None]).sum(1) / w.sum(1)[:, None]
        d = fc - c1[:, None]
        sgn = torch.where(_dot(nrm, d) >= 0, 1.0, -1.0)
        self.nrm = nrm * sgn[..., None]
        self.vol = (_dot(d, self.nrm) * area).sum(1) / 3.0
        gd = (fc - c1[:, None]).reshape(-1, 3)[gent]
        gn, gfc = self.nrm.reshape(-1, 3)[gent], fc.reshape(-1, 3)[gent]
        dx = gd.norm(dim=-1)
        self.gvol = area.reshape(-1)[gent] * 2.0 * dx
        self.cc = torch.cat([c1, gfc + gn * dx[:, None]])
        self.gn, self.garea = gn, area.reshape(-1)[gent]
        self.fc, self.area = fc, area
        self.nbi = torch.where(mask, self.nb, torch.zeros_like(self.nb))
        self.dn = (self.cc[self.nbi] - c1[:, None]) * mask[..., None]
        self.w = torch.where(mask, 1.0 / _dot(self.dn, self.dn).clamp_min(1e-300), torch.zeros_like(area))
        self.df = (fc - c1[:, None]) * mask[..., None]
        self.k3 = self.df.norm(dim=-1) ** 3
        self.lsq = torch.linalg.inv((self.dn[..., :, None] * self.dn[..., None, :] * self.w[..., None, None]).sum(1))
        self.lsq = 0.5 * (self.lsq + self.lsq.transpose(1, 2))
        self.ds = area / self.vol[:, None]
        # the neighbour's side: its offset to the face centre and the owner of its gradient
        self.own = torch.where(self.nbi >= n, torch.arange(n, device=DEV)[:, None].expand_as(self.nbi), self.nbi)
        self.df1 = (fc - self.cc[self.nbi]) * mask[..., None]

    def gradients(self, q, limited=True):
        """Gradients [N][k][3] and limiters [N][k] of the columns of q [N+G][k]."""
        n = self.n
        dq = (q[self.nbi] - q[:n, None]) * self.mask[..., None]
        g = torch.einsum("nmk,nmd,nm->nkd", dq, self.dn, self.w)
        g = torch.einsum("nde,nke->nkd", self.lsq, g)
        if not limited:
            return g, torch.ones_like(g[..., 0])
        du = dq.amax(1).clamp_min(0.0)
        dd = dq.amin(1).clamp_max(0.0)
        out = torch.full_like(du, 2.0)
        dmm2 = (du - dd) ** 2
        for t in range(self.nb.shape[1]):
            k3 = self.k3[:, t, None]
            delta = torch.einsum("nkd,nd->nk", g, self.df[:, t])
            y = dmm2 / k3 - 1.0
            sig = torch.where(dmm2 <= k3, 1.0, torch.where(dmm2 <= 2.0 * k3, 2 * y ** 3 - 3 * y ** 2 + 1.0, 0.0))
            r = torch.where(delta > 0, du, dd) / torch.where(delta.abs() > 1e-6, delta, 1.0)
            lim = torch.where((delta.abs() > 1e-6) & (r < 2.0), r - 0.25 * r * r, 1.0) * 0.8
            lim = torch.where(sig == 1.0, 1.0, sig + (1.0 - sig) * lim)
            out = torch.where(self.mask[:, t, None], torch.minimum(out, lim), out)
        return g, out


def _lsqrt(x):
    return x.clamp(1e-12, 1e30).sqrt()


class _Euler:
    """The explicit second-order Euler iteration on a _Geometry."""

    def __init__(self, geo, transposed):
        self.m, self.transposed = geo, transposed

    def init(self, mach):
        mach = torch.tensor([_f32(x) for x in mach], dtype=torch.float64, device=DEV)
        p, t = P_INF, _f32(T_INF)
        r = p / t
        v = mach * math.sqrt(1.4 * p / r)
        q = torch.cat([torch.full((1,), r, dtype=torch.float64, device=DEV), r * v,
                       (p / 0.4 + 0.5 * r * _dot(v, v)).reshape(1)])
        self.q = q.expand(self.m.cc.shape[0], 5).clone()

    def ghosts(self, bcs):
        m = self.m
        for bc in bcs:
            a, b = m.regions[bc[1]]
            i, nrm = m.gcell[a:b], m.gn[a:b]
            q = self.q[i]
            r, u, e = q[:, 0], q[:, 1:4], q[:, 4]
            if bc[0] == "slip":
                g = torch.cat([r[:, None], u - 2.0 * _dot(nrm, u)[:, None] * nrm, e[:, None]], 1)
            else:
                im = torch.tensor([_f32(x) for x in bc[2:5]], dtype=torch.float64, device=DEV)
                ip, it = _f32(bc[5]), _f32(bc[6])
                v = u / r[:, None]
                p = 0.4 * (e - 0.5 / r * _dot(u, u))
                mach = (_dot(v, v) / (1.4 * p / r)).sqrt()
                inflow = _dot(v, nrm) < 0

                def state(rr, vv, pp):
                    rr, pp = rr.expand_as(r), pp.expand_as(r)
                    vv = vv.expand_as(v)
                    return torch.cat([rr[:, None], rr[:, None] * vv,
                                      (pp / 0.4 + 0.5 * rr * _dot(vv, vv))[:, None]], 1)

                one = torch.ones_like(r)
                idens = ip / it
                sup = state(idens * one, im * math.sqrt(1.4 * ip / idens) * one[:, None], ip * one)
                rs = p / it
                sub = state(rs, im * (1.4 * p / rs).sqrt()[:, None], p)
                outs = state(ip / (p / r), v, ip * one)
                g = torch.where(inflow[:, None], torch.where((mach > 1)[:, None], sup, sub),
                                torch.where((mach > 1)[:, None], q, outs))
            self.q[m.n + a:m.n + b] = g

    def iterate(self, bcs, cfl):
        """One iteration; (sum of the squared residuals, its density part)."""
        m, n, cfl = self.m, self.m.n, _f32(cfl)
        self.ghosts(bcs)
        q = self.q
        g, lim = self.g, self.lim = m.gradients(q)
        gt = g
        if self.transposed:
            gt = g.clone()
            gt[:, 1:4] = g[:, 1:4].transpose(1, 2)
        f = torch.zeros(n, 5, dtype=torch.float64, device=DEV)
        dts = torch.zeros(n, dtype=torch.float64, device=DEV)
        for t in range(m.nb.shape[1]):
            o, ds, nrm = m.own[:, t], m.ds[:, t], m.nrm[:, t]
            qa = q[:n] + torch.einsum("nkd,nd->nk", gt, m.df[:, t]) * lim
            qb = q[m.nbi[:, t]] + torch.einsum("nkd,nd->nk", gt[o], m.df1[:, t]) * lim[o]
            fl, sp = 0.0, []
            for s in (qa, qb):
                r, u, e = s[:, 0], s[:, 1:4], s[:, 4]
                uu = _dot(u, u)
                p = 0.4 * (e - 0.5 * uu / r)
                v = _dot(u, nrm) / r
                fl = fl + torch.cat([(v * r)[:, None], u * v[:, None] + nrm * p[:, None], (v * (e + p))[:, None]], 1)
                sp.append(uu.sqrt() / r + _lsqrt(1.4 * p / r))
            eig = torch.maximum(*sp)
            ok = m.mask[:, t]
            f += torch.where(ok[:, None], (fl - (qb - qa) * eig[:, None]) * (0.5 * ds)[:, None], 0.0)
            dts += torch.where(ok, eig * ds, 0.0)
        new = q.clone()
        new[:n] = q[:n] - f * (cfl / dts)[:, None]
        self.q = new
        return (f.square().sum(1) * m.vol).sum(), (f[:, 0].square() * m.vol).sum()

    def force(self, region):
        a, b = self.m.regions[region]
        q = self.q[self.m.gcell[a:b]]
        p = 0.4 * (q[:, 4] - 0.5 * _dot(q[:, 1:4], q[:, 1:4]) / q[:, 0])
        return ((p * self.m.garea[a:b])[:, None] * self.m.gn[a:b]).sum(0)


def _nsi64(m, case, nu, u_inf):
    """Artificial compressibility (beta = 2) in float64."""
    n, beta2, cfl = m.n, 4.0, _f32(case["cfl"])
    ui = torch.tensor(u_inf, dtype=torch.float64, device=DEV)
    q = torch.cat([torch.zeros(1, dtype=torch.float64, device=DEV), ui]).expand(m.cc.shape[0], 4).clone()
    hist = []

    def ghosts(q):
        for name, (a, b) in m.regions.items():
            i, nrm = m.gcell[a:b], m.gn[a:b]
            p, u = q[i, 0], q[i, 1:4]
            if name == "cylinder":
                g = torch.cat([p[:, None], -u], 1)
            elif name == "sides":
                g = torch.cat([p[:, None], u - 2.0 * _dot(nrm, u)[:, None] * nrm], 1)
            else:
                inflow = (_dot(ui.expand_as(nrm), nrm) < 0)[:, None]
                g = torch.where(inflow, torch.cat([p[:, None], ui.expand_as(u)], 1),
                                torch.cat([torch.zeros_like(p)[:, None], u], 1))
            q[n + a:n + b] = g

    def face_gradient(ga, du, d, w, nrm):
        gn = torch.einsum("nkd,nd->nk", ga, nrm)
        if case["corrected"]:
            gn = gn + (du - torch.einsum("nkd,nd->nk", ga, d)) * (w * _dot(d, nrm))[:, None]
        return gn

    for _ in range(case["iters"]):
        ghosts(q)
        g, lim = m.gradients(q, case["limited"])
        r = torch.zeros(n, 4, dtype=torch.float64, device=DEV)
        sr = torch.zeros(n, dtype=torch.float64, device=DEV)
        for t in range(m.nb.shape[1]):
            o, ds, nrm, j = m.own[:, t], m.ds[:, t], m.nrm[:, t], m.nbi[:, t]
            qa = q[:n] + torch.einsum("nkd,nd->nk", g, m.df[:, t]) * lim
            qb = q[j] + torch.einsum("nkd,nd->nk", g[o], m.df1[:, t]) * lim[o]
            ua, ub = _dot(qa[:, 1:4], nrm), _dot(qb[:, 1:4], nrm)
            lam = torch.maximum(ua.abs() + (ua * ua + beta2).sqrt(), ub.abs() + (ub * ub + beta2).sqrt())
            fl = torch.cat([(beta2 * (ua + ub))[:, None], qa[:, 1:4] * ua[:, None] + nrm * qa[:, :1] +
                            qb[:, 1:4] * ub[:, None] + nrm * qb[:, :1]], 1)
            fl = (fl - lam[:, None] * (qb - qa)) * (0.5 * ds)[:, None]
            ga = 0.5 * (g[:, 1:4] + g[o][:, 1:4])
            vis = face_gradient(ga, q[j, 1:4] - q[:n, 1:4], m.dn[:, t], m.w[:, t], nrm)
            fl[:, 1:4] -= vis * (nu * ds)[:, None]
            ok = m.mask[:, t]
            r += torch.where(ok[:, None], fl, 0.0)
            sr += torch.where(ok, (lam + 2.0 * nu * m.w[:, t].sqrt()) * ds, 0.0)
        hist.append((r.square().sum(1) * m.vol).sum())
        q = q.clone()
        q[:n] = q[:n] - r * (cfl / sr)[:, None]
    # force of the current state; its ghosts are those of the last iteration
    a, b = m.regions["cylinder"]
    i, nrm = m.gcell[a:b], m.gn[a:b]
    g = m.gradients(q, False)[0][i, 1:4]
    d = m.cc[n + a:n + b] - m.cc[i]
    gq = q[n + a:n + b]
    vis = face_gradient(g, gq[:, 1:4] - q[i, 1:4], d, 1.0 / _dot(d, d), nrm)
    pf = 0.5 * (q[i, 0] + gq[:, 0])
    force = (m.garea[a:b][:, None] * (pf[:, None] * nrm - nu * vis)).sum(0)
    return {"velocity": q[:, 1:4], "pressure": q[:, 0], "history": torch.stack(hist), "force": force}


def _transport64(m, case, u, phi, const):
    n, nu, dt = m.n, _f32(0.002), _f32(1e-4)
    for _ in range(case["iters"]):
        u = u.clone()
        u[n:] = u[m.gcell]
        g, lim = m.gradients(u[:, None])
        g, lim = g[:, 0], lim[:, 0]
        r = torch.zeros(n, dtype=torch.float64, device=DEV)
        for t in range(m.nb.shape[1]):
            o, ds, nrm, j = m.own[:, t], m.ds[:, t], m.nrm[:, t], m.nbi[:, t]
            a, b = u[:n], u[j]
            if case["second"]:
                a = a + _dot(g, m.df[:, t]) * lim
                b = b + _dot(g[o], m.df1[:, t]) * lim[o]
                an = bn = _dot(nrm, const)
            else:
                an, bn = _dot(nrm, phi[:n]), _dot(nrm, phi[j])
            conv = (an * a + bn * b - torch.maximum(an.abs(), bn.abs()) * (b - a)) * 0.5 * ds
            lap = _dot(g + g[o], nrm) * 0.5 * ds
            r += torch.where(m.mask[:, t], nu * lap - conv, 0.0)
        u[:n] += dt * r
    return u


def _predict64(m, w, scale, mach):
    """The network on every cell: the wall is the airfoil's contour extruded along y, the cells are at mid-span."""
    mv = torch.tensor([_f32(x) for x in mach], dtype=torch.float64, device=DEV)
    x = m.cc[:m.n]
    a, b = m.regions["wing"]
    pts = m.points[m.gent[a:b]]                                    # [faces][4][3]
    lo, hi = pts.reshape(-1, 3).amin(0), pts.reshape(-1, 3).amax(0)
    centre, length = pts.mean(1).mean(0), (hi - lo).amax()
    # each quad's two ends in the x-z plane
    first = pts[:, 0]
    far = (pts[:, :, ::2] - first[:, None, ::2]).norm(dim=-1).argmax(1)
    p0 = first[:, ::2]
    p1 = pts[torch.arange(pts.shape[0], device=DEV), far][:, ::2]
    best = torch.full((m.n,), 1e300, dtype=torch.float64, device=DEV)
    for k in range(0, p0.shape[0], 64):
        s, e = p0[k:k + 64], p1[k:k + 64] - p0[k:k + 64]
        v = x[:, None, ::2] - s
        t = (_dot(v, e) / _dot(e, e)).clamp(0.0, 1.0)
        best = torch.minimum(best, (v - t[..., None] * e).square().sum(-1).amin(1))

    def squash(u):
        return u / (1.0 + u * u).sqrt()

    speed = mv.norm()
    par = torch.stack([speed, mv[2] / speed, mv[0] / speed, torch.ones_like(speed)]).expand(m.n, 4)
    f = torch.cat([squash((x - centre) / length), squash(best.sqrt() / length)[:, None], par], 1)
    w1, w2, w3, w4 = (t.reshape(r, c) for t, (r, c) in zip(w.split([2048, 16384, 16384, 2048]),
                                                         ((128, 16), (128, 128), (128, 128), (16, 128))))
    act = torch.nn.functional.silu
    y = act(act(act(f @ w1[:, :8].T) @ w2.T) @ w3.T) @ w4[:5].T
    q = _Euler(m, True)
    q.init(mach)
    out = q.q[:m.n] + scale * y
    return {"rho": out[:, 0], "rhou": out[:, 1:4], "rhoe": out[:, 4]}
