"""Work that users of redynela_gb300 have it do, as cases for timing and for comparing outputs.

Every case goes through the public entry points (``GpuDomain``, ``BatchDomain`` and the C ABI of
``include/dnl_gpu.h``).  Meshes are the repository's own generators (Taylor bars of quads,
hexahedra and tetrahedra, the two-material bar, batches of uneven bars) with every node moved a
few per cent of a cell by the seed, as meshes of real parts are not perfect grids; materials and
speeds are drawn from the ranges of ``meshes.taylor_batch``.

kinds:

* ``study``    a parameter study's evaluation: the handle back to its initial state, the first
               steps of an impact, the final state to the host
* ``forces``   the drop-in of Domain::computeInternalForces on host arrays
* ``static``   the same without a handle, on device arrays of the caller
* ``step``     explicit steps in the middle of an impact, then an output frame
* ``host``     one step for a host program that owns the nodal state
* ``batch``    many uneven bars advanced together
* ``tangent``  a run with its derivatives (forward mode)
* ``gradient`` a loss gradient (reverse mode)
"""

from __future__ import annotations

import ctypes as C
import dataclasses
import math

import numpy as np
import torch

from redynela_gb300 import dynela, meshes

AXI, HEX, PLANE, TET4, TET10, HEX1 = (meshes.ELQUA4NAX, meshes.ELHEX8N3D, meshes.ELQUA4N2D,
                                      meshes.ELTET4N3D, meshes.ELTET10N3D, meshes.ELHEX8N3D_1PT)
NAMES = {"axi": AXI, "hex": HEX, "plane": PLANE, "tet4": TET4, "tet10": TET10, "hex1pt": HEX1}


def listed():
    return [
        # the sample deck's own mesh (5 x 50), the smallest real one: launches and latency
        {"name": "study axi 5x50", "kind": "study", "elem": "axi", "nr": 5, "nz": 50, "steps": 200},
        # a host code (the reference's strategies) that calls the force pass each step, plane strain
        {"name": "forces plane 17x163", "kind": "forces", "elem": "plane", "nr": 17, "nz": 163, "steps": 1},
        # a caller with its own device memory, near the entry's largest mesh
        {"name": "static hex 24x97", "kind": "static", "elem": "hex", "nr": 24, "nz": 97, "steps": 1},
        # two bonded materials, one with a tabulated hardening law (Samples/Traction's pattern)
        {"name": "study two materials 20x200", "kind": "study", "elem": "axi", "law": "table", "nr": 20, "nz": 200, "steps": 40},
        # a fine axisymmetric bar
        {"name": "step axi 40x400", "kind": "step", "elem": "axi", "nr": 40, "nz": 400, "steps": 40},
        # tetrahedra (what a mesher gives for a real part)
        {"name": "step tet4 9x41", "kind": "step", "elem": "tet4", "nr": 9, "nz": 41, "steps": 20},
        # the one-point hexahedron with hourglass control
        {"name": "step hex1pt 32x256", "kind": "step", "elem": "hex1pt", "nr": 32, "nz": 256, "steps": 10},
        # a medium 3D bar with the Pulse time step
        {"name": "step hex 15x121", "kind": "step", "elem": "hex", "nr": 15, "nz": 121, "steps": 10},
        # the benchmark's 3D bar, 505,600 hexahedra: the largest
        {"name": "step hex 40x400", "kind": "step", "elem": "hex", "nr": 40, "nz": 400, "steps": 10},
        # a host program that keeps the nodal state, one step a call
        {"name": "host hex 16x100", "kind": "host", "elem": "hex", "nr": 16, "nz": 100, "steps": 1},
        # a calibration over many specimens
        {"name": "batch 32 bars", "kind": "batch", "elem": "axi", "nr": 24, "nz": 240, "count": 32, "steps": 20},
        # parameter identification on the 20 x 200 bar (the repository's gradient workload)
        {"name": "gradient axi 20x200", "kind": "gradient", "elem": "axi", "nr": 20, "nz": 200, "steps": 150},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["study", "forces", "static", "step", "step", "step", "host", "batch", "tangent", "gradient"])
    if kind == "study":
        c = {"kind": kind, "elem": rng.choice(["axi", "plane"]), "nr": _log(rng, 4, 24), "nz": _log(rng, 30, 240), "steps": _log(rng, 40, 300)}
        return dict(c, law="table") if c["elem"] == "axi" and rng.random() < 0.4 else c
    if kind == "forces":
        e = rng.choice(["axi", "plane", "hex", "tet4"])
        two = e in ("axi", "plane")
        return {"kind": kind, "elem": e, "nr": _log(rng, 5, 40 if two else 13), "nz": _log(rng, 50, 400) if two else _log(rng, 10, 60), "steps": 1}
    if kind == "static":
        e = rng.choice(["axi", "plane", "hex", "tet4", "tet10"])
        two = e in ("axi", "plane")
        top = {"hex": 24, "tet4": 12, "tet10": 6}.get(e, 60)
        return {"kind": kind, "elem": e, "nr": _log(rng, 5, top), "nz": _log(rng, 50, 600) if two else _log(rng, 10, 80), "steps": 1}
    if kind == "step":
        e = rng.choice(["axi", "plane", "hex", "hex", "tet4", "hex1pt"])
        if e in ("axi", "plane"):
            return {"kind": kind, "elem": e, "nr": _log(rng, 5, 60), "nz": _log(rng, 50, 600), "steps": _log(rng, 10, 60)}
        top, high = {"hex": (30, 200), "tet4": (14, 80), "hex1pt": (36, 300)}[e]
        return {"kind": kind, "elem": e, "nr": _log(rng, 6, top), "nz": _log(rng, 20, high), "steps": _log(rng, 4, 20)}
    if kind == "host":
        return {"kind": kind, "elem": rng.choice(["hex", "axi", "hex1pt"]), "nr": _log(rng, 6, 18), "nz": _log(rng, 20, 120), "steps": 1}
    if kind == "batch":
        return {"kind": kind, "elem": "axi", "nr": _log(rng, 8, 30), "nz": _log(rng, 60, 240), "count": _log(rng, 4, 40), "steps": _log(rng, 5, 20)}
    if kind == "tangent":
        e = rng.choice(["axi", "plane", "hex"])
        two = e != "hex"
        return {"kind": kind, "elem": e, "nr": _log(rng, 5, 24 if two else 8), "nz": _log(rng, 20, 200 if two else 24), "steps": _log(rng, 10, 60)}
    return {"kind": kind, "elem": rng.choice(["axi", "plane"]), "nr": _log(rng, 5, 24), "nz": _log(rng, 40, 240), "steps": _log(rng, 40, 150)}


# ------------------------------------------------------------------------------- the models
ADVANCE = 20  # untimed steps of the step, host and batch cases, so that stresses and speeds fit


def _model(case, seed):
    """The case's model: its generator's mesh with moved nodes, a drawn material and speed."""
    rng = np.random.default_rng([int(seed), 20])
    et, nr, nz = NAMES[case["elem"]], case["nr"], case["nz"]
    slow = case["kind"] in ("step", "host")  # long evolutions: speeds that distort no element badly
    speed = float(rng.uniform(80.0, 140.0) if slow else rng.uniform(150.0, 300.0))
    mat = dict(A=float(rng.uniform(60e6, 150e6)), B=float(rng.uniform(200e6, 400e6)), n=float(rng.uniform(0.2, 0.5)))
    tend = 1.0  # no case reaches it
    if case.get("law") == "table":
        m = meshes.impact_two_materials(nr, nz, speed=speed, tend=tend)
    elif et == AXI:
        m = meshes.taylor_axi(nr, nz, speed=speed, tend=tend, **mat)
    elif et == PLANE:
        m = meshes.taylor_plane(nr, nz, speed=speed, tend=tend, **mat)
    elif et == HEX:
        m = meshes.taylor_hex(nr, nz, speed=speed, tend=tend, **mat)
    elif et == HEX1:
        m = meshes.taylor_hex_1pt(nr, nz, speed=speed, tend=tend, **mat)
    else:
        m = meshes.taylor_tet(nr, nz, quadratic=et == TET10, speed=speed, tend=tend, **mat)
    m = _moved(m, rng)
    if slow:
        m = dataclasses.replace(m, initial_velocity=_mid_impact(m, speed))
    return m


def _moved(m, rng):
    """Nodes moved by up to 3 % of the first element's edge; planes of boundary conditions kept."""
    edge = float(np.linalg.norm(m.coords[m.conn[0, 1]] - m.coords[m.conn[0, 0]]))
    up = m.dim - 1  # the bar's axis
    d = np.zeros_like(m.coords)
    d[:, :m.dim] = rng.uniform(-0.03, 0.03, size=(m.N, m.dim)) * edge
    d[m.coords[:, up] == 0.0, up] = 0.0
    if m.dim == 2:
        d[m.coords[:, 0] == 0.0, 0] = 0.0
    return dataclasses.replace(m, coords=m.coords + d)


def _mid_impact(m, speed):
    """Velocities of a bar some microseconds after impact: the lower third is being squeezed
    (axial speed growing from 0, lateral speeds that keep the volume), the rest still flies."""
    up = m.dim - 1
    x, L = m.coords, float(m.coords[:, up].max())
    c = 0.35 * L
    v = np.zeros((m.N, 3))
    v[:, up] = -speed * np.minimum(1.0, x[:, up] / c)
    zone = x[:, up] < c
    lateral = speed / c * (1.0 if m.etype == PLANE else 0.5)
    for k in range(up):
        v[zone, k] = lateral * x[zone, k] * (1.0 - x[zone, up] / c)
    return v


def _batch_models(case, seed):
    """Uneven bars as meshes.taylor_batch draws them; their sizes go with the case, the rest with the seed."""
    size, rng = np.random.default_rng([case["count"], case["nr"], case["nz"]]), np.random.default_rng([int(seed), 21])
    out = []
    for _ in range(case["count"]):
        nr, nz = int(size.integers(4, case["nr"] + 1)), int(size.integers(40, case["nz"] + 1))
        m = meshes.taylor_axi(nr, nz, speed=float(rng.uniform(150.0, 300.0)), A=float(rng.uniform(60e6, 150e6)),
                              B=float(rng.uniform(200e6, 400e6)), n=float(rng.uniform(0.2, 0.5)), tend=1.0)
        out.append(_moved(m, rng))
    return out


def _loaded_state(m, seed):
    """Stresses around the yield surface, strains, and four displacement increments that load and
    unload in turn (smooth fields and a little noise, strain increments of some 1e-4)."""
    rng = np.random.default_rng([int(seed), 22])
    two = m.dim == 2
    n = m.E * m.nip
    evp = rng.uniform(1e-10, 0.4, n)
    evp[rng.uniform(size=n) < 0.2] = 1e-10

    def sym(scale):
        t = rng.normal(scale=scale, size=(n, 3, 3))
        t = 0.5 * (t + t.transpose(0, 2, 1))
        if two:
            t[:, 0, 2] = t[:, 2, 0] = t[:, 1, 2] = t[:, 2, 1] = 0.0
        return t

    S = sym(1.0)
    S -= np.trace(S, axis1=1, axis2=2)[:, None, None] / 3.0 * np.eye(3)
    q = np.sqrt(1.5 * np.sum(S * S, axis=(1, 2)))
    S *= ((m.A + m.B * evp ** m.n) * rng.uniform(0.7, 1.05, n) / q)[:, None, None]
    st = dict(S=S, Eps=sym(2e-2), EpsPlas=sym(1e-2), p=rng.normal(scale=1e8, size=n), evp=evp)
    x = m.coords
    L = x.max(axis=0) - x.min(axis=0)
    edge = float(np.linalg.norm(x[m.conn[0, 1]] - x[m.conn[0, 0]]))
    dus = []
    for _ in range(2):
        G = rng.normal(scale=3e-4, size=(3, 3))
        du = x @ G.T
        for k in range(m.dim):
            w = rng.integers(1, 5, size=3) * math.pi / np.where(L > 0, L, 1.0)
            du[:, k] += 2e-4 / w[:m.dim].max() * np.sin(x @ w + rng.uniform(0, 6))
        du += rng.normal(scale=5e-5 * edge, size=du.shape)
        du[:, m.dim:] = 0.0
        if m.dim == 2:
            du[x[:, 0] == 0.0, 0] = 0.0
        dus += [du, -du]
    st["du"] = dus
    st["coords"] = [x + du for du in dus]
    return st


# ------------------------------------------------------------------- the no-allocation entry
class _StaticArgs(C.Structure):  # dnl_static_args
    _fields_ = [("etype", C.c_int), ("num_nodes", C.c_int), ("num_elements", C.c_int),
                ("conn", C.c_void_p), ("node_start", C.c_void_p), ("node_entry", C.c_void_p),
                ("coords", C.c_void_p), ("du", C.c_void_p), ("ip", C.c_void_p), ("fint", C.c_void_p),
                ("young", C.c_double), ("poisson", C.c_double), ("density", C.c_double),
                ("A", C.c_double), ("B", C.c_double), ("n", C.c_double)]


_SYM = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _ip_array(m, st):
    """The entry's documented layout: S | Eps | EpsPlas (symmetric components) | p | evp | evp^n."""
    ns = 6 if m.dim == 3 else 4
    rows = [st[k][:, i, j] for k in ("S", "Eps", "EpsPlas") for i, j in _SYM[:ns]]
    return np.stack(rows + [st["p"], st["evp"], st["evp"] ** m.n])


def _static_entry():
    L = dynela.lib()
    L.dnl_internal_forces_static.argtypes = [C.POINTER(_StaticArgs), C.c_void_p, C.POINTER(C.c_int)]
    L.dnl_internal_forces_static.restype = C.c_int
    return L.dnl_internal_forces_static


# ----------------------------------------------------------------------------------- prepare
NODAL = ("coords", "du", "v", "a", "disp")


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "steps": case["steps"], "k": 0}
    if kind == "batch":
        s["b"] = dynela.BatchDomain(_batch_models(case, seed))
        s["b"].prologue()
        s["b"].step(4 * ADVANCE)
        return s
    m = s["m"] = _model(case, seed)
    if kind == "static":
        st = _loaded_state(m, seed)
        dev = torch.device("cuda")
        entry = np.argsort(m.conn.ravel(), kind="stable").astype(np.int32)
        start = np.concatenate([[0], np.cumsum(np.bincount(m.conn.ravel(), minlength=m.N))]).astype(np.int32)
        up = lambda a, t=torch.float64: torch.tensor(np.ascontiguousarray(a), dtype=t, device=dev)  # noqa: E731
        s["conn"], s["start"], s["entry"] = up(m.conn.T, torch.int32), up(start, torch.int32), up(entry, torch.int32)
        s["ip"] = up(_ip_array(m, st))
        s["x"], s["du"] = [up(x.T) for x in st["coords"]], [up(u.T) for u in st["du"]]
        s["fint"] = torch.zeros(m.N * m.dim, dtype=torch.float64, device=dev)
        s["call"] = _static_entry()
        return s
    d = s["d"] = dynela.GpuDomain(m)
    if kind == "forces":
        st = _loaded_state(m, seed)
        d.set_state(**{k: st[k] for k in ("S", "Eps", "EpsPlas", "p", "evp")})
        s["x"], s["du"] = st["coords"], st["du"]
        return s
    if kind in ("tangent", "gradient"):
        s["dts"] = _schedule(m, case["steps"])
        d.prologue()
        rng = np.random.default_rng([int(seed), 23])
        s["dL"] = np.zeros((m.N, 3))
        s["dL"][:, :m.dim] = rng.normal(size=(m.N, m.dim))
        return s
    d.prologue()
    if kind in ("step", "host"):
        d.step(ADVANCE)
    if kind == "host":
        # page-locked arrays: the state in, the state out, exchanged from call to call
        s["io"] = [{k: torch.zeros((m.N, 3), dtype=torch.float64).pin_memory().numpy() for k in NODAL} for _ in range(2)]
        st = d.get_state(*NODAL)
        for k in NODAL:
            s["io"][0][k][:] = st[k]
    return s


def _schedule(m, steps):
    """A step-size schedule: half the quad's or hexahedron's smallest edge over the sound speed."""
    x = m.coords[m.conn]
    edge = min(float(np.linalg.norm(x[:, b] - x[:, a], axis=1).min()) for a, b in ((0, 1), (1, 2), (0, 3 if m.dim == 2 else 4)))
    c = math.sqrt(m.young * (1 - m.poisson) / (m.density * (1 + m.poisson) * (1 - 2 * m.poisson)))
    return np.full(steps, 0.5 * edge / c)


# --------------------------------------------------------------------------------------- run
def run(s):
    kind, k = s["kind"], s["k"]
    s["k"] += 1
    if kind == "study":
        d, m = s["d"], s["m"]
        if m.initial_velocity is None:
            d.reset(m)
        else:  # several materials stay; speeds by node
            d.reset()
            d.set_state(v=m.initial_velocity)
        d.step(s["steps"])
        return d.get_state("coords", "v", "S", "p", "evp")
    if kind == "forces":
        return s["d"].internal_forces(s["x"][k % 4], s["du"][k % 4], 1e-8)
    if kind == "static":
        m, ptr = s["m"], torch.Tensor.data_ptr
        args = _StaticArgs(m.etype, m.N, m.E, ptr(s["conn"]), ptr(s["start"]), ptr(s["entry"]), ptr(s["x"][k % 4]),
                           ptr(s["du"][k % 4]), ptr(s["ip"]), ptr(s["fint"]), m.young, m.poisson, m.density, m.A, m.B, m.n)
        bad = C.c_int(-1)
        rc = s["call"](C.byref(args), torch.cuda.current_stream().cuda_stream or None, C.byref(bad))
        if rc:
            raise RuntimeError(f"dnl_internal_forces_static: status {rc}, element {bad.value}")
        return s["fint"], s["ip"]
    if kind == "step":
        s["d"].step(s["steps"])
        return s["d"].get_state("coords", "v", "disp")
    if kind == "host":
        src, dst = s["io"][k % 2], s["io"][(k + 1) % 2]
        s["d"].step_host(s["steps"], src, dst)
        return dst
    if kind == "batch":
        b = s["b"]
        b.step_graph(s["steps"])
        return np.concatenate([b.coords(i) for i in range(len(b.models))])
    if kind == "tangent":
        s["d"].reset()
        return s["d"].sensitivities(s["dts"])
    return s["d"].adjoint_forward(s["dts"]), s["d"].adjoint_backward(s["dL"])


# -------------------------------------------------------------------------------------- work
# FP64 operations (a fused multiply-add is two) that one integration point of a pass cannot do
# without: kinematics, polar decomposition, radial return of the yielding third, three rotated
# tensors, forces
_FLOPS = {AXI: 350, PLANE: 330, HEX: 900, TET4: 700, TET10: 800, HEX1: 1300}


def _counts(et, nr, nz):
    """(nodes, elements) of the generator's mesh, without building it."""
    if et in (AXI, PLANE):
        return (nr + 1) * (nz + 1), nr * nz
    layer = meshes.taylor_hex(nr, 1)
    n, e = layer.N // 2 * (nz + 1), layer.E * nz
    return (n, e) if et in (HEX, HEX1) else (n, 6 * e) if et == TET4 else (n + 7 * e, 6 * e)


def work(case):
    et, kind, steps = NAMES[case["elem"]], case["kind"], case["steps"]
    if kind == "batch":  # the mean of the drawn sizes
        N, E = _counts(et, (4 + case["nr"]) // 2, (40 + case["nz"]) // 2)
        N, E = N * case["count"], E * case["count"]
    else:
        N, E = _counts(et, case["nr"], case["nz"])
    dim = 2 if et in (AXI, PLANE) else 3
    nip, nen = meshes.NIP_OF[et], meshes.NEN_OF[et]
    ncomp = 15 if dim == 2 else 21
    state = 8 * ncomp * E * nip       # integration-point state
    nodal = 8 * dim * N
    mesh = 4 * nen * E
    if kind in ("forces", "static"):  # coordinates and increments in, state in and out, forces out
        return {"bytes": 2 * state + 3 * nodal + mesh, "flops": _FLOPS[et] * E * nip}
    if kind == "host":                # five nodal fields in and out, state in and out
        return {"bytes": 2 * state + 10 * 24 * N + mesh, "flops": (_FLOPS[et] * E * nip + 30 * dim * N) * steps}
    # a run reads its initial state and writes its final one; derivatives: four copies beside it
    # (forward), the run, its repetition and the way back (reverse)
    copies = {"tangent": 5}.get(kind, 1)
    passes = {"tangent": 3.0, "gradient": 3.0}.get(kind, 1.0)
    return {"bytes": copies * (2 * state + 10 * nodal) + mesh,
            "flops": passes * steps * (_FLOPS[et] * E * nip + 30 * dim * N)}


# ------------------------------------------------------------------------------------- exact
# The same mathematics in plain 64-bit torch, written element by element over whole arrays: the
# element pass (incremental log strain by the Jacobi polar decomposition with its stopping test,
# J2 radial return, element-mean pressure, rotated tensors, forces), lumped mass, critical time
# step and the Chung-Hulbert update.


def _shape(et):
    """Shape values (q, k), derivatives (q, k, c) and weight at the Gauss points."""
    if et == TET4:
        return np.full((1, 4), 0.25), np.array([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], float), 1 / 6
    if et == TET10:
        # the reference's tables, with the two constants its unparenthesised macros give
        r5 = math.sqrt(5.0)
        a4, b4, a4n, b4n = 1 - 1 / r5, 1 + 3 / r5, -1 - 1 / r5, -1 + 3 / r5
        ea, eb = (0, 1, 0, 0, 1, 2), (1, 2, 2, 3, 3, 3)
        N, D = np.zeros((4, 10)), np.zeros((4, 10, 3))
        for p in range(4):
            N[p, :4] = [0.1 if i == p else -0.1 for i in range(4)]
            N[p, 4:] = [(1 + r5) / 10 if p in (a, b) else (3 - r5) / 10 for a, b in zip(ea, eb)]
            for c in range(3):
                D[p, 0, c] = -3 / r5 if p == 0 else 1 / r5
                D[p, c + 1, c] = 3 / r5 if p == c + 1 else -1 / r5
                for m, (a, b) in enumerate(zip(ea, eb)):
                    da, db = (-1 if a == 0 else int(c == a - 1)), int(c == b - 1)
                    if da == -1 and db == 1:
                        D[p, 4 + m, c] = 4 / r5 if p == 0 else (-4 / r5 if p == b else 0.0)
                    elif da == -1:
                        D[p, 4 + m, c] = b4n if p == b else a4n
                    elif da or db:
                        D[p, 4 + m, c] = b4 if p == (b if da else a) else a4
        return N, D, 1 / 24
    three = et in (HEX, HEX1)
    sign = np.array([(sx, sy) for sx, sy in ((-1, -1), (1, -1), (1, 1), (-1, 1))], float)
    if three:
        sign = np.array([(*xy, z) for z in (-1, 1) for xy in sign])
    pts = np.zeros((1, 3)) if et == HEX1 else sign / math.sqrt(3.0)
    d = sign.shape[1]
    f = 1 + pts[:, None, :] * sign[None]  # (q, k, d)
    D = np.stack([sign[None, :, c] * np.prod(np.delete(f, c, axis=2), axis=2) for c in range(d)], axis=2) / 2 ** d
    return np.prod(f, axis=2) / 2 ** d, D, 8.0 if et == HEX1 else 1.0


class _Plain:
    R23, R32 = math.sqrt(2 / 3), math.sqrt(3 / 2)

    def __init__(self, m):
        self.m, self.dev = m, torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.dim, self.axi = m.dim, m.etype == AXI
        up = lambda a: torch.tensor(np.asarray(a, dtype=float), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.up, self.conn = up, torch.tensor(np.asarray(m.conn), device=self.dev)
        N, D, self.w = _shape(m.etype)
        self.N, self.D = up(N), up(D)
        E, q = m.E, N.shape[0]
        self.S, self.Ep, self.Epl = (torch.zeros(E, q, 3, 3, dtype=torch.float64, device=self.dev) for _ in range(3))
        self.p, self.evp = torch.zeros_like(self.S[..., 0, 0]), torch.full_like(self.S[..., 0, 0], 1e-10)
        laws = m.material_laws()
        em = torch.tensor(np.zeros(E, int) if m.elem_material is None else np.asarray(m.elem_material), device=self.dev)
        pick = lambda v: up(v)[em][:, None]  # noqa: E731  per element, over its points
        self.laws, self.em = laws, em[:, None].expand(E, q)
        G = pick([0.5 * a.young / (1 + a.poisson) for a in laws])
        self.G, self.K = G, pick([a.young / (3 * (1 - 2 * a.poisson)) for a in laws])
        self.rho = pick([a.density for a in laws])
        self.young, self.nu = pick([a.young for a in laws]), pick([a.poisson for a in laws])
        self.x = up(m.coords)
        z = torch.zeros_like(self.x)
        v = z + up(m.v0) if m.initial_velocity is None else up(m.initial_velocity)
        self.du, self.v, self.a, self.disp = z.clone(), v.clone(), z.clone(), z.clone()

    def law(self, evp):
        """Yield stress and slope at evp."""
        sig, h = torch.zeros_like(evp), torch.zeros_like(evp)
        for i, a in enumerate(self.laws):
            at = self.em == i
            if a.law == meshes.HARD_POWER:
                A, B, n = a.params
                s_, h_ = A + B * evp ** n, n * B * evp ** (n - 1)
            elif a.law == meshes.HARD_TABULAR:
                X, Y = self.up(a.table_x), self.up(a.table_y)
                j = torch.searchsorted(X[1:].contiguous(), evp.contiguous()).clamp(max=len(X) - 2)
                h_ = (Y[j + 1] - Y[j]) / (X[j + 1] - X[j])
                s_ = (evp - X[j]) / (X[j + 1] - X[j]) * (Y[j + 1] - Y[j]) + Y[j]
            else:  # no hardening attached: never yields
                s_, h_ = torch.full_like(evp, 1e300), torch.zeros_like(evp)
            sig, h = torch.where(at, s_, sig), torch.where(at, h_, h)
        return sig, h

    def kinematics(self, x):
        xe = x[self.conn][..., :self.dim]
        J = torch.einsum("ekr,qkc->eqrc", xe, self.D)
        det = torch.linalg.det(J)
        B = torch.einsum("qkl,eqlc->eqkc", self.D, torch.linalg.inv(J))
        R = torch.einsum("qk,ek->eq", self.N, xe[..., 0]) if self.axi else None
        W = self.w * det * (2 * math.pi * R if self.axi else 1.0)
        return B, W, R

    def polar(self, F):
        """R and ln U by cyclic-free Jacobi rotations of F^T F, stopped at 1e-9."""
        C = F.transpose(-1, -2) @ F
        V = torch.eye(3, dtype=torch.float64, device=self.dev).expand_as(C).clone()
        for _ in range(29):
            o = torch.stack([C[..., 0, 1], C[..., 0, 2], C[..., 1, 2]], -1)
            b = o.abs()
            q1 = b[..., 0] > b[..., 1]
            p0 = torch.where(q1, b[..., 0], b[..., 1]) > b[..., 2]
            k = torch.where(p0, torch.where(q1, 0, 1), 2)
            x = o.gather(-1, k[..., None])[..., 0]
            go = x.abs() >= 1e-9
            if not bool(go.any()):
                break
            p, q = (k == 2).long(), 2 - (k == 0).long()
            dg = torch.diagonal(C, dim1=-2, dim2=-1)
            al = (dg.gather(-1, q[..., None]) - dg.gather(-1, p[..., None]))[..., 0] / (2 * torch.where(go, x, 1.0))
            t = 1 / (al.abs() + torch.sqrt(al * al + 1)) * torch.where(al < 0, -1.0, 1.0)
            c = 1 / torch.sqrt(1 + t * t)
            s = torch.where(go, t * c, 0.0)
            c = torch.where(go, c, 1.0)
            Q = torch.eye(3, dtype=torch.float64, device=self.dev).expand_as(C).clone()
            ix = lambda i, j: (3 * i + j)[..., None]  # noqa: E731
            Qf = Q.view(*Q.shape[:-2], 9)
            for i, j, val in ((p, p, c), (q, q, c), (p, q, s), (q, p, -s)):
                Qf.scatter_(-1, ix(i, j), val[..., None])
            C = Q.transpose(-1, -2) @ C @ Q
            V = V @ Q
        lam = torch.diagonal(C, dim1=-2, dim2=-1)
        lnU = (V * (0.5 * torch.log(lam))[..., None, :]) @ V.transpose(-1, -2)
        return F @ ((V * lam.rsqrt()[..., None, :]) @ V.transpose(-1, -2)), lnU

    def forces(self):
        """The element pass on x and du: updates the integration-point state, returns N x dim."""
        B, W, Rad = self.kinematics(self.x)
        ue = self.du[self.conn][..., :self.dim]
        F = torch.eye(3, dtype=torch.float64, device=self.dev).expand_as(self.S).clone()
        F[..., :self.dim, :self.dim] += torch.einsum("ekr,eqkc->eqrc", ue, B)
        if self.axi:
            F[..., 2, 2] += torch.einsum("qk,ek->eq", self.N, ue[..., 0]) / Rad
        R, dE = self.polar(F)
        tr = torch.diagonal(dE, dim1=-2, dim2=-1).sum(-1)
        I = torch.eye(3, dtype=torch.float64, device=self.dev)
        S = self.S + 2 * self.G[..., None, None] * (dE - tr[..., None, None] / 3 * I)
        norm = torch.sqrt((S * S).sum((-1, -2)))
        s0, h = self.law(self.evp)
        yields = self.R32 * norm > s0
        G2 = 2 * self.G
        gam = torch.where(yields, (norm - self.R23 * s0) / (G2 * (1 + h / (3 * self.G))), 0.0)
        on = yields.clone()
        while bool(on.any()):
            sv, h = self.law(torch.where(yields, self.evp + self.R23 * gam, self.evp))
            df = self.R32 * G2 + self.R23 * h
            f = df * gam - (self.R32 * norm - sv + h * self.R23 * gam)
            on = on & ((f / sv).abs() > 1e-8)
            dg = -f / df
            dg = torch.where((dg < 0) & (dg.abs() > gam), -0.9 * gam, dg)
            gam = torch.where(on, gam + dg, gam)
        n1 = S / torch.where(yields, norm, 1.0)[..., None, None]
        S = S - (G2 * gam)[..., None, None] * n1
        Epl = self.Epl + gam[..., None, None] * n1
        self.evp = self.evp + self.R23 * gam
        self.p = self.p + self.K * tr.mean(1, keepdim=True)
        Rt = R.transpose(-1, -2)
        self.S, self.Ep, self.Epl = R @ S @ Rt, R @ (self.Ep + dE) @ Rt, R @ Epl @ Rt
        sig = self.S + self.p[..., None, None] * I
        fe = -torch.einsum("eqkc,eqcr,eq->ekr", B, sig[..., :self.dim, :self.dim], W)
        if self.axi:
            fe[..., 0] -= torch.einsum("qk,eq->ek", self.N, sig[..., 2, 2] * W / Rad)
        if self.m.etype == HEX1:
            fe -= self.hourglass(B[:, 0], W[:, 0])
        return self.gather(fe)

    def hourglass(self, b, V):
        s = self.up([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
        h = torch.stack([s[:, 0] * s[:, 1], s[:, 1] * s[:, 2], s[:, 2] * s[:, 0], s[:, 0] * s[:, 1] * s[:, 2]])
        g = h - torch.einsum("qk,ekr,ejr->eqj", h, self.x[self.conn], b)
        qv = torch.einsum("eqk,ekr->eqr", g, self.v[self.conn])
        ah = 0.25 * self.m.hourglass * self.rho[:, 0] * self.sound()[:, 0] * V ** (2 / 3)
        return ah[:, None, None] * torch.einsum("eqk,eqr->ekr", g, qv)

    def gather(self, fe):
        out = torch.zeros(self.m.N, fe.shape[-1], dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.conn.reshape(-1), fe.reshape(-1, fe.shape[-1]))

    def sound(self):
        # the mean density of the element's nodes, a node's that of the last element holding it
        if not hasattr(self, "ro"):
            conn, last = np.asarray(self.m.conn), np.zeros(self.m.N, dtype=int)
            np.maximum.at(last, conn.ravel(), np.repeat(np.arange(conn.shape[0]), conn.shape[1]))
            self.ro = self.rho[:, 0][torch.tensor(last, device=self.dev)]
        ro = self.ro[self.conn].mean(1, keepdim=True)
        return torch.sqrt(self.young * (1 - self.nu) / (ro * (1 + self.nu) * (1 - 2 * self.nu)))

    def frequency(self):
        """The largest frequency: Courant's estimate, or the power iteration of Pulse."""
        if self.m.method == meshes.COURANT:
            x = self.x[self.conn]
            if self.dim == 2:
                a, b = x[:, 2] - x[:, 0], x[:, 1] - x[:, 3]
                num = a[:, 0] * -b[:, 1] + b[:, 0] * a[:, 1]
                l = num / torch.sqrt(2 * (a[:, :2].square().sum(1) + b[:, :2].square().sum(1)))
            elif self.m.etype == HEX1:
                B, W, _ = self.kinematics(self.x)
                l = W[:, 0] / torch.stack([0.5 * torch.linalg.cross(x[:, c] - x[:, a], x[:, d] - x[:, b]).norm(dim=1) for a, b, c, d in (
                    (0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7))]).amax(0)
            else:
                l = torch.stack([(x[:, i] - x[:, j]).norm(dim=1) for i, j in ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))]).amin(0)
            return 2.0 / float((l / self.sound()[:, 0]).amin())
        B, W, _ = self.kinematics(self.x)
        lam, mu = (self.K - 2 * self.G / 3)[..., None, None], self.G[..., None, None]
        I = torch.eye(3, dtype=torch.float64, device=self.dev)
        if not hasattr(self, "ev"):
            n = 3 * self.m.N
            self.ev, self.f0 = (1.0 - 2.0 / (n - 1) * torch.arange(n, dtype=torch.float64, device=self.dev)).view(-1, 3), 0.0
        for _ in range(1000):
            g = torch.einsum("ekr,eqkc->eqrc", self.ev[self.conn], B)
            sg = lam * torch.diagonal(g, dim1=-2, dim2=-1).sum(-1)[..., None, None] * I + mu * (g + g.transpose(-1, -2))
            self.ev = self.gather(torch.einsum("eqkc,eqcr,eq->ekr", B, sg, W)) / self.mass[:, None]
            f = float(self.ev.abs().amax())
            self.ev = self.ev / f
            done, self.f0 = abs(f - self.f0) / f < 1e-4, f
            if done:
                break
        return math.sqrt(f)

    def start(self):
        r = self.m.rho_b
        self.am, self.beta = (2 * r - 1) / (1 + r), (5 - 3 * r) / ((1 + r) ** 2 * (2 - r))
        self.gamma = 1.5 - self.am
        self.so = self.m.safety * math.sqrt(12 * (1 + r) ** 3 * (2 - r) / (10 + 15 * r - r * r + r ** 3 - r ** 4))
        B, W, _ = self.kinematics(self.x)
        self.mass = self.gather((self.rho[..., None] * self.N[None] * W[..., None]).sum(1)[..., None])[:, 0]
        self.fix = torch.zeros(self.m.N, 3, dtype=torch.bool, device=self.dev)
        for bc in self.m.bcs:
            for c in range(3):
                if bc.val[c] == 1.0:
                    self.fix[torch.tensor(np.asarray(bc.nodes), device=self.dev), c] = True
        self.forces()
        self.t, self.ts, self.lts, self.inc = 0.0, 0.0, 0.0, 0
        self.dt = self.cdt = self.so / self.frequency()
        self.ldt = 0.0

    def step(self, n):
        free = (~self.fix).to(torch.float64)
        for _ in range(n):
            self.inc += 1
            dt = self.dt
            self.du, self.v, self.a = self.du * free, self.v * free, self.a * free
            f = torch.zeros_like(self.x)
            f[:, :self.dim] = self.forces()
            du = (self.a * (dt * (0.5 - self.beta)) + self.v) * dt
            v = self.a * (dt * (1 - self.gamma)) + self.v
            a = (f / self.mass[:, None] - self.am * self.a) / (1 - self.am)
            self.v = (v + dt * self.gamma * a) * free
            self.du = (du + dt * dt * self.beta * a) * free
            self.a = a * free
            self.disp = self.disp + self.du
            self.x = self.x + self.du
            self.t += dt
            if self.inc % self.m.freq == 0:
                self.dt = self.so / self.frequency()
                self.lts, self.ldt, self.ts, self.cdt = self.ts, self.cdt, self.t, self.dt
            elif self.ts != self.lts:
                y = (self.t - self.lts) / (self.ts - self.lts)
                self.dt = y * self.cdt + (1 - y) * self.ldt

    def out(self, *names):
        get = dict(coords=self.x, du=self.du, v=self.v, a=self.a, disp=self.disp, S=self.S, p=self.p.expand_as(self.evp), evp=self.evp)
        return {k: get[k].cpu().numpy() for k in names}


def exact(case, seed):
    kind, et, steps = case["kind"], NAMES[case["elem"]], case["steps"]
    if kind in ("tangent", "gradient"):
        return None  # derivatives of a whole run: minutes in plain torch
    if kind == "batch":
        ms = _batch_models(case, seed)
        if sum(m.E for m in ms) * (4 * ADVANCE + steps) > 2e6:
            return None  # bar after bar, over 20 seconds
        outs = []
        for m in ms:
            r = _Plain(m)
            r.start()
            r.step(4 * ADVANCE + steps)
            outs.append(r.out("coords")["coords"])
        return np.concatenate(outs)
    _, E = _counts(et, case["nr"], case["nz"])
    advance = ADVANCE if kind in ("step", "host") else 0
    if E * meshes.NIP_OF[et] * (advance + steps) > 1e8 or (et == HEX and kind in ("step", "host") and E > 3e4):
        return None  # over 20 seconds
    m = _model(case, seed)
    r = _Plain(m)
    if kind in ("forces", "static"):
        st = _loaded_state(m, seed)
        for k, name in (("S", "S"), ("Ep", "Eps"), ("Epl", "EpsPlas"), ("p", "p"), ("evp", "evp")):
            setattr(r, k, r.up(st[name]).view_as(getattr(r, k)))
        r.x, r.du = r.up(st["coords"][0]), r.up(st["du"][0])
        f = r.forces().reshape(-1).cpu().numpy()
        if kind == "forces":
            return f
        n = m.E * m.nip
        back = {a: b.reshape((n,) + b.shape[2:]).cpu().numpy() for a, b in dict(
            S=r.S, Eps=r.Ep, EpsPlas=r.Epl, p=r.p.expand_as(r.evp), evp=r.evp).items()}
        return f, _ip_array(m, back)
    r.start()
    r.step(advance + steps)
    return r.out(*{"study": ("coords", "v", "S", "p", "evp"), "step": ("coords", "v", "disp"), "host": NODAL}[kind])
