"""The element cycle as programs use it: workloads to time, and their values in 64 bits.

A case is one call pattern on one deck: an engine keeps a handle (``ECycle``) with the
model on the GPU, advances it by a number of cycles and reads the nodes back into its
own pinned arrays, as the RESOL hook does at every output interval or coupling step.
Two patterns differ: a design study calls the adjoint, and an engine with its own device
pool calls the entry point that allocates nothing.

Every call goes on from the state the last one left, until the job's last cycle (JOB);
the next call then begins the job again, as a parameter study does.  The seed
makes the velocity field, and the yield stresses and thicknesses where a deck has them per
element; the mesh, with its nodes moved off the regular grid, follows from the case.

The FP64 form's results are returned in 64 bits.  The split form computes elements,
velocities and forces in 32 bits; what it returns is taken in 32 bits, as the reference
writes its animation files.

``exact`` restates the cycle (SFORC3 and CFORC3 chains, ASSPAR4 to DEPLA) in plain
torch, FP64; the gradient of the adjoint case is torch's own reverse mode.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from openradioss_b200 import abi, adjoint, decks
from openradioss_b200.ecycle import ECycle, load_library

DTMX_ADJOINT = 1.4e-7       # below every element step of the 1 mm plate: dt does not depend on the design
W_PLASTIC = 1e-4            # m/J: weight of the plastic work beside the centre's deflection
POOL_MAX_HEXAS = 32768      # OR_NOALLOC_MAX_SLOTS / 8


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a coupled program that exchanges every cycle: one cycle a call on a crash rail (rigid
        # link, 3 points, /SHFRA/V4 frames, yield cap); latency and host work
        dict(name="rail_one_cycle", kind="rail", edge=5e-3, precision="fp64", cycles=1),
        # the C1 validation block between two time-history outputs, element state included
        dict(name="block_fp64", kind="block", nx=10, ny=10, nz=40, law=1, frame=0, precision="fp64", cycles=200),
        # a medium solid part of odd sizes, both forms, FP64 in the convected frame (Iframe 2)
        dict(name="block_split", kind="block", nx=37, ny=41, nz=83, law=2, frame=0, precision="split", cycles=100),
        dict(name="block_frame_fp64", kind="block", nx=23, ny=29, nz=61, law=2, frame=1, precision="fp64", cycles=100),
        # the headline plate (200 x 200, 5 points, Johnson-Cook) between two outputs
        dict(name="plate_split", kind="plate", n=200, points=5, ipla=0, law=2, precision="split", cycles=100),
        # a smaller one in FP64, 3 points with the Newton return (Iplas 1): the general shell kernels, a ragged size
        dict(name="plate_newton_fp64", kind="plate", n=151, points=3, ipla=1, law=2, precision="fp64", cycles=100),
        # a large sheet, beyond what one wave of the GPU holds
        dict(name="sheet_split", kind="plate", n=600, points=5, ipla=0, law=2, precision="split", cycles=100),
        # many independent parts of uneven size with time steps of their own
        dict(name="parts_split", kind="parts", parts=64, smallest=1000, largest=50000, precision="split", cycles=200),
        # the largest mesh: 2 M hexas with a shell skin on shared nodes; and a quarter-million in FP64
        dict(name="mixed_split", kind="mixed", nx=100, ny=100, nz=200, precision="split", cycles=200),
        dict(name="mixed_fp64", kind="mixed", nx=50, ny=50, nz=100, precision="fp64", cycles=100),
        # design sensitivities of the plate (forward with checkpoints, reverse), FP64
        dict(name="adjoint_plate", kind="adjoint", n=200, checkpoint=50, cycles=100),
        # an engine that owns every device array: the entry point that allocates nothing, FP64
        dict(name="pool_block", kind="pool", nx=24, ny=24, nz=48, law=2, cycles=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rail", "block", "block", "plate", "plate", "plate", "parts", "mixed", "adjoint", "pool"])
    precision = rng.choice(["split", "split", "fp64"])
    law = rng.choice([1, 2, 2])
    if kind == "rail":
        return dict(kind=kind, edge=round(math.exp(rng.uniform(math.log(2e-3), math.log(1e-2))), 5),
                    precision=precision, cycles=rng.choice([1, 1, 2, 5]))
    if kind in ("block", "pool"):
        most = POOL_MAX_HEXAS if kind == "pool" else 500000
        while True:
            nx, ny, nz = _log(rng, 3, 60), _log(rng, 3, 60), _log(rng, 6, 150)
            if 500 <= nx * ny * nz <= most:
                break
        if kind == "pool":
            return dict(kind=kind, nx=nx, ny=ny, nz=nz, law=law, cycles=rng.randint(20, 100))
        # the convected frame in FP64: in 32 bits its own rounding moves the results by 1e-4
        frame = rng.choice([0, 0, 1])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, law=law, frame=frame, precision="fp64" if frame else precision,
                    cycles=rng.randint(50, 150))
    if kind == "plate":
        return dict(kind=kind, n=_log(rng, 20, 600), points=rng.choice([5, 5, 5, 3]), ipla=rng.choice([0, 0, 1]),
                    law=law, precision=precision, cycles=rng.randint(40, 120))
    if kind == "parts":
        smallest = _log(rng, 500, 4000)
        return dict(kind=kind, parts=rng.randint(4, 64), smallest=smallest, largest=smallest * rng.randint(4, 25),
                    precision=precision, cycles=rng.randint(50, 200))
    if kind == "mixed":
        nx, ny = _log(rng, 6, 70), _log(rng, 6, 70)
        return dict(kind=kind, nx=nx, ny=ny, nz=_log(rng, 12, 150), precision=precision, cycles=rng.randint(50, 150))
    return dict(kind=kind, n=_log(rng, 30, 200), checkpoint=rng.choice([20, 50]), cycles=rng.randint(40, 120))


# ---------------------------------------------------------------------------
# decks
# ---------------------------------------------------------------------------
def _block_part(rng, nx, ny, nz, law, frame, speed):
    """A block of about 1 mm hexas (nodes moved by up to 5 % of the edge) thrown at its clamped base."""
    x, conn = decks.hex_block(nx, ny, nz, 1e-3)
    base = np.isclose(x[:, 2], 0.0)
    moved = np.random.Generator(np.random.PCG64(nx + ny + nz))
    x[~base] += moved.uniform(-5e-5, 5e-5, size=(int((~base).sum()), 3))
    p = decks.new_part(x)
    decks.add_hex(p, conn, decks.steel_elastic() if law == 1 else decks.steel_jc(), decks.solid_prop(jcvt=frame))
    p["icodt"][base] = 7
    p["v"][~base] = speed
    p["v"][~base] += rng.uniform(-0.2, 0.2, size=(int((~base).sum()), 3))
    return p


def _plate_speed(rng, law):
    """Beyond yield for Johnson-Cook; an elastic plate keeps its energy, so less."""
    return float(rng.uniform(30.0, 40.0) if law == 2 else rng.uniform(8.0, 12.0))


def _plate_part(rng, n, speed, **kw):
    """A plate of n x n 1 mm shells, edges held, thrown along its normal, under a slight pressure."""
    p = decks.c2_shell_plate(n=n, size=n * 1e-3, pressure=1e4, seed=n, **kw)["parts"][0]
    free = p["icodt"] == 0
    p["icodt"][~free] = 7
    p["v"][free, 2] = speed + rng.uniform(-0.2, 0.2, size=int(free.sum()))
    return p


def _sizes(c):
    """The parts case's parts, as (is hexa, law, element count asked for): sizes even on a log scale, shuffled."""
    f = np.linspace(0.0, 1.0, c["parts"])
    nel = np.exp(np.log(c["smallest"]) + f * (np.log(c["largest"]) - np.log(c["smallest"])))
    order = np.random.Generator(np.random.PCG64(c["parts"])).permutation(c["parts"])
    return [(i % 2 == 0, 1 + (i // 2) % 2, float(nel[k])) for i, k in enumerate(order)]


def _hexa_edge(nel):
    return max(3, int(round((nel / 4.0) ** (1.0 / 3.0))))


def _plate_edge(nel):
    return max(4, int(round(math.sqrt(nel))))


def make_deck(c, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = c["kind"]
    if kind == "rail":
        return decks.hat_rail(h=c["edge"], mass=5.0, v0=float(rng.uniform(8.0, 12.0)))
    if kind in ("block", "pool"):
        speed = [0.0, 0.0, -float(rng.uniform(8.0, 12.0) if c["law"] == 1 else rng.uniform(30.0, 50.0))]
        return decks.deck([_block_part(rng, c["nx"], c["ny"], c["nz"], c["law"], c.get("frame", 0), speed)])
    if kind == "plate":
        return decks.deck([_plate_part(rng, c["n"], _plate_speed(rng, c["law"]), npt=c["points"],
                                       ipla=c["ipla"], law=c["law"])])
    if kind == "parts":
        parts = []
        for is_hex, law, nel in _sizes(c):
            if is_hex:
                n = _hexa_edge(nel)
                way = rng.normal(size=3)
                way *= rng.uniform(5.0, 20.0) / np.linalg.norm(way)
                parts.append(_block_part(rng, n, n, 4 * n, law, 0, way))
            else:
                parts.append(_plate_part(rng, _plate_edge(nel), float(rng.uniform(5.0, 12.0)), law=law))
        return decks.deck(parts)
    if kind == "mixed":
        d = decks.c4_mixed_mesh(nx=c["nx"], ny=c["ny"], nz=c["nz"], vz=-float(rng.uniform(15.0, 25.0)))
        p = d["parts"][0]
        free = p["icodt"] == 0
        p["v"][free] += rng.uniform(-0.5, 0.5, size=(int(free.sum()), 3))
        return d
    nel = c["n"] ** 2
    p = _plate_part(rng, c["n"], _plate_speed(rng, 2), jc_a=rng.uniform(300e6, 400e6, nel),
                    thke=rng.uniform(0.9e-3, 1.1e-3, nel))
    d = decks.deck([p])
    d["dtmx"] = DTMX_ADJOINT
    return d


# ---------------------------------------------------------------------------
# the framework's calls
# ---------------------------------------------------------------------------
LEAD = 64       # cycles that the coupled program has run before the call in question
JOB = 5000      # cycles of a job


def prepare(c, seed):
    d = make_deck(c, seed)
    if c["kind"] == "pool":
        return _prepare_pool(c, d)
    split = c.get("precision") == "split"
    h = ECycle(d, precision=abi.OR_PREC_SPLIT if split else abi.OR_PREC_FP64)
    s = dict(case=c, handle=h, deck=d)
    if c["kind"] == "adjoint":
        s["node"] = adjoint.centre_node(d)
        return s
    # the engine's arrays: pinned, all parts in one, the rotations where the model is all shells
    rows = [p["x"].shape[0] for p in d["parts"]]
    rot = not h.hex_groups
    s["out"] = {k: torch.zeros((sum(rows), 3), dtype=torch.float64).pin_memory()
                for k in (("d", "v", "vr") if rot else ("d", "v"))}
    dp = C.POINTER(C.c_double)
    s["args"] = []
    for part, first in enumerate(np.cumsum([0] + rows[:-1])):
        at = lambda k: C.cast(s["out"][k].data_ptr() + 24 * int(first), dp) if k in s["out"] else None
        s["args"].append((part, None, at("d"), at("v"), at("vr")))
    if split:
        s["out32"] = {k: torch.empty_like(a, dtype=torch.float32) for k, a in s["out"].items()}
    if c["kind"] == "rail":
        h.step(LEAD)
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "pool":
        return _run_pool(s)
    h = s["handle"]
    if h.times[0].ncycle >= JOB:
        h.reset()
    if c["kind"] == "adjoint":
        r = h.adjoint(c["cycles"], node=s["node"], w_plastic=W_PLASTIC, checkpoint=c["checkpoint"])
        return dict(J=r["J"], dA=r["dA"][0], dthk=r["dthk"][0], dms=r["dms"][0], din=r["din"][0])
    h.step(c["cycles"])
    for part, x, d, v, vr in s["args"]:
        h._call("get_nodes", part, x, d, v, vr)
    if "out32" in s:
        return {k: s["out32"][k].copy_(a) for k, a in s["out"].items()}
    out = dict(s["out"])
    if c["kind"] == "block":
        out.update(h.hex_state(0))
    return out


def _prepare_pool(c, d):
    """Device arrays of one hexa group in the engine's layout, with its Parith/ON tables."""
    p = d["parts"][0]
    g = p["hex"][0]
    conn = (g["ixs"][:, 1:9] - 1).astype(np.int32)
    numnod, nel = p["x"].shape[0], conn.shape[0]
    adsky = np.zeros(numnod + 1, np.int32)
    adsky[1:] = np.cumsum(np.bincount(conn.ravel(), minlength=numnod))
    iads = np.empty(8 * nel, np.int32)
    iads[np.argsort(conn.ravel(), kind="stable")] = np.arange(8 * nel, dtype=np.int32)
    put = lambda a, t: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    f64, i32 = torch.float64, torch.int32
    a = dict(x=put(p["x"], f64), d=torch.zeros((numnod, 3), dtype=f64, device="cuda"), v=put(p["v"], f64),
             ms=put(p["ms"], f64), icodt=put(p["icodt"], i32), conn=put(conn, i32), iads=put(iads, i32),
             adsky=put(adsky, i32), sig=torch.zeros((6, nel), dtype=f64, device="cuda"), vol0=put(g["vol0"], f64),
             rho=torch.full((nel,), g["mat"]["rho0"], dtype=f64, device="cuda"))
    for k in ("eint", "qvis", "pla", "epsd"):
        a[k] = torch.zeros(nel, dtype=f64, device="cuda")
    f = load_library().or_ecycle_hex_step_noalloc
    P = C.c_void_p
    f.argtypes = [C.c_int, P, C.c_int, C.POINTER(abi.Time), C.c_int] + [P] * 5 + [C.c_int] + [P] * 3 + \
                 [C.POINTER(abi.Material), C.POINTER(abi.SolidProp)] + [C.c_double] * 3 + [P] * 7
    f.restype = C.c_int
    t, mat, prop = abi.initial_time(), abi.make_material(g["mat"]), abi.make_solid_prop(g["prop"])
    ptr = lambda k: P(a[k].data_ptr())
    args = (c["cycles"], C.byref(t), numnod, *map(ptr, ("x", "d", "v", "ms", "icodt")), nel,
            *map(ptr, ("conn", "iads", "adsky")), C.byref(mat), C.byref(prop), 0.9, 1e20, abi.DT_GROWTH_REF,
            *map(ptr, ("sig", "eint", "rho", "qvis", "pla", "epsd", "vol0")))
    return dict(case=c, call=f, args=args, arrays=a, keep=(t, mat, prop))


def _run_pool(s):
    rc = s["call"](0, C.c_void_p(torch.cuda.current_stream().cuda_stream), *s["args"])
    if rc:
        raise RuntimeError(f"or_ecycle_hex_step_noalloc: {abi.ERROR_NAMES.get(rc, rc)}")
    return {k: s["arrays"][k] for k in ("x", "d", "v", "sig", "eint", "rho", "qvis", "pla", "epsd")}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(c):
    """(hexas, hexa law 2 share, shells, points, nodes) of a case."""
    k = c["kind"]
    if k in ("block", "pool"):
        return c["nx"] * c["ny"] * c["nz"], c["law"] - 1, 0, 0, (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)
    if k in ("plate", "adjoint"):
        return 0, 0, c["n"] ** 2, c.get("points", 5), (c["n"] + 1) ** 2
    if k == "rail":
        rows, cols = 2 * round(0.03 / c["edge"]) + round(0.05 / c["edge"]), round(0.3 / c["edge"])
        return 0, 0, rows * cols, 3, (rows + 1) * (cols + 1)
    if k == "mixed":
        skin = 2 * (c["nx"] + c["ny"]) * c["nz"]
        return c["nx"] * c["ny"] * c["nz"], 1, skin, 5, (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)
    hexas = shells = nodes = 0
    for is_hex, _, nel in _sizes(c):
        if is_hex:
            n = _hexa_edge(nel)
            hexas, nodes = hexas + 4 * n ** 3, nodes + (n + 1) ** 2 * (4 * n + 1)
        else:
            n = _plate_edge(nel)
            shells, nodes = shells + n * n, nodes + (n + 1) ** 2
    return hexas, 0.5, shells, 5, nodes


ON_CHIP = 60e6      # bytes of state that registers and shared memory of the GPU could hold


def work(c):
    """State read and written once a cycle (once a pass where it could stay on the chip all along),
    the nodes read back once; floating-point operations of the elements and nodes in every cycle."""
    hexas, law2, shells, points, nodes = _counts(c)
    s = 4 if c.get("precision") == "split" else 8
    rot = shells > 0
    # hexa: 11 reals and the law's plastic strain in, 10 out, connectivity; shell: points x 6 in and out, 13 reals
    one = hexas * ((21 + 4 * law2) * s + 32) + shells * ((12 * points + 13) * s + 16) + \
        nodes * (97 + 7 * s + (7 * s if rot else 0))
    flops = hexas * 1300.0 + shells * (700.0 + 60.0 * points) + nodes * 40.0
    n, sweeps = c["cycles"], 1
    back = nodes * 24.0 * (2 if hexas else 3)
    if c["kind"] == "adjoint":      # forward, forward again from checkpoints with every state kept, reverse
        sweeps, back = 3, shells * 16.0 + nodes * 16.0
        flops *= 5.0 / 3.0          # the reverse element is about three forward ones
    if c["kind"] == "pool":
        back = 0.0
    return dict(bytes=back + one * (1 if one < ON_CHIP and sweeps == 1 else n * sweeps), flops=flops * n * sweeps)


# ---------------------------------------------------------------------------
# the same in 64 bits: plain torch
# ---------------------------------------------------------------------------
# COQINI's rules (coqini.F:45-130), REAL literals: positions, membrane weights, bending weights
RULES = {3: ((-.5, 0., .5), (.25, .5, .25), (-.0833333, 0., .0833333)),
         5: ((-.5, -.25, 0., .25, .5), (.125, .25, .25, .25, .125), (-.0520833, -.0625, 0., .0625, .0520833))}
PAIRS = ((0, 6), (1, 7), (2, 4), (3, 5))
MODES = ((1, -1, 1, -1, 1, -1, 1, -1), (1, 1, -1, -1, -1, -1, 1, 1), (1, -1, -1, 1, -1, 1, 1, -1),
         (1, -1, 1, -1, -1, 1, -1, 1))
FACES = ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7))


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a, least=0.0):
    r = torch.sqrt(_dot(a, a))[..., None]
    return a / r.clamp_min(least) if least else torch.where(r == 0, a, a / torch.where(r == 0, 1.0, r))


def _hexa(g, st, x, v, dt1):
    """SFORC3 of one group: corner forces to add (nel, 8, 3), new state, element step."""
    m, p = g["mat"], g["prop"]
    X, V = x[g["conn"]], v[g["conn"]]
    frame = None
    if p["jcvt"]:
        d = [X[:, b] - X[:, a] for a, b in PAIRS]
        a17, a28 = d[0] + d[3], d[1] + d[2]
        r, s, t = _unit(d[0] + d[1] - d[2] - d[3]), _unit(a17 + a28), _unit(a17 - a28)
        for _ in range(3):
            r, s, t = (_unit(torch.linalg.cross(s, t) + r), _unit(torch.linalg.cross(t, r) + s),
                       _unit(torch.linalg.cross(r, s) + t))
        e3 = _unit(torch.linalg.cross(r, s))
        frame = torch.stack([r, torch.linalg.cross(e3, r), e3], -1)          # columns e1 e2 e3
        X, V = X @ frame, V @ frame
    d = [X[:, b] - X[:, a] for a, b in PAIRS]
    j1 = d[0] + d[1] - d[2] - d[3]
    a, b = d[0] + d[3], d[1] + d[2]
    j4, j7 = a + b, a - b
    c1 = torch.linalg.cross(j4, j7)
    vol = _dot(j1, c1) / 64.0
    k = (1.0 / 64.0 / vol)[:, None]
    i1, i2, i3 = k * c1, k * torch.linalg.cross(j7, j1), k * torch.linalg.cross(j1, j4)
    # rows of the inverse Jacobian: PX, PY, PZ of the corners 1..4 (5..8 are the opposite ones')
    P = torch.stack([-i1 - i2 - i3, -i1 - i2 + i3, i1 - i2 + i3, i1 - i2 - i3], 1)      # (nel, 4, 3)
    sign = x.new_tensor(MODES)
    H = torch.einsum("jk,ekc->ejc", sign[:3], X)
    PH = torch.einsum("eqc,ejc->eqj", P, H)
    area = torch.full_like(vol, 1e-20)
    for f in FACES:
        x13, x24 = X[:, f[2]] - X[:, f[0]], X[:, f[3]] - X[:, f[1]]
        s, t = x13 - x24, x13 + x24
        area = torch.maximum(area, _dot(s, s) * _dot(t, t) - _dot(s, t) ** 2)
    length = 4.0 * vol / torch.sqrt(area)
    dv = torch.stack([V[:, a] - V[:, b] for a, b in PAIRS], 1)
    L = torch.einsum("eqi,eqj->eij", dv, P)                     # dv_i / dx_j
    gam = sign.expand(len(vol), 4, 8).clone()
    for q, (a, b) in enumerate(PAIRS):
        gam[:, :3, a] = gam[:, :3, a] - PH[:, q]
        gam[:, :3, b] = gam[:, :3, b] + PH[:, q]
    hg = torch.einsum("ejk,ekc->ejc", gam, V)
    dxx, dyy, dzz = L[:, 0, 0], L[:, 1, 1], L[:, 2, 2]
    d4, d5, d6 = L[:, 0, 1] + L[:, 1, 0], L[:, 1, 2] + L[:, 2, 1], L[:, 0, 2] + L[:, 2, 0]
    wzz, wyy, wxx = (0.5 * dt1 * w for w in (L[:, 1, 0] - L[:, 0, 1], L[:, 0, 2] - L[:, 2, 0], L[:, 2, 1] - L[:, 1, 2]))
    rho0, vol0 = m["rho0"], g["vol0"]
    dvol = vol - (rho0 / st["rho"]) * vol0
    rho = rho0 * (vol0 / vol)
    S = st["sig"]
    if p["jcvt"]:
        sg = list(S)
    else:
        q1, q2, q3 = 2 * S[3] * wzz, 2 * S[5] * wyy, 2 * S[4] * wxx
        sg = [S[0] - q1 + q2, S[1] + q1 - q3, S[2] - q2 + q3, S[3] + wzz * (S[0] - S[1]) + wyy * S[4] - wxx * S[5],
              S[4] + wxx * (S[1] - S[2]) + wzz * S[5] - wyy * S[3], S[5] + wyy * (S[2] - S[0]) + wxx * S[3] - wzz * S[4]]
    G = m["shear"]
    ssp = math.sqrt((1.333 * G + m["bulk"]) / rho0)
    mean, div = (sg[0] + sg[1] + sg[2]) / 3.0, (dxx + dyy + dzz) / 3.0
    for i, e in enumerate((dxx, dyy, dzz)):
        sg[i] = sg[i] - mean + 2 * dt1 * G * (e - div)
    for i, e in enumerate((d4, d5, d6)):
        sg[3 + i] = sg[3 + i] + dt1 * G * e
    pla, epsd = st["pla"], st["epsd"]
    if m["law"] == 2:
        aj2 = torch.sqrt(3.0 * (0.5 * (sg[0] ** 2 + sg[1] ** 2 + sg[2] ** 2) + sg[3] ** 2 + sg[4] ** 2 + sg[5] ** 2))
        epsd = torch.sqrt(dxx ** 2 + dyy ** 2 + dzz ** 2 + 0.5 * (d4 ** 2 + d5 ** 2 + d6 ** 2))
        ca, cb, cn = m["jc_a"], m["jc_b"], m["jc_n"]
        some = pla > 0
        safe = torch.where(some, pla, 1.0)
        ak = torch.where(some, ca + cb * safe ** cn, ca)
        qh = torch.where(some, cb * cn * safe ** (cn - 1.0), 0.0)
        scale = torch.clamp(ak / aj2.clamp_min(1e-15), max=1.0)
        dpla = (1.0 - scale) * aj2 / (3.0 * G + qh)
        ak = ak + dpla * qh
        scale = torch.clamp(ak / aj2.clamp_min(1e-15), max=1.0)
        sg = [scale * s for s in sg]
        pla = pla + dpla
    al = vol ** (1.0 / 3.0)
    ad = torch.clamp(-dxx - dyy - dzz, min=0.0)
    qaa = p["qa"] ** 2 * ad
    qx = p["qb"] * ssp + al * qaa
    qnew = rho * ad * al * (qaa * al + p["qb"] * ssp)
    step = 0.9 * length / (qx + torch.sqrt(qx * qx + ssp * ssp))
    pres = m["bulk"] * (vol0 / vol - 1.0)
    sg = [sg[0] - pres, sg[1] - pres, sg[2] - pres] + sg[3:]
    p2 = -(S[0] + sg[0] + S[1] + sg[1] + S[2] + sg[2]) / 3.0 if m["law"] == 1 else 0.0
    einc = (vol - 0.5 * dvol) * 0.5 * dt1 * (
        dxx * (S[0] + sg[0] + p2) + dyy * (S[1] + sg[1] + p2) + dzz * (S[2] + sg[2] + p2) +
        d4 * (S[3] + sg[3]) + d5 * (S[4] + sg[4]) + d6 * (S[5] + sg[5])) - 0.5 * dvol * (st["qvis"] + qnew + p2)
    eint = (st["eint"] * vol0 + einc) / vol0
    caq = 0.25 * p["qh"]
    fcl = caq * rho * al * al
    fcq, fcl = (fcl * caq * 100.0)[:, None, None], (fcl * ssp)[:, None, None]
    h = hg * (fcl + hg.abs() * fcq)
    F = -torch.einsum("ejk,ejc->ekc", gam, h)
    s1, s2, s3 = ((sg[i] - qnew) * vol for i in range(3))
    s4, s5, s6 = (sg[i] * vol for i in (3, 4, 5))
    T = torch.stack([s1, s4, s6, s4, s2, s5, s6, s5, s3], -1).reshape(-1, 3, 3)
    f = torch.einsum("eij,eqj->eqi", T, P)
    for q, (a, b) in enumerate(PAIRS):
        F[:, a] -= f[:, q]
        F[:, b] += f[:, q]
    if frame is not None:
        F = F @ frame.transpose(1, 2)
    return F, dict(sig=torch.stack(sg), eint=eint, rho=rho, qvis=qnew, pla=pla, epsd=epsd), step.min()


def _shell(g, st, x, v, w, dt1):
    """CFORC3 of one group (Ishell 1): corner forces and moments to add, new state, element step."""
    m, p = g["mat"], g["prop"]
    X, V, W = x[g["conn"]], v[g["conn"]], w[g["conn"]]
    d21, d31, d41 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0], X[:, 3] - X[:, 0]
    d32, d34 = X[:, 2] - X[:, 1], X[:, 2] - X[:, 3]
    e1, e2 = d21 + d34, d32 + d41
    e3 = torch.linalg.cross(e1, e2)
    if p["ishfram"] == 2:
        e1 = _unit(e1 * _dot(e2, e2)[:, None] + torch.linalg.cross(e2, e3), 1e-20)
        e3 = _unit(e3, 1e-20)
        e2 = _unit(torch.linalg.cross(e3, e1), 1e-20)
    else:
        e3 = _unit(e3, 1e-20)
        e1 = _unit(e1 + torch.linalg.cross(e2, e3) * torch.sqrt(_dot(e1, e1) / _dot(e2, e2))[:, None], 1e-20)
        e2 = torch.linalg.cross(e3, e1)
    E = torch.stack([e1, e2, e3], -1)
    x2, y2, x3, y3, x4, y4 = (_dot(e, d) for d in (d21, d31, d41) for e in (e1, e2))
    px1, py1, px2, py2 = 0.5 * (y2 - y4), 0.5 * (x4 - x2), 0.5 * y3, -0.5 * x3
    area = (2.0 * (py2 * px1 - py1 * px2)).clamp_min(1e-20)
    vhx, vhy = (-x2 + x3 - x4) / area, (-y2 + y3 - y4) / area
    thk = st["thk"] if p["ithk"] > 0 else g["thke"]
    nu, G, ym, shf = m["nu"], m["shear"], m["young"], p["shf"]
    with torch.no_grad():       # CDLEN3 / CDT3: the step is the same for every design
        al = [x2 ** 2 + y2 ** 2, (x3 - x2) ** 2 + (y3 - y2) ** 2, (x4 - x3) ** 2 + (y4 - y3) ** 2, x4 ** 2 + y4 ** 2,
              (x4 - x2) ** 2 + (y4 - y2) ** 2, x3 ** 2 + y3 ** 2]
        least = torch.stack(al).amin(0)
        size = torch.maximum(area ** 2 / torch.maximum(al[4], al[5]), least)
        size = torch.minimum(size, 0.5 * (least + size) / max(p["hm"], p["hf"]))
        step = (0.9 * torch.sqrt(size) / m["ssp_shell"]).min()
    Vl, Wl = V @ E, W @ E
    vx, vy, vz = (Vl[:, :, i] for i in range(3))
    rx, ry = Wl[:, :, 0], Wl[:, :, 1]
    vz13, vz24 = vz[:, 0] - vz[:, 2], vz[:, 1] - vz[:, 3]
    exz, eyz = px1 * vz13 + px2 * vz24, py1 * vz13 + py2 * vz24
    away = lambda a: torch.copysign(a.abs().clamp_min(1e-20), a)
    t1 = 0.25 * dt1 * (vz13 - vz24) ** 2 / away(py2 + py1)
    t2 = 0.25 * dt1 * (vz13 + vz24) ** 2 / away(px2 - px1)
    vx13, vx24 = vx[:, 0] - vx[:, 2] - t1, vx[:, 1] - vx[:, 3] + t1
    vy13, vy24 = vy[:, 0] - vy[:, 2] + t2, vy[:, 1] - vy[:, 3] + t2
    rx13, rx24, ry13, ry24 = rx[:, 0] - rx[:, 2], rx[:, 1] - rx[:, 3], ry[:, 0] - ry[:, 2], ry[:, 1] - ry[:, 3]
    fac = dt1 / area
    exx, eyy = fac * (px1 * vx13 + px2 * vx24), fac * (py1 * vy13 + py2 * vy24)
    exy = fac * (py1 * vx13 + py2 * vx24 + px1 * vy13 + px2 * vy24)
    exz, eyz = fac * (exz + 0.25 * area * ry.sum(1)), fac * (eyz - 0.25 * area * rx.sum(1))
    kxx, kyy = fac * (px1 * ry13 + px2 * ry24), fac * (-py1 * rx13 - py2 * rx24)
    kxy = fac * (py1 * ry13 + py2 * ry24 - px1 * rx13 - px2 * rx24)
    z0, wf, wm = (x.new_tensor(np.float32(r).astype(np.float64))[:, None] for r in RULES[p["npt"]])
    dx, dy, dxy = (a + z0 * thk * b for a, b in ((exx, kxx), (eyy, kyy), (exy, kxy)))
    S = st["sig"]                                               # (points, 5, nel)
    a1, a2 = ym / (1.0 - nu * nu), nu * ym / (1.0 - nu * nu)
    sx, sy, sxy = S[:, 0] + a1 * dx + a2 * dy, S[:, 1] + a2 * dx + a1 * dy, S[:, 2] + G * dxy
    syz, szx = S[:, 3] + G * shf * eyz, S[:, 4] + G * shf * exz
    pla = st["pla"]
    ezz = -nu * (dx + dy) / (1.0 - nu)
    if m["law"] == 2:
        ca, cb, cn, cap = st["jc_a"], m["jc_b"], m["jc_n"], m["sigmax"]
        hard = lambda e: torch.where(e > 0, ca + cb * torch.exp(cn * torch.log(torch.where(e > 0, e, 1.0))), ca + 0 * e)
        yld = hard(pla).clamp_max(cap)
        svm2 = sx * sx + sy * sy - sx * sy + 3.0 * sxy * sxy
        flows = svm2 > yld * yld
        if p["ipla"] == 0:
            svm = torch.sqrt(torch.where(flows, svm2, yld * yld))
            rr = torch.where(flows, yld / (svm + 1e-15), 1.0)
            sx, sy, sxy = sx * rr, sy * rr, sxy * rr
            dpla = torch.where(flows, (svm - yld) / ym, 0.0)
            pla = pla + dpla
            ezp = dpla * 0.5 * (sx + sy) / yld
            st = dict(st, work=st["work"] + (yld * dpla * area * wf * thk).sum())
        else:                   # Newton, three iterations (m2cplr.F:231-378)
            A, B = 0.25 * (sx + sy) ** 2, 0.75 * (sx - sy) ** 2 + 3.0 * sxy ** 2
            svm = torch.sqrt(A + B)
            n1, n2 = 1.0 / (1.0 - nu), 1.0 / (1.0 + nu)
            h = torch.where(yld >= cap, 0.0, cn * cb * torch.exp((cn - 1.0) * torch.log(pla + 1e-7)))
            dj = (svm - yld) / (3.0 * G + h)
            for _ in range(3):
                di = dj
                yi = hard(pla + di).clamp_max(cap)
                dr = 0.5 * ym * di / yi
                P, Q = 1.0 / (1.0 + dr * n1), 1.0 / (1.0 + 3.0 * dr * n2)
                f = A * P * P + B * Q * Q - yi * yi
                df = -(A * n1 * P ** 3 + 3.0 * B * n2 * Q ** 3) * (ym - dr * 2.0 * h) / yi - 2.0 * h * yi
                dj = torch.where(di > 0, (di - f / df).clamp_min(0.0), 0.0)
            t1, t2 = (sx + sy) * P, (sx - sy) * Q
            sx, sy = torch.where(flows, 0.5 * (t1 + t2), sx), torch.where(flows, 0.5 * (t1 - t2), sy)
            sxy = torch.where(flows, sxy * Q, sxy)
            pla = torch.where(flows, pla + di, pla)
            ezp = torch.where(flows, dr * t1 / ym, 0.0)
        ezz = (-(dx + dy) * nu - (1.0 - 2.0 * nu) * ezp) / (1.0 - nu)
    sig = torch.stack([sx, sy, sxy, syz, szx], 1)
    thn = (st["thk"] + (ezz * wf * thk).sum(0)).clamp_min(1e-30)
    N, M = (wf[..., None] * sig.transpose(1, 2)).sum(0).T, (wm[..., None] * sig.transpose(1, 2)).sum(0).T
    # CHVIS3
    a, b = px1 * vhx + py1 * vhy, px2 * vhx + py2 * vhy
    gam = torch.stack([1.0 - a, -1.0 - b, 1.0 + a, -1.0 + b], 1)
    sh3 = shf / (3.0 * (1.0 + nu))
    r1 = 25.0 * m["rho0"]
    h1q = r1 * 0.5 * p["hm"] * thk * torch.sqrt(area)
    h2q = r1 * 0.5 * p["hf"] * math.sqrt(sh3) * thk ** 2
    h3q = 0.5 * p["hr"] * r1 * 0.072169 * thk ** 2 * area
    hh1 = p["hm"] * 0.125 * ym * thk * dt1
    hh2 = p["hf"] * 0.125 * ym * sh3 * thk ** 3 * dt1 / (px1 ** 2 + py1 ** 2 + px2 ** 2 + py2 ** 2)
    rates = [_dot(c, gam) for c in (vx, vy, vz)]
    hour = [st["hourg"][i] + rates[i] * k for i, k in enumerate((hh1, hh1, hh2))]
    full = [(hour[i] + rates[i] * q * rates[i].abs())[:, None] * gam for i, q in enumerate((h1q, h1q, h2q))]
    alt = x.new_tensor([1.0, -1.0, 1.0, -1.0])
    g4, g5 = _dot(rx, alt), _dot(ry, alt)
    h4, h5 = g4 * h3q * g4.abs(), g5 * h3q * g5.abs()
    # CFINT3
    f1, f2, f3, f4, f5 = (N[i] * thk for i in range(5))
    m4, m5 = 0.25 * f4 * area, 0.25 * f5 * area
    corner = lambda a, b, h: torch.stack([a + h[:, 0], b + h[:, 1], h[:, 2] - a, -a - b - (h[:, 0] + h[:, 1] + h[:, 2]) + a],
                                         1)
    F = torch.stack([corner(f1 * px1 + f3 * py1, f1 * px2 + f3 * py2, full[0]),
                     corner(f2 * py1 + f3 * px1, f2 * py2 + f3 * px2, full[1]),
                     corner(f5 * px1 + f4 * py1, f5 * px2 + f4 * py2, full[2])], -1) @ E.transpose(1, 2)
    k1, k2, k3 = (M[i] * thk ** 2 for i in range(3))
    ends = lambda a, b, c, h: torch.stack([a + c + h, b + c - h, -a + c + h, -b + c - h], 1)
    ml = torch.stack([ends(-k2 * py1 - k3 * px1, -k2 * py2 - k3 * px2, -m4, h4),
                      ends(k1 * px1 + k3 * py1, k1 * px2 + k3 * py2, m5, h5)], -1)
    Mo = ml @ E[:, :, :2].transpose(1, 2)
    load = -p["pressure"] * 0.125 * torch.linalg.cross(X[:, 2] - X[:, 0], X[:, 3] - X[:, 1])
    return -F + load[:, None], -Mo, dict(st, sig=sig, pla=pla, thk=thn, hourg=torch.stack(hour)), step


def _part_model(p, device):
    """A part's arrays and groups on the device, FP64."""
    put = lambda a: torch.tensor(np.asarray(a, np.float64), device=device)
    ind = lambda a: torch.tensor(np.asarray(a, np.int64), device=device)
    free = lambda code: put(np.stack([(np.asarray(code) & b) == 0 for b in (4, 2, 1)], 1))
    model = dict(ms=put(p["ms"]), inr=put(p["inr"]), free=free(p["icodt"]), free_r=free(p["icodr"]), hex=[], shell=[],
                 links=[ind(r["nodes"]) for r in p.get("rlinks", [])])
    state = dict(x=put(p["x"]), d=put(np.zeros_like(p["x"])), v=put(p["v"]), w=put(p["vr"]), groups=[],
                 dt2=0.0, dt2old=1e30)
    for g in p["hex"]:
        nel = g["ixs"].shape[0]
        model["hex"].append(dict(conn=ind(g["ixs"][:, 1:9] - 1), vol0=put(g["vol0"]), mat=g["mat"], prop=g["prop"]))
        zero = put(np.zeros(nel))
        state["groups"].append(dict(sig=put(np.zeros((6, nel))), eint=zero, rho=zero + g["mat"]["rho0"], qvis=zero,
                                    pla=zero, epsd=zero))
    for g in p["shell"]:
        nel, npt = g["ixc"].shape[0], g["prop"]["npt"]
        thke = put(np.full(nel, g["prop"]["thk"]) if g.get("thke") is None else g["thke"])
        jc_a = put(np.full(nel, g["mat"]["jc_a"]) if g.get("jc_a") is None else g["jc_a"])
        model["shell"].append(dict(conn=ind(g["ixc"][:, 1:5] - 1), thke=thke, mat=g["mat"], prop=g["prop"]))
        state["groups"].append(dict(sig=put(np.zeros((npt, 5, nel))), pla=put(np.zeros((npt, nel))), thk=thke,
                                    hourg=put(np.zeros((3, nel))), jc_a=jc_a, work=put(0.0)))
    return model, state


def _cycle(model, s, dtmx):
    """One explicit cycle: elements, assembly, time step, nodes."""
    x, v, w, dt1 = s["x"], s["v"], s["w"], s["dt2"]
    f, mo = torch.zeros_like(x), torch.zeros_like(x)
    steps, groups = [], []
    nh = len(model["hex"])
    for g, st in zip(model["hex"], s["groups"][:nh]):
        F, new, step = _hexa(g, st, x, v, dt1)
        f = f.index_add(0, g["conn"].reshape(-1), F.reshape(-1, 3))
        groups.append(new)
        steps.append(step)
    for g, st in zip(model["shell"], s["groups"][nh:]):
        F, M, new, step = _shell(g, st, x, v, w, dt1)
        f = f.index_add(0, g["conn"].reshape(-1), F.reshape(-1, 3))
        mo = mo.index_add(0, g["conn"].reshape(-1), M.reshape(-1, 3))
        groups.append(new)
        steps.append(step)
    dt2 = min(1e6, float(torch.stack(steps).min()), float(np.float32(1.1)) * s["dt2old"], dtmx)
    dt12 = 0.5 * (dt1 + dt2)
    div = lambda a, b: torch.where(b[:, None] > 0, a / torch.where(b > 0, b, 1.0)[:, None], 0.0)
    a, ar = div(f, model["ms"]) * model["free"], div(mo, model["inr"]) * model["free_r"]
    for nodes in model["links"]:            # rigid velocity links, all translations
        ms = model["ms"][nodes, None]
        a = a.clone()
        a[nodes] = (ms * a[nodes]).sum(0) / ms.sum() * model["free"][nodes]
    v = v * model["free"] + dt12 * a
    w = w * model["free_r"] + dt12 * ar
    u = dt2 * v
    return dict(x=x + u, d=s["d"] + u, v=v, w=w, groups=groups, dt2=dt2, dt2old=dt2)


def exact(c, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    hexas, _, shells, points, _ = _counts(c)
    cost = (hexas + shells * (1 + points) / 2.0) * c["cycles"]
    if cost > (3e9 if device == "cuda" else 2e6) or (c["kind"] == "adjoint" and device == "cpu"):
        return None
    d = make_deck(c, seed)
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, d, device)
    ends = []
    with torch.no_grad():
        for p in d["parts"]:
            model, s = _part_model(p, device)
            for _ in range(c["cycles"] + (LEAD if c["kind"] == "rail" else 0)):
                s = _cycle(model, s, d["dtmx"])
            ends.append({k: s[k].cpu() for k in ("x", "d", "v", "w")})
    out = {k: torch.cat([e[k] for e in ends]) for k in ("x", "d", "v", "w")}
    first = {k: a.cpu() for k, a in s["groups"][0].items()}
    if c["kind"] == "pool":
        return dict(x=out["x"], d=out["d"], v=out["v"], **first)
    got = dict(d=out["d"], v=out["v"])
    if not hexas:
        got["vr"] = out["w"]
    if c["kind"] == "block" and c["precision"] == "fp64":
        got.update(first)
    return got


def _exact_adjoint(c, d, device):
    """The forward run cycle by cycle, each recomputed in the reverse sweep."""
    model, s = _part_model(d["parts"][0], device)
    leaf = lambda a: a.clone().requires_grad_(True)
    st = s["groups"][0]
    ms, inr, thk, jc_a = leaf(model["ms"]), leaf(model["inr"]), leaf(st["thk"]), leaf(st["jc_a"])

    def one(dt2, dt2old, x, dd, v, w, sig, pla, t, hourg, work, ms, inr, ca):
        now = dict(x=x, d=dd, v=v, w=w, dt2=dt2, dt2old=dt2old,
                   groups=[dict(sig=sig, pla=pla, thk=t, hourg=hourg, jc_a=ca, work=work)])
        e = _cycle(dict(model, ms=ms, inr=inr), now, d["dtmx"])
        g = e["groups"][0]
        return (e["dt2"], e["x"], e["d"], e["v"], e["w"], g["sig"], g["pla"], g["thk"], g["hourg"], g["work"])

    cur = [s["x"], s["d"], s["v"], s["w"], st["sig"], st["pla"], thk, st["hourg"], st["work"]]
    dt2, dt2old = s["dt2"], s["dt2old"]
    for _ in range(c["cycles"]):
        dt2, *cur = checkpoint(one, dt2, dt2old, *cur, ms, inr, jc_a, use_reentrant=False)
        dt2old = dt2
    J = cur[1][adjoint.centre_node(d), 2] + W_PLASTIC * cur[-1]
    g = torch.autograd.grad(J, (jc_a, thk, ms, inr))
    return dict(J=float(J.detach()), **{k: a.cpu() for k, a in zip(("dA", "dthk", "dms", "din"), g)})
