"""Performance cases of the D3Q19 stream-and-collide framework.

Each case is a call that a program using ``freelb_b200`` makes: so many time
steps of a lattice that it holds, the output and convergence calls between
them, or a gradient.  ``listed`` has the fixed cases, ``draw`` more of the same
ranges; ``exact`` restates a case in 64 bits with plain torch.
"""
import ctypes
import math

import numpy as np
import torch

import freelb_b200 as F
from freelb_b200 import _capi, geometry

# D3Q19 in the framework's order: rest, 6 axis, 12 diagonal; the opposite of odd i is i + 1
VEL = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
       (1, 1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, -1, -1),
       (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]
WEIGHT = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [0] + [i + 1 if i % 2 else i - 1 for i in range(1, 19)]
ELEM = {"fp32": 4, "fp16s": 2, "fp64": 8, "fp32s": 4}
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases

def cavity(name, nx, ny, nz, steps, storage="fp32", model="bgk", graph=False, autotune=False):
    return {"name": name, "kind": "cavity", "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "storage": storage, "model": model, "graph": graph, "autotune": autotune}


def listed():
    return [
        # a small cavity stepped on its way to an answer in seconds: launches count
        cavity("cavity 30 fp32 bgk", 30, 30, 30, 200, graph=True),
        # the cavity benchmark's own shape
        cavity("cavity 100 fp32 bgk", 100, 100, 100, 100),
        # the headline size in both storages, with the launch shape tuned as the benchmark does
        cavity("cavity 512 fp32 bgk", 512, 512, 512, 20, autotune=True),
        cavity("cavity 512 fp16s bgk", 512, 512, 512, 20, storage="fp16s", autotune=True),
        # the 256^3 configuration with the moment-space collision (stochastic rounding)
        cavity("cavity 256 fp16s mrt", 256, 256, 256, 20, storage="fp16s", model="mrt"),
        # a box whose rows are not a multiple of any tile or vector, with the turbulence model
        cavity("box 317 fp32 les", 317, 203, 121, 20, model="les"),
        # the accuracy reference of the other storages
        cavity("box 141 fp64 bgk", 141, 160, 118, 10, storage="fp64"),
        # a domain of uneven blocks with their device halos
        {"name": "blocks 256 fp32 bgk", "kind": "blocks", "ni": 256, "steps": 10,
         "storage": "fp32", "model": "bgk", "bseed": 0},
        # a parameter study: independent cavities stepped together
        {"name": "ensemble 48 fp32 bgk", "kind": "ensemble", "count": 48, "lo": 32, "hi": 128,
         "steps": 20, "storage": "fp32", "bseed": 0},
        # the gradient of an objective by the porosity field, tau and the lid velocity
        {"name": "adjoint 128 fp32s", "kind": "adjoint", "ni": 128, "steps": 40, "every": 10,
         "storage": "fp32s"},
        # half-way walls: boundary managers are applied after every single step
        {"name": "halfway 96 fp32 bgk", "kind": "halfway", "nx": 96, "ny": 96, "nz": 96,
         "steps": 40, "storage": "fp32"},
        # between outputs: some steps, then fields, conservation sums and the convergence check
        {"name": "monitor 200 fp32 bgk", "kind": "monitor", "nx": 200, "ny": 200, "nz": 200,
         "steps": 4, "storage": "fp32", "model": "bgk"},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity"] * 6 + ["blocks", "ensemble", "adjoint", "halfway", "monitor"])
    storage = rng.choice(["fp32", "fp32", "fp32", "fp16s", "fp16s", "fp64", "fp32s"])
    if kind in ("cavity", "halfway", "monitor"):
        top = 350 if kind == "cavity" else 220
        while True:
            n = [log_int(rng, 10, top) for _ in range(3)]
            if n[0] * n[1] * n[2] <= 3e7:
                break
        cells = n[0] * n[1] * n[2]
        case = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "storage": storage}
        if kind == "halfway":
            return dict(case, steps=log_int(rng, 10, 60))
        case["model"] = rng.choice(["bgk", "bgk", "mrt", "les"])
        if kind == "monitor":
            return dict(case, steps=log_int(rng, 1, 20))
        return dict(case, steps=log_int(rng, 4, min(200, max(8, 8e8 / cells))),
                    graph=rng.random() < 0.3, autotune=False)
    if kind == "blocks":
        return {"kind": kind, "ni": rng.choice([96, 128, 160, 192]), "steps": log_int(rng, 4, 20),
                "storage": rng.choice(["fp32", "fp32", "fp16s", "fp64"]),
                "model": rng.choice(["bgk", "mrt", "les"]), "bseed": rng.randrange(1000)}
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randrange(4, 49), "lo": 32,
                "hi": rng.randrange(48, 129), "steps": log_int(rng, 5, 40),
                "storage": rng.choice(["fp32", "fp16s"]), "bseed": rng.randrange(1000)}
    every = rng.randrange(2, 12)
    return {"kind": "adjoint", "ni": rng.randrange(24, 129), "steps": every * rng.randrange(1, 5),
            "every": every, "storage": rng.choice(["fp32s", "fp32s", "fp32", "fp64"])}


# ---------------------------------------------------------------------------
# geometry shared by the framework's runs and the 64-bit restatement

def tau_of(case):
    if case["kind"] == "adjoint":
        return 3 * 0.1 * case["ni"] / 500 + 0.5
    return 0.51 if case.get("model") == "les" else 0.53


def blocks_of(case):
    """The blocks of a case: (nx, ny, nz, ox, oy, oz, tau) with their overlap layer."""
    tau = tau_of(case)
    if case["kind"] == "blocks":
        b = geometry.uneven_blocks(case["ni"], edges=(32, 48, 64, 96), seed=case["bseed"])
        return [t + (tau,) for t in geometry.block_tuples(b)]
    if case["kind"] == "ensemble":
        rng = np.random.default_rng(case["bseed"])
        size = rng.integers(case["lo"], case["hi"] + 1, size=case["count"])
        re = np.exp(rng.uniform(math.log(100.0), math.log(3000.0), size=case["count"]))
        return [(int(n) + 2,) * 3 + (0, 0, 0, 3 * 0.1 * int(n) / r + 0.5)
                for n, r in zip(size, re)]
    n = (case["ni"],) * 3 if "ni" in case else (case["nx"], case["ny"], case["nz"])
    return [tuple(v + 2 for v in n) + (0, 0, 0, tau)]


def box_flags(nx, ny, nz):
    """Cavity flags of an nx x ny x nz stored mesh: 1 void, 2 fluid, 4 wall, 8 lid."""
    f = np.ones((nz, ny, nx), dtype=np.uint8)
    f[1:-1, 1:-1, 1:-1] = 4
    f[2:-2, 2:-2, 2:-2] = 2
    f[-2, 2:-2, 2:-2] = 8
    return f


def block_flags(case, blocks):
    if case["kind"] != "blocks":
        return [box_flags(*b[:3]) for b in blocks]
    g = box_flags(*(case["ni"] + 2,) * 3)
    return [np.ascontiguousarray(g[b[5]:b[5] + b[2], b[4]:b[4] + b[1], b[3]:b[3] + b[0]])
            for b in blocks]


def lid_velocity(seed):
    return 0.08 + 0.04 * np.random.default_rng(seed).random()


def flow(b, seed):
    """A smooth flow of the seed on block b (its global position counts): rho, (ux, uy, uz)."""
    rng = np.random.default_rng(seed)
    axes = [torch.arange(n, dtype=torch.float64, device=DEV) + o
            for n, o in zip(b[:3], b[3:6])]
    x, y, z = axes[0][None, None, :], axes[1][None, :, None], axes[2][:, None, None]

    def field(amp):
        out = torch.zeros(b[2], b[1], b[0], dtype=torch.float64, device=DEV)
        for _ in range(2):
            k = rng.uniform(0.02, 0.2, 3)
            out += amp * torch.cos(k[0] * x + rng.uniform(0, 6.28)) * \
                torch.cos(k[1] * y + rng.uniform(0, 6.28)) * \
                torch.cos(k[2] * z + rng.uniform(0, 6.28))
        return out
    return 1.0 + field(0.01), [field(0.03) for _ in range(3)]


def equilibrium(i, rho, u):
    cu = sum(c * v for c, v in zip(VEL[i], u) if c) if i else 0.0
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    return WEIGHT[i] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * u2)


def stored(f, i, storage):
    """Population i as the storage holds it, and back."""
    if storage == "fp16s":
        return ((f - WEIGHT[i]) * 1024.0).to(torch.float16)
    if storage == "fp32s":
        return (f - WEIGHT[i]).to(torch.float32)
    return f.to(torch.float64 if storage == "fp64" else torch.float32)


def as_f64(v, i, storage):
    v = v.to(torch.float64)
    return v / 1024.0 + WEIGHT[i] if storage == "fp16s" else v + WEIGHT[i] \
        if storage == "fp32s" else v


# ---------------------------------------------------------------------------
# prepare and run

class _Device:
    """Device memory of a lattice for torch, without a copy; a tensor made of it keeps the
    lattice."""

    def __init__(self, lat, ptr, shape, strides, typestr):
        self.lat = lat
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape,
                                         "strides": strides, "typestr": typestr, "version": 3}


def device_view(lat, ptr, shape, strides, typestr):
    size = int(typestr[2:])
    return torch.as_tensor(_Device(lat, ptr, shape, tuple(s * size for s in strides), typestr),
                           device=DEV)


def pointers(lat):
    """Device addresses of the current populations, flags, RHO and VELOCITY."""
    p = [ctypes.c_void_p() for _ in range(4)]
    _capi.call("flb_device_pointers", lat._h, *[ctypes.byref(v) for v in p])
    return [v.value for v in p]


def places(lat, real):
    """(base, pitch, plane) of every block in the lattice's arrays, read off marks that are put
    into its RHO field."""
    if lat.nblocks == 1:
        lo = lat.layout()
        return [(0, lo.pitch_x, lo.plane)]
    stride = lat.layout().dir_stride
    rho = device_view(lat, pointers(lat)[2], (stride,), (1,), real)
    out = []
    for k, (nx, ny, nz) in enumerate(lat.shapes):
        marks = np.zeros((nz, ny, nx), dtype=lat.real)
        marks[0, 0, 0], marks[0, 1, 0], marks[1, 0, 0] = 2, 3, 4
        lat.upload_field("rho", marks, block=k)
        at = [int(torch.nonzero(rho == v)[0, 0]) for v in (2, 3, 4)]
        out.append((at[0], at[1] - at[0], at[2] - at[0]))
        lat.upload_field("rho", np.ones_like(marks), block=k)
    return out


class State:
    """A lattice with the seed's flow in it, and views of what a pass returns."""

    def __init__(self, case, seed):
        self.case = case
        kind, storage = case["kind"], case["storage"]
        self.blocks = blocks_of(case)
        kw = {"storage": storage, "model": case.get("model", "bgk")}
        if kind == "adjoint":
            kw["model"] = "brinkman"
        if kind == "halfway":
            kw["tasks"] = ((2 | 4 | 8, "bulk"),)
        if kind in ("blocks", "ensemble"):
            # a halo block takes the lattice's tau, an independent one its own
            self.lat = F.Lattice.blocks([b[:6] + (1.0 / b[6],) for b in self.blocks],
                                        self.blocks[0][6],
                                        mode="halo" if kind == "blocks" else "independent", **kw)
        else:
            self.lat = F.Lattice(*self.blocks[0][:3], self.blocks[0][6], **kw)
        lat = self.lat
        self.real = "<f8" if storage == "fp64" else "<f4"
        self.elem = {"fp32": "<f4", "fp16s": "<f2", "fp64": "<f8", "fp32s": "<f4"}[storage]
        self.stride = lat.layout().dir_stride
        flags = block_flags(case, self.blocks)
        for k, f in enumerate(flags):
            lat.upload_flags(f, block=k)
        if case.get("autotune") or kind == "ensemble":
            lat.autotune(trial_steps=2)
        self.places = places(lat, self.real)
        self.views = {}
        ulid = lid_velocity(seed)
        vel = pointers(lat)[3]
        for k, (b, f) in enumerate(zip(self.blocks, flags)):
            rho, u = flow(b, seed)
            for i, v in enumerate(self.pops()[k]):
                v.copy_(stored(equilibrium(i, rho, u), i, storage))
            del rho, u
            base, pitch, plane = self.places[k]
            ux = device_view(lat, vel + base * int(self.real[2:]), (b[2], b[1], b[0]),
                             (plane, pitch, 1), self.real)
            ux.copy_(torch.from_numpy(f).to(DEV) == 8)
            ux *= ulid
        if kind == "adjoint":
            lat.upload_field("alpha", alpha_of(case, seed).astype(lat.real))
        if kind == "halfway":
            self.walls = [F.BounceBackManager(lat, 4, 1, kind="normal"),
                          F.BounceBackManager(lat, 8, 1, kind="movingwall")]

    def pops(self):
        """The current populations of every block, [19, nz, ny, nx] each, as stored."""
        ptr = pointers(self.lat)[0]
        if ptr not in self.views:
            size = int(self.elem[2:])
            self.views[ptr] = [device_view(self.lat, ptr + base * size, (19, b[2], b[1], b[0]),
                                           (self.stride, plane, pitch, 1), self.elem)
                               for b, (base, pitch, plane) in zip(self.blocks, self.places)]
        return self.views[ptr]

    def fields(self):
        b, (base, pitch, plane) = self.blocks[0], self.places[0]
        _, _, rho, vel = pointers(self.lat)
        return [device_view(self.lat, rho, (b[2], b[1], b[0]), (plane, pitch, 1),
                            self.real),
                device_view(self.lat, vel, (3, b[2], b[1], b[0]), (self.stride, plane, pitch, 1),
                            self.real)]


def alpha_of(case, seed):
    n = case["ni"] + 2
    return np.random.default_rng(seed + 1).uniform(0.0, 0.05, size=n ** 3).astype(np.float32)


def prepare(case, seed):
    return State(case, seed)


def run(state):
    case, lat = state.case, state.lat
    if case["kind"] == "adjoint":
        objective = lat.adjoint_forward(case["steps"], case["every"])
        alpha, tau, ulid = lat.adjoint_backward()
        return {"objective": objective, "alpha": alpha, "tau": tau, "ulid": ulid,
                "pops": state.pops()}
    if case["kind"] == "halfway":
        for _ in range(case["steps"]):
            lat.step(1)
            for wall in state.walls:
                wall.apply()
        return {"pops": state.pops()}
    lat.step(case["steps"], graph=case.get("graph", case["kind"] == "ensemble"))
    if case["kind"] == "monitor":
        lat.compute_rhou(key=2)
        sums = lat.conservation(key=2)
        change = lat.tolerance_u(key=2)
        return {"pops": state.pops(), "fields": state.fields(), "sums": sums, "change": change}
    return {"pops": state.pops()}


# ---------------------------------------------------------------------------
# what a pass needs, and how close it has to come

def cells_of(case):
    return sum(b[0] * b[1] * b[2] for b in blocks_of(case))


def work(case):
    """The populations read once and written once however many steps a pass has (and the fields
    that it writes), and the arithmetic of all its steps."""
    cells, size = cells_of(case), ELEM[case["storage"]]
    flops = {"bgk": 250, "mrt": 400, "les": 330}[case.get("model", "bgk")]
    nbytes = cells * (2 * 19 * size + 1)
    if case["kind"] == "adjoint":
        return {"bytes": nbytes + cells * (size + 8), "flops": cells * case["steps"] * 3 * flops}
    if case["kind"] == "monitor":
        nbytes += cells * 4 * max(size, 4)
    return {"bytes": nbytes, "flops": cells * case["steps"] * flops}


def tolerance(case):
    """Four times what a pass differs by from its 64-bit restatement or from other orders of its
    sums: a few roundings of the storage a step, relative to the populations (FP32, FP64) or to
    their deviations from rest (FP32S, FP16S)."""
    storage = case["storage"]
    if storage == "fp16s":
        return {"rel": 2e-3, "max": 0.05}
    if case["kind"] == "adjoint":
        return {"fp64": {"rel": 1e-12, "max": 1e-9}, "fp32s": {"rel": 6e-5, "max": 2e-3},
                "fp32": {"rel": 5e-4, "max": 2e-2}}[storage]
    if storage == "fp64":
        return {"rel": 2e-14, "max": 1e-12}
    if storage == "fp32s":
        return {"rel": 5e-6, "max": 5e-4}
    return {"rel": 1.2e-5, "max": 1e-3}


# ---------------------------------------------------------------------------
# the 64-bit restatement: R holds the populations after streaming, P the ones before it

def moment_basis():
    rows = []
    for x, y, z in VEL:
        c = x * x + y * y + z * z
        rows.append([1, 19 * c - 30, (21 * c * c - 53 * c + 24) / 2, x, (5 * c - 9) * x, y,
                     (5 * c - 9) * y, z, (5 * c - 9) * z, 3 * x * x - c,
                     (3 * c - 5) * (3 * x * x - c), y * y - z * z, (3 * c - 5) * (y * y - z * z),
                     x * y, y * z, x * z, x * (y * y - z * z), y * (z * z - x * x),
                     z * (x * x - y * y)])
    return torch.tensor(rows, dtype=torch.float64, device=DEV).T


def shift_of(i, nx, ny):
    return VEL[i][0] + nx * (VEL[i][1] + ny * VEL[i][2])


def stream(P, nx, ny):
    return [torch.roll(p, shift_of(i, nx, ny)) for i, p in enumerate(P)]


def moments(R, alpha=None):
    rho = sum(R)
    mom = [sum(VEL[i][a] * R[i] for i in range(19) if VEL[i][a]) for a in range(3)]
    den = rho if alpha is None else rho + 0.5 * alpha
    return rho, [m / den for m in mom]


def relax(R, model, omega, alpha=None):
    rho, u = moments(R, alpha)
    if model == "mrt":
        M = moment_basis()
        rate = torch.full((19,), 1.2, dtype=torch.float64, device=DEV)
        rate[[0, 3, 5, 7]] = 0.0
        rate[[9, 11, 13, 14, 15]] = omega
        A = M.T @ torch.diag(rate / (M * M).sum(1)) @ M
        out = [r.clone() for r in R]
        for j in range(19):
            n = R[j] - equilibrium(j, rho, u)
            for i in range(19):
                out[i] -= A[i, j] * n
        return out
    if model == "les":
        total = 0.0
        for a in range(3):
            for b in range(a, 3):
                pi = sum(VEL[i][a] * VEL[i][b] * R[i] for i in range(19)
                         if VEL[i][a] * VEL[i][b]) - rho * u[a] * u[b]
                if a == b:
                    pi = pi - rho / 3.0
                total = total + pi * pi * (1.0 if a == b else 2.0)
        rt = 1.0 / omega
        coeff = 0.1 * 0.1 * 9.0 * 2.0 * math.sqrt(2.0) / rho
        omega = 1.0 / (rt + 0.5 * (torch.sqrt(rt * rt + coeff * torch.sqrt(total)) - rt))
    out = []
    for i in range(19):
        f = omega * equilibrium(i, rho, u) + (1.0 - omega) * R[i]
        if alpha is not None:
            cu = sum(c * v for c, v in zip(VEL[i], u))
            force = sum(-alpha * u[a] * (3.0 * (VEL[i][a] - u[a]) + 9.0 * cu * VEL[i][a])
                        for a in range(3))
            f = f + (1.0 - 0.5 * omega) * WEIGHT[i] * force
        out.append(f)
    return out


def collide(R, flags, model, omega, ulid, walls=True, alpha=None):
    """P of the cells with these R: fluid cells relax, walls reflect, void cells keep R."""
    bulk = flags == 2 if walls else flags != 1
    new = relax(R, model, omega, alpha)
    out = []
    for i in range(19):
        f = torch.where(bulk, new[i], R[i])
        if walls and i:
            f = torch.where(flags == 4, R[OPP[i]], f)
            f = torch.where(flags == 8, R[OPP[i]] + 6.0 * WEIGHT[i] * ulid * VEL[i][0], f)
        out.append(f)
    return out


def halfway(P, flags, nx, ny, ulid):
    """The boundary managers on the stored state: links into void cells come back."""
    out = list(P)
    for flag, u in ((4, 0.0), (8, ulid)):
        for k in range(1, 19):
            j, s = OPP[k], shift_of(k, nx, ny)
            link = (flags == flag) & (torch.roll(flags, -s) == 1)
            back = P[k] + 6.0 * WEIGHT[j] * u * VEL[j][0]
            out[j] = torch.where(torch.roll(link, s), torch.roll(back, s), out[j])
    return out


def exchange(R, blocks, ni):
    """Overlap cells take what crosses into their block from the cell's owner."""
    n = ni + 2
    inner = (slice(1, -1),) * 3

    def part(b, lo=0):
        return tuple(slice(o + lo, o + m - lo) for o, m in zip(b[5:2:-1], b[2::-1]))
    own = torch.zeros(n, n, n, dtype=torch.bool, device=DEV)
    own[1:-1, 1:-1, 1:-1] = True
    for i in range(1, 19):
        whole = torch.zeros(n, n, n, dtype=torch.float64, device=DEV)
        for b, r in zip(blocks, R):
            whole[part(b, 1)] = r[i].view(b[2], b[1], b[0])[inner]
        for b, r in zip(blocks, R):
            cross = torch.zeros(b[2], b[1], b[0], dtype=torch.bool, device=DEV)
            for a, c in enumerate(VEL[i]):  # axis 2 - a of the tensor
                side = [slice(None)] * 3
                side[2 - a] = 0 if c > 0 else -1
                if c:
                    cross[tuple(side)] = True
            cross &= own[part(b)]
            r[i] = torch.where(cross, whole[part(b)], r[i].view(b[2], b[1], b[0])).reshape(-1)


def exact_adjoint(case, seed, P, flags, b, omega, ulid):
    alpha = torch.from_numpy(alpha_of(case, seed)).to(DEV).to(torch.float64)
    tau = torch.tensor(1.0 / omega, dtype=torch.float64, device=DEV)
    lid = torch.tensor(ulid, dtype=torch.float64, device=DEV)
    fluid = flags == 2

    def step(R, al, t, u):
        C = collide(list(R), flags, "bgk", 1.0 / t, u, alpha=al)
        return torch.stack(stream(C, b[0], b[1]))

    def score(R, al):
        _, u = moments(list(R), al)
        return ((u[0] ** 2 + u[1] ** 2 + u[2] ** 2) * fluid).sum()
    R = torch.stack(stream(P, b[0], b[1]))
    kept = []
    with torch.no_grad():
        for _ in range(case["steps"]):
            kept.append(R)
            R = step(R, alpha, tau, lid)
    last, al = R.clone().requires_grad_(), alpha.clone().requires_grad_()
    objective = score(last, al)
    lam, g = torch.autograd.grad(objective, (last, al))
    gt, gu = 0.0, 0.0
    for R0 in reversed(kept):
        v = [t.clone().requires_grad_() for t in (R0, alpha, tau, lid)]
        lam, ga, t1, u1 = torch.autograd.grad(step(*v), v, lam)
        g, gt, gu = g + ga, gt + float(t1), gu + float(u1)
    P = [torch.roll(R[i], -shift_of(i, b[0], b[1])) for i in range(19)]
    return P, {"objective": float(objective), "alpha": g, "tau": gt, "ulid": gu}


def exact(case, seed):
    cells, steps, storage = cells_of(case), case["steps"], case["storage"]
    if case["kind"] == "adjoint" and cells * steps > 1e8 or cells * steps > 3e9:
        return None
    if steps * (case.get("count", 1) + 30 * (case["kind"] == "blocks")) > 3000:
        return None
    arith = np.float64 if storage == "fp64" else np.float32
    ulid = float(arith(lid_velocity(seed)))
    blocks, model, more = blocks_of(case), case.get("model", "bgk"), {}
    flags = [torch.from_numpy(f).to(DEV).reshape(-1) for f in block_flags(case, blocks)]
    P, omega = [], [float(arith(1.0 / b[6])) for b in blocks]
    for b in blocks:
        rho, u = flow(b, seed)
        P.append([as_f64(stored(equilibrium(i, rho, u), i, storage), i, storage).reshape(-1)
                  for i in range(19)])
    del rho, u
    if case["kind"] == "adjoint":
        P[0], more = exact_adjoint(case, seed, P[0], flags[0], blocks[0], omega[0], ulid)
        steps = 0
    for _ in range(steps):
        for k, b in enumerate(blocks):
            R = stream(P[k], b[0], b[1])
            P[k] = None
            P[k] = collide(R, flags[k], model, omega[k], ulid, walls=case["kind"] != "halfway")
            del R
            if case["kind"] == "halfway":
                P[k] = halfway(P[k], flags[k], b[0], b[1], ulid)
        if case["kind"] == "blocks":
            R = [stream(p, b[0], b[1]) for p, b in zip(P, blocks)]
            exchange(R, blocks, case["ni"])
            P = [[torch.roll(r[i], -shift_of(i, b[0], b[1])) for i in range(19)]
                 for r, b in zip(R, blocks)]
    if case["kind"] == "monitor":
        b, fluid = blocks[0], flags[0] == 2
        rho, u = moments(stream(P[0], b[0], b[1]))
        lid = torch.where(flags[0] == 8, ulid, 0.0).to(torch.float64)
        zero = torch.zeros_like(lid)
        vel = torch.stack([torch.where(fluid, v, w) for v, w in zip(u, (lid, zero, zero))])
        sums = [rho[fluid].sum()] + [(rho * v)[fluid].sum() for v in u]
        more = {"fields": [torch.where(fluid, rho, 1.0).view(b[2], b[1], b[0]),
                           vel.view(3, b[2], b[1], b[0])],
                "sums": torch.stack(sums).cpu().numpy(),
                "change": float(max(v[fluid].abs().max() for v in u))}
    pops = []
    for b, p in zip(blocks, P):
        for i in range(19):
            if storage == "fp16s":
                p[i] = (p[i] - WEIGHT[i]) * 1024.0
            elif storage == "fp32s":
                p[i] = p[i] - WEIGHT[i]
        pops.append(torch.stack(p).view(19, b[2], b[1], b[0]))
    return dict(more, pops=pops)
