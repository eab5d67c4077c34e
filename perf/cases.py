"""The work that users of the engine have it do, as timed cases.

One pass is what a program does between two looks at its lattice: advance it by some time steps and
read the fields (or the conservation sums, or the steady-state residual).  The lattice lives on from
pass to pass, as it does in a run.  Sizes are those of the reference's drivers and published runs and of
the benchmark's configurations, with odd and ragged ones beside them.

  listed()            the cases that are timed by name
  draw(rng)           another case of the same ranges
  prepare(case, seed) lattices on the GPU, started from smooth (Shan-Chen: noisy) seeded fields
  run(state)          one pass; returns the fields read and the populations in their own buffer
  work(case)          bytes and operations that a pass cannot do without
  exact(case, seed)   the same pass in 64 bits, in plain torch
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lbm-arrayfire_b200"))
import lbm_b200 as lb  # noqa: E402

STORAGE = {"f32": lb.F32, "f16s": lb.F16S, "bf16s": lb.BF16S, "f64": lb.F64}
TORCH_TYPE = {"f32": torch.float32, "f16s": torch.float16, "bf16s": torch.bfloat16, "f64": torch.float64}
SCALE = {"f32": 1.0, "f16s": 16384.0, "bf16s": 1.0, "f64": 1.0}


# ---- the cases -------------------------------------------------------------------------------
def listed():
    return [
        # a viewer on the smallest cavity: fields every 10 iterations, as the reference's window draws them
        {"name": "lid128_f32_frame", "kind": "lid2d", "nx": 128, "ny": 128, "storage": "f32", "steps": 10, "read": "fields"},
        # the same cavity run to its steady state, the residual watched every 1000 steps
        {"name": "lid128_f16s_steady", "kind": "lid2d", "nx": 128, "ny": 128, "storage": "f16s", "steps": 1000, "read": "residual"},
        # the Karman street at the benchmark's size, reported every 100 steps
        {"name": "channel1024_f32", "kind": "channel2d", "nx": 1024, "ny": 256, "storage": "f32", "steps": 100, "read": "fields"},
        # the reference's published channel size (rows that are no multiple of 16), its own boundaries
        {"name": "channel1000_f16s", "kind": "channel2d_ref", "nx": 1000, "ny": 300, "storage": "f16s", "steps": 100, "read": "fields"},
        # the reference's largest published cavity
        {"name": "lid4096_f32", "kind": "lid2d", "nx": 4096, "ny": 4096, "storage": "f32", "steps": 50, "read": "fields"},
        # a double-precision reference run on an odd channel
        {"name": "channel1501_f64", "kind": "channel2d", "nx": 1501, "ny": 451, "storage": "f64", "steps": 50, "read": "fields"},
        # phase separation at the benchmark's size, the mass watched
        {"name": "shanchen1024_bf16s", "kind": "shanchen", "nx": 1024, "ny": 1024, "storage": "bf16s", "steps": 50, "read": "sums"},
        # a larger, ragged one in full precision
        {"name": "shanchen2049_f32", "kind": "shanchen", "nx": 2049, "ny": 1537, "storage": "f32", "steps": 50, "read": "fields"},
        # the benchmark's headline: MRT cavity, 16-bit storage
        {"name": "mrt256_f16s", "kind": "lid3d_mrt", "nx": 256, "ny": 256, "nz": 256, "storage": "f16s", "steps": 20, "read": "fields"},
        # and in plain single precision
        {"name": "mrt256_f32", "kind": "lid3d_mrt", "nx": 256, "ny": 256, "nz": 256, "storage": "f32", "steps": 20, "read": "fields"},
        # flow past a sphere in an odd duct
        {"name": "duct251_f16s", "kind": "duct3d", "nx": 251, "ny": 83, "nz": 83, "storage": "f16s", "steps": 50, "read": "fields"},
        # an ensemble of cavities and ducts of uneven sizes and Reynolds numbers
        {"name": "ensemble_f16s", "kind": "ensemble", "members2": 12, "members3": 4, "storage": "f16s", "steps": 50, "read": "fields"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A length of the range: as it falls, or rounded to a multiple of 16 or 64, as users choose them."""
    n = _log(rng, lo, hi)
    m = rng.choice([1, 1, 16, 64])
    return max(lo, n // m * m)


def draw(rng):
    kind = rng.choice(["lid2d", "lid2d", "channel2d", "channel2d_ref", "shanchen", "shanchen", "lid3d_mrt", "lid3d_mrt_ref", "lid3d", "duct3d", "ensemble"])
    c = {"kind": kind, "storage": rng.choice(["f32", "f32", "f16s", "f16s", "bf16s", "f64"]), "read": rng.choice(["fields", "fields", "sums", "residual"])}
    if kind == "ensemble":
        c.update(members2=rng.randint(4, 12), members3=rng.randint(1, 4), read="fields", storage=rng.choice(["f32", "f16s", "bf16s"]))
    elif "3d" in kind:
        n = _side(rng, 48, 200)
        c.update(nx=n, ny=n, nz=n)
        if kind == "duct3d":
            c.update(nx=min(3 * n, 400), ny=_side(rng, 40, 120), nz=_side(rng, 40, 120))
    else:
        c.update(nx=_side(rng, 100, 3000), ny=_side(rng, 64, 2000))
    if kind == "lid2d" and c["storage"] in ("f32", "f64"):
        c["absolute"] = rng.random() < 0.25
    cells = c.get("nx", 500) * c.get("ny", 1000) * c.get("nz", 1)
    most = 2.0e8 if "nz" in c else 4.0e8
    c["steps"] = max(2, min(_log(rng, 4, 500), int(most / cells)))
    return c


# ---- lattice facts, written out here so that exact() needs nothing of the engine -----------------
def velocities(dim):
    """D2Q9 and D3Q27 in the reference's order (cpp/d2q9_bgk_lid.cpp:72-79, cpp/d3q27_bgk_lid.cpp:98-107)."""
    if dim == 2:
        c = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
    else:
        c = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0),
             (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1), (1, 1, 1), (-1, 1, 1),
             (1, -1, 1), (-1, -1, 1), (1, 1, -1), (-1, 1, -1), (1, -1, -1), (-1, -1, -1)]
    w = [{2: [4 / 9, 1 / 9, 1 / 36], 3: [8 / 27, 2 / 27, 1 / 54, 1 / 216]}[dim][sum(map(abs, v))] for v in c]
    return c, w, [c.index(tuple(-a for a in v)) for v in c]


def shape_of(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if "nz" in case else ())


def omega_of(case):
    """Relaxation from the Reynolds number by the drivers' rule tau = 3 nu + 1/2."""
    kind = case["kind"]
    nu = {"lid2d": 0.1 * case["nx"] / max(100.0, case["nx"]), "channel2d": 0.04 * max(20, case["ny"] // 6) / 100.0,
          "channel2d_ref": 0.04 * max(20, case["ny"] // 6) / 100.0, "lid3d": max(0.02, 0.05 * case["nx"] / 400.0),
          "duct3d": max(0.02, 0.04 * case["ny"] / 4.0 / 40.0), "shanchen": 1.0 / 6.0}.get(kind, 0.05 * case["nx"] / 1000.0)
    return 1.0 / (3.0 * nu + 0.5)


def rates_of(case):
    """Relaxation rates by moment row: the benchmark's two values, or the reference's set (rust/examples/d3q27_mrt_lid.rs:111-150)."""
    if case["kind"] == "lid3d_mrt_ref":
        return [1.3, 1.3, 1.3, 1.3, 1.1, 1.1, 1.1, 0.9, 1.1, 1.1, 1.2, 1.2, 1.2, 1.2, 1.2, 1.2, 0.9, 1.2, 1.2, 1.2, 1.2, 1.2, 1.2, 1.1, 1.1, 1.1, 1.1]
    sv = 1.0 / (3.0 * 0.05 * 256 / 1000.0 + 0.5)
    return [sv if r in (4, 5, 6, 8, 9) else 1.2 for r in range(27)]


def members_of(case):
    """The ensemble's members: lids of 64 to 768 a side, ducts (4 L, L, L) with L of 32 to 64."""
    rng = np.random.default_rng(1000 * case["members2"] + case["members3"])
    out = []
    for _ in range(case["members2"]):
        n = int(rng.integers(1, 13)) * 64
        out.append({"kind": "lid2d", "nx": n, "ny": n, "storage": case["storage"]})
    for _ in range(case["members3"]):
        n = int(rng.choice([32, 48, 64]))
        out.append({"kind": "duct3d", "nx": 4 * n, "ny": n, "nz": n, "storage": case["storage"]})
    return out


def sphere_of(case):
    """Centre and radius of the obstacle (circle or sphere)."""
    if "nz" in case:
        return case["nx"] / 4.0, case["ny"] / 2.0, case["nz"] / 2.0, min(case["ny"], case["nz"]) / 8.0
    return case["nx"] // 5 + 1, case["ny"] // 2, 0.0, case["ny"] // 12 + 1


# ---- inputs ------------------------------------------------------------------------------------
def start_fields(case, seed, dev):
    """rho and u in 64 bits: low modes of 3 % (walls have their own classes); Shan-Chen: rho = 0.693 with noise, at rest."""
    rng = np.random.default_rng(seed)
    shape = shape_of(case)
    if case["kind"] == "shanchen":
        rho = torch.from_numpy(0.693 + rng.uniform(-0.01, 0.01, shape[::-1])).to(dev)
        return rho, [torch.zeros_like(rho) for _ in shape]
    axes = [torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n) for n in shape]

    def modes(amp):
        total = 0.0
        for _ in range(3):
            term = torch.full((1,) * len(shape), amp * float(rng.uniform(0.3, 1.0)) / 3, device=dev, dtype=torch.float64)
            for a, ax in enumerate(axes):
                at = [1] * len(shape)
                at[len(shape) - 1 - a] = -1
                term = term * torch.sin(int(rng.integers(1, 4)) * ax + float(rng.uniform(0, 6.28))).reshape(at)
            total = total + term
        return total

    return 1.0 + modes(0.01), [modes(0.03) for _ in shape]


def equilibrium(dim, i, rho, u):
    c, w, _ = velocities(dim)
    eu = sum(float(c[i][a]) * u[a] for a in range(dim) if c[i][a]) if any(c[i]) else torch.zeros_like(rho)
    usq = sum(a * a for a in u)
    return w[i] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * usq)


def start_populations(case, seed, dev):
    """F = feq(rho, u) as the caller hands it over: 64 bits for double-precision lattices, else 32."""
    rho, u = start_fields(case, seed, dev)
    dim = len(u)
    q = 9 if dim == 2 else 27
    F = torch.empty((q,) + tuple(rho.shape), device=dev, dtype=torch.float64 if case["storage"] == "f64" else torch.float32)
    for i in range(q):
        F[i] = equilibrium(dim, i, rho, u)
    return F


def lattice_of(case):
    """The descriptor and mask of a case, by the engine's own set-up calls."""
    kind, storage = case["kind"], STORAGE[case["storage"]]
    arithmetic = lb.ARITH_ABSOLUTE if case.get("absolute") else lb.ARITH_DEVIATION
    shape = shape_of(case)
    if kind == "shanchen":
        return lb.make_desc(lb.D2Q9, lb.SHANCHEN, storage, shape, omega=1.0, sc_G=-5.5), None
    if kind.startswith("lid3d_mrt"):
        basis = lb.MRT_REF if kind.endswith("ref") else lb.MRT_GRAM_SCHMIDT
        d = lb.make_desc(lb.D3Q27, lb.MRT, storage, shape, mrt_s=rates_of(case), mrt_basis=basis)
        return d, lb.setup_cavity3d(d, 0.05)
    d = lb.make_desc(lb.D2Q9 if len(shape) == 2 else lb.D3Q27, lb.BGK, storage, shape, omega=omega_of(case), arithmetic=arithmetic)
    if kind == "lid2d":
        return d, lb.setup_cavity2d(d, 0.1)
    if kind == "lid3d":
        return d, lb.setup_cavity3d(d, 0.05)
    ox, oy, oz, r = sphere_of(case)
    if kind == "duct3d":
        return d, lb.setup_duct3d(d, 0.04, ox, oy, oz, r)
    return d, lb.setup_channel2d(d, 0.04, ox, oy, r, 0 if kind.endswith("ref") else 1)


class _Buffer:
    """Device memory of a lattice as a tensor's source; the tensor keeps it, and it the lattice."""

    def __init__(self, ptr, nbytes, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def populations_view(lattice, storage, views):
    """The lattice's current population buffer as a tensor (no copy)."""
    ptr, nbytes = lattice.device_populations()
    if ptr not in views:
        views[ptr] = torch.as_tensor(_Buffer(ptr, nbytes, lattice), device="cuda").view(TORCH_TYPE[storage])
    return views[ptr]


def field_buffers(desc, storage):
    t = torch.float64 if storage == "f64" else torch.float32
    return torch.empty(desc.cells, device="cuda", dtype=t), torch.empty(desc.dim * desc.cells, device="cuda", dtype=t)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        parts = members_of(case)
        descs, masks = zip(*(lattice_of(m) for m in parts))
        batch = lb.Batch(list(descs), list(masks))
        for k, m in enumerate(parts):
            batch.set_populations(k, start_populations(m, seed + 100 * k, "cuda").reshape(-1).cpu().numpy())
        return {"case": case, "batch": batch, "fields": [field_buffers(d, case["storage"]) for d in descs]}
    d, mask = lattice_of(case)
    lattice = lb.Lattice(d, mask)
    F = start_populations(case, seed, "cuda").reshape(-1)
    torch.cuda.synchronize()
    lattice.set_populations(F)
    return {"case": case, "lattice": lattice, "fields": field_buffers(d, case["storage"]), "views": {}}


def run(state):
    case = state["case"]
    if "batch" in state:
        batch = state["batch"]
        batch.step(case["steps"])
        for k, (rho, u) in enumerate(state["fields"]):
            code = lb.lib().lbm_batch_get_macros(batch._h, k, ctypes.c_void_p(rho.data_ptr()), ctypes.c_void_p(u.data_ptr()), lb.DTYPE_F32, lb.DEVICE)
            if code:
                raise RuntimeError(lb.lib().lbm_last_error().decode())
        return {"fields": state["fields"]}
    lattice = state["lattice"]
    lattice.step(case["steps"])
    out = {}
    if case["read"] == "sums":
        out["sums"] = lattice.sums()
    elif case["read"] == "residual":
        out["residual"] = lattice.residual()
    else:
        lattice.macros_into(*state["fields"])
        out["rho"], out["u"] = state["fields"]
    out["populations"] = populations_view(lattice, case["storage"], state["views"])
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """Bytes: the populations and the mask read once and the populations written once a pass, and the
    fields written.  Operations: one collision a cell and step, in its usual count of adds and multiplies."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c in members_of(case) if case["kind"] == "ensemble" else [case]:
        cells = math.prod(shape_of(c))
        dim = len(shape_of(c))
        q, s = (9 if dim == 2 else 27), {"f32": 4, "f64": 8}.get(c["storage"], 2)
        fields = (dim + 1) * (8 if c["storage"] == "f64" else 4) if case["read"] == "fields" else 0
        mask = 0 if c["kind"] == "shanchen" else 1
        total["bytes"] += cells * (2 * q * s + fields + mask)
        per = {"shanchen": 150, "lid3d_mrt": 330, "lid3d_mrt_ref": 330}.get(c["kind"], 90 if dim == 2 else 250)
        total["flops"] += float(cells) * case["steps"] * per
    return total


# ---- the same in 64 bits --------------------------------------------------------------------------
def cell_rules(case, dev):
    """Per cell what the drivers overwrite: solid, forced rho, forced u (values), equilibrium, zero-gradient (tensors of [.., y, x])."""
    shape = shape_of(case)
    x, y = (torch.arange(n, device=dev).reshape([-1 if k == a else 1 for k in range(len(shape))][::-1]) for a, n in enumerate(shape[:2]))
    full = shape[::-1]
    no = torch.zeros(full, dtype=torch.bool, device=dev)
    rules = {"solid": no, "rho": no, "rho_is": torch.ones(full, device=dev, dtype=torch.float64), "ux": no, "uyz": no, "ux_is": 0.0, "eq": no, "zero": no}
    kind, nx, ny = case["kind"], shape[0], shape[1]
    if kind == "shanchen":
        return rules
    z = torch.arange(shape[2], device=dev).reshape(-1, 1, 1) if len(shape) == 3 else None
    if kind.startswith("lid"):
        solid = no | (x == 0) | (x == nx - 1) | (y == 0)
        if z is not None:
            solid = solid | (y == ny - 1) | (z == 0)
        lid = (no | ((y == ny - 1) if z is None else (z == shape[2] - 1))) & ~solid
        rules.update(solid=solid, rho=solid, rho_is=torch.zeros_like(rules["rho_is"]), ux=solid | lid, uyz=solid | lid, ux_is=(0.1 if z is None else 0.05) * lid.double())
        return rules
    ox, oy, oz, r = sphere_of(case)
    far = (x - ox) ** 2 + (y - oy) ** 2 + ((z - oz) ** 2 if z is not None else 0)
    solid = no | (far <= r * r) | (y == 0) | (y == ny - 1)
    if z is not None:
        solid = solid | (z == 0) | (z == shape[2] - 1)
    inlet, outlet = (no | (x == 0)), (no | (x == nx - 1))
    rho_is = (~solid).double()
    if kind.endswith("ref"):  # u_x and rho forced at the inlet, rho at the outlet, walls' end cells included
        rho_is = torch.where(inlet | outlet, torch.ones_like(rho_is), rho_is)
        rules.update(solid=solid, rho=solid | inlet | outlet, rho_is=rho_is, ux=solid | inlet, uyz=solid, ux_is=0.04 * (inlet & ~solid).double())
    else:
        inlet, outlet = inlet & ~solid, outlet & ~solid
        rules.update(solid=solid, rho=solid | inlet, rho_is=rho_is, ux=solid | inlet, uyz=solid | inlet, ux_is=0.04 * inlet.double(), eq=inlet, zero=outlet)
    return rules


def moment_rows():
    """The reference's 27 moments, row by row (rust/examples/d3q27_mrt_lid.rs:167-193)."""
    c, _, _ = velocities(3)
    rows = []
    for x, y, z in c:
        rows.append([1, x, y, z, x * y, x * z, y * z, x * x + y * y + z * z, x * x - y * y, x * x - z * z, x * y * y, x * z * z, y * x * x,
                     z * x * x, y * z * z, z * y * y, x * y * z, x * x * y * y, x * x * z * z, y * y * z * z, x * x * y * z, x * y * y * z,
                     x * y * z * z, x * y * y * z * z, x * x * y * z * z, x * x * y * y * z, x * x * y * y * z * z])
    return np.array(rows, dtype=np.float64).T


def reference_moments(rho, u):
    """The reference's equilibrium moments (rust/examples/d3q27_mrt_lid.rs:357-383)."""
    x, y, z = u
    t = rho / 3.0
    n = rho / 9.0
    return [rho, rho * x, rho * y, rho * z, rho * x * y, rho * x * z, rho * y * z, rho + rho * (x * x + y * y + z * z), rho * (x * x - y * y),
            rho * (x * x - z * z), t * x, t * x, t * y, t * z, t * y, t * z, 0.0 * rho, t * (1 / 3 + x * x + y * y), t * (1 / 3 + x * x + z * z),
            t * (1 / 3 + y * y + z * z), t * y * z, t * x * z, t * x * y, n * x, n * y, n * z, x * x + y * y + z * z + rho / 27.0]


def exact_steps(case, seed, steps, dev):
    """(rho, u) of the last step and the populations before and after it, in 64 bits."""
    F = start_populations(case, seed, dev).double()
    dim = F.dim() - 1
    c, w, opp = velocities(dim)
    q = len(c)
    rules = cell_rules(case, dev)
    omega = omega_of(case)
    mrt = None
    if case["kind"].startswith("lid3d_mrt"):
        M = moment_rows()
        if case["kind"] == "lid3d_mrt":
            for k in range(27):
                for j in range(k):
                    M[k] -= (M[k] @ M[j]) / (M[j] @ M[j]) * M[j]
        mrt = torch.from_numpy(np.linalg.inv(M) @ np.diag(rates_of(case))).to(dev), torch.from_numpy(M).to(dev)
    last = F
    for _ in range(steps):
        last = F
        S = torch.empty_like(F)
        for i in range(q):
            S[i] = torch.roll(F[i], shifts=tuple(c[i][a] for a in range(dim))[::-1], dims=tuple(range(dim)))
            if c[i][0] == -1 and case["kind"] in ("channel2d", "duct3d"):
                S[i] = torch.where(rules["zero"], torch.roll(F[i], shifts=tuple((c[i][a] if a else 0) for a in range(dim))[::-1], dims=tuple(range(dim))), S[i])
        rho = S.sum(0)
        u = [sum(float(c[i][a]) * S[i] for i in range(q) if c[i][a]) / rho for a in range(dim)]
        rho = torch.where(rules["rho"], rules["rho_is"], rho)
        u[0] = torch.where(rules["ux"], torch.as_tensor(rules["ux_is"], device=dev, dtype=torch.float64), u[0])
        for a in range(1, dim):
            u[a] = torch.where(rules["uyz"], torch.zeros_like(u[a]), u[a])
        seen, shifted = u, u
        if case["kind"] == "shanchen":
            psi = 1.0 - torch.exp(-rho)
            pull = [sum(w[i] * c[i][a] * torch.roll(psi, shifts=(-c[i][1], -c[i][0]), dims=(0, 1)) for i in range(1, 9) if c[i][a]) for a in (0, 1)]
            force = [5.5 * psi * s for s in pull]
            shifted = [u[a] + force[a] / rho for a in (0, 1)]
            seen = [u[a] + force[a] / (2.0 * rho) for a in (0, 1)]
        F = torch.empty_like(S)
        if mrt is not None:
            flat = S.reshape(27, -1)
            m = mrt[1] @ flat
            if case["kind"].endswith("ref"):
                for k, v in enumerate(reference_moments(rho, u)):
                    m[k] -= v.reshape(-1)
            else:
                m -= mrt[1] @ torch.stack([equilibrium(3, i, rho, u).reshape(-1) for i in range(27)])
            F = (flat - mrt[0] @ m).reshape(S.shape)
            del m
        else:
            for i in range(q):
                e = equilibrium(dim, i, rho, shifted)
                F[i] = torch.where(rules["eq"], e, omega * e + (1.0 - omega) * S[i])
        if case["kind"] != "shanchen":
            for i in range(1, q):
                F[opp[i]] = torch.where(rules["solid"], S[i], F[opp[i]])
    return rho, seen, last, F


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "ensemble":
        fields = []
        for k, m in enumerate(members_of(case)):
            rho, u, _, _ = exact_steps(m, seed + 100 * k, case["steps"], dev)
            fields.append((rho.reshape(-1), torch.cat([a.reshape(-1) for a in u])))
        return {"fields": fields}
    rho, u, before, F = exact_steps(case, seed, case["steps"], dev)
    c, w, _ = velocities(F.dim() - 1)
    out = {}
    if case["read"] == "fields":
        out["rho"], out["u"] = rho.reshape(-1), torch.cat([a.reshape(-1) for a in u])
    elif case["read"] == "sums":
        sums = [F.sum()] + [sum(float(v[a]) * F[i].sum() for i, v in enumerate(c) if v[a]) if a < len(u) else F.new_zeros(()) for a in range(3)]
        out["sums"] = np.array([float(s) for s in sums])
    else:
        out["residual"] = None
    if case["storage"] in ("f16s", "bf16s"):
        F = (F - F.new_tensor(w).reshape((-1,) + (1,) * (F.dim() - 1))) * SCALE[case["storage"]]
    # (phase separation amplifies 16-bit rounding within tens of steps: only its mass is comparable)
    out["populations"] = None if case["kind"] == "shanchen" and case["storage"] in ("f16s", "bf16s") else F.reshape(-1)
    return out
