"""Timed cases of the space-charge framework: what a tracking program has it do.

Every case goes through the package's public entry points with beams of the kind they meet: a bunch of 0.2 mm and
about a millimetre behind an injector linac, chirped, at 100-500 MeV for the FP32 form; down to 6.5 MeV (the
entrance of the first cavity of the regression line) for the FP64 form.  Kinds:

  kick   one SpaceCharge.apply on a beam that lives on the GPU (the body of a device-resident tracking loop)
  host   one SpaceCharge.apply on numpy arrays (the plugin inside the reference's own track())
  field  one SpaceCharge.el_field on numpy arrays (the reference's public stage method)
  batch  one recorded kick of several uneven beams (BeamBatch.graph().replay())
  track  one whole track() of a FODO line: transport, kicks and the beam moments of every step

``exact`` restates the kick with torch in float64 (the formulas of ocelot/cpbd/sc.py and coord_transform.py).
"""
import math
import random

import numpy as np
import torch

from ocelot_gb300 import ParticleArray, SpaceCharge
from ocelot_gb300.batch import BeamBatch
from ocelot_gb300.beam import DeviceParticleArray
from ocelot_gb300.serve import fodo
from ocelot_gb300.track import track

M_E_EV = 9.10938215e-31 * 299792458.0 ** 2 / 1.6021766208e-19
EPS0 = 1.0 / (4e-7 * math.pi) / 299792458.0 ** 2

#: sigma of x', y', the uncorrelated energy spread and the linear chirp [1/m] of every beam
SIG_ANGLE, SIG_P, CHIRP = 2e-5, 2e-4, -1.0


def _case(name, kind, form, n, mesh, energy=0.130, charge=250e-12, sx=200e-6, st=1e-3, dz=0.1, **more):
    return dict(name=name, kind=kind, form=form, n=n, nx=mesh[0], ny=mesh[1], nz=mesh[2], energy=energy, charge=charge,
                sx=sx, st=st, dz=dz, **more)


def listed():
    return [
        # a first look at a lattice with few particles; an odd count, rows as from_host lays them out
        _case("kick32_10k_32", "kick", "fp32", 10007, (32, 32, 32), energy=0.25),
        # the regression line's beam (10k particles, default mesh) at its 6.5 MeV entrance
        _case("kick64_10k_63_low", "kick", "fp64", 10000, (63, 63, 63), energy=0.0065, dz=0.005),
        # the plain-form workload's size: 200k particles on the default mesh, both forms
        _case("kick32_200k_63", "kick", "fp32", 200000, (63, 63, 63)),
        _case("kick64_200k_63", "kick", "fp64", 200000, (63, 63, 63)),
        # the same through numpy arrays: what the plugin does inside the reference's track()
        _case("host64_200k_63", "host", "fp64", 200000, (63, 63, 63)),
        # the field at given points, odd count and uneven mesh
        _case("field64_100k_40x48x100", "field", "fp64", 100003, (40, 48, 100)),
        # the headline size: 2M particles, 64^3, both forms
        _case("kick32_2m_64", "kick", "fp32", 2000000, (64, 64, 64)),
        _case("kick64_2m_64", "kick", "fp64", 2000000, (64, 64, 64)),
        # the largest: 10M particles on a fine mesh along the bunch
        _case("kick32_10m_128x128x256", "kick", "fp32", 10000000, (128, 128, 256), energy=0.25, dz=0.05),
        # a parameter scan: uneven beams kicked together
        _case("batch32_16", "batch", "fp32", 400000, (64, 64, 64), beams=16),
        # whole tracking calls: FP32 with first-order maps; FP64 with second-order maps at low energy
        _case("track32_200k_63", "track", "fp32", 200000, (63, 63, 63), energy=0.25, dz=0.25, cells=4, order=1),
        _case("track64_10k_31_order2", "track", "fp64", 10000, (31, 31, 31), energy=0.05, dz=0.25, cells=2, order=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choice(("kick", "kick", "kick", "kick", "host", "field", "batch", "track"))
    form = "fp64" if kind == "field" else "fp32" if kind == "batch" else rng.choice(("fp32", "fp64"))
    big = {"kick": 6e6, "host": 1e6, "field": 1e6, "batch": 1e6, "track": 4e5}[kind] / (3 if form == "fp64" else 1)
    n = int(_log(rng, 5e3, big))
    if rng.random() < 0.5:
        n += n & 1
    if rng.random() < 0.5:
        m = rng.choice((16, 24, 31, 32, 47, 48, 63, 64, 95, 96))
        mesh = (m, m, m)
    else:
        t = rng.randint(16, 100)
        mesh = (t, t if rng.random() < 0.5 else rng.randint(16, 100), rng.randint(16, 200))
    if kind == "track":
        mesh = tuple(min(v, 64) for v in mesh)
    energy = _log(rng, 0.1, 0.5) if form == "fp32" else _log(rng, 0.0065, 0.5)
    charge, sx, st = rng.uniform(20e-12, 500e-12), _log(rng, 100e-6, 300e-6), _log(rng, 3e-4, 1e-3)
    if kind == "track":  # many kicks with metres of transport behind each: an accelerated, longer bunch
        energy = _log(rng, 0.2, 0.5) if form == "fp32" else _log(rng, 0.05, 0.5)
        charge, sx, st = rng.uniform(20e-12, 250e-12), _log(rng, 150e-6, 300e-6), _log(rng, 6e-4, 1e-3)
    # the step is shorter where space charge is stronger: the kick of one step [rad] stays a small part of the beam's
    # angles, also after the thousands of kicks without transport that timing takes
    gamma = energy * 1e9 / M_E_EV
    per_metre = 2 * charge * 299792458.0 / (2.5 * st) / (17045.0 * gamma ** 3 * sx)
    dz = min(rng.uniform(0.05, 0.25), (1e-6 if form == "fp32" else 2e-5) / per_metre)
    c = _case("", kind, form, n, mesh, energy=energy, charge=charge, sx=sx, st=st, dz=0.25 if kind == "track" else dz)
    if kind == "batch":
        c["beams"] = rng.randint(2, 16)
    if kind == "track":
        c["cells"], c["order"] = rng.randint(1, 3), rng.choice((1, 2))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _beam(n, seed, sx, st, charge):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rp = torch.randn((6, n), generator=g, dtype=torch.float64, device="cuda")
    for row, sig in enumerate((sx, SIG_ANGLE, sx, SIG_ANGLE, st, SIG_P)):
        rp[row] *= sig
    rp[5] += CHIRP * rp[4]
    return rp, torch.full((n,), charge / n, dtype=torch.float64, device="cuda")


def _members(case, seed):
    """(n, mesh, energy, rp, q) of each beam of a batch: sizes and meshes spread below the case's own."""
    rng = random.Random(seed * 1000003 + 17)
    small = ((32, 32, 32), (48, 48, 48), (32, 32, 128))
    for b in range(case["beams"]):
        # sizes and meshes depend on the place in the batch alone, so that every seed costs the same
        n = max(5000, int(case["n"] * (1.0, 0.3, 2.5, 0.1)[b % 4])) + (b % 3)
        mesh = (case["nx"], case["ny"], case["nz"]) if b % 2 == 0 else small[b // 2 % 3]
        rp, q = _beam(n, seed * 64 + b, case["sx"] * rng.uniform(0.7, 1.4), case["st"], case["charge"])
        yield n, mesh, case["energy"] * rng.uniform(1.0, 1.5), rp, q


def _process(case):
    return SpaceCharge(step=1, nmesh_xyz=[case["nx"], case["ny"], case["nz"]], precision=case["form"])


def _field_inputs(case, seed):
    """Rest-frame positions [N, 3] before the scaling of z, charges and gamma."""
    rp, q = _beam(case["n"], seed, case["sx"], case["st"], case["charge"])
    return rp[[0, 2, 4]].T.contiguous().cpu().numpy(), q.cpu().numpy(), case["energy"] * 1e9 / M_E_EV


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "dz": case["dz"], "case": case}
    if kind == "batch":
        s["batch"] = BeamBatch()
        s["rp"] = []
        for n, mesh, energy, rp, q in _members(case, seed):
            s["batch"].add(rp, q, energy, mesh, case["dz"])
            s["rp"].append(rp)
        s["batch"].commit()
        s["graph"] = s["batch"].graph()
        return s
    s["sc"] = _process(case)
    s["sc"].prepare(None)
    if kind == "field":
        s["X"], s["Q"], s["gamma"] = _field_inputs(case, seed)
        return s
    rp, q = _beam(case["n"], seed, case["sx"], case["st"], case["charge"])
    if kind == "kick":
        s["beam"] = DeviceParticleArray(rp, q, case["energy"])
        return s
    pa = ParticleArray(case["n"])
    pa.rparticles[...] = rp.cpu().numpy()
    pa.q_array = q.cpu().numpy()
    pa.E = case["energy"]
    s["beam"] = pa
    if kind == "track":
        s["line"] = fodo(case["cells"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "kick":
        s["sc"].apply(s["beam"], s["dz"])
        return s["beam"].rparticles
    if kind == "host":
        s["sc"].apply(s["beam"], s["dz"])
        return s["beam"].rparticles
    if kind == "field":
        X = s["X"].copy()  # el_field scales its z in place
        E = s["sc"].el_field(X, s["Q"], s["gamma"], s["sc"].nmesh_xyz)
        return [X, E]
    if kind == "batch":
        s["graph"].replay()
        return list(s["rp"])
    # track: the beam file's particles go into each tracking run
    src = s["beam"]
    pa = ParticleArray(src.size())
    pa.rparticles[...] = src.rparticles
    pa.q_array = src.q_array
    pa.E = src.E
    tws, pa = track(s["line"], pa, sc=s["sc"], unit_step=s["dz"], order=s["case"]["order"])
    return [pa.rparticles, np.array([[t.s, t.E, t.xx, t.pxpx, t.yy, t.pypy, t.tautau, t.pp] for t in tws])]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _kick_work(n, mesh, form, moved=104):
    """Bytes: the particles in and out, the charges, the charge grid out and the potential in (each once).  Operations:
    a few hundred per particle and the transforms of the padded grid (one real transform forward and one back over
    half the spectrum, 2.5 M log2 M each), and one cell integral per cell of the mesh."""
    w = 8 if form == "fp64" else 4
    cells = mesh[0] * mesh[1] * mesh[2]
    padded = 8 * cells
    return {"bytes": moved * n + 2 * w * cells, "flops": 200 * n + 2 * 2.5 * padded * math.log2(padded) + 100 * cells}


def _steps(case):
    total = 2.4 * case["cells"]
    return max(1, math.ceil(total / case["dz"] - 1e-9))


def work(case):
    mesh = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "batch":
        small = ((32, 32, 32), (48, 48, 48), (32, 32, 128))
        out = {"bytes": 0, "flops": 0}
        for b in range(case["beams"]):
            n = max(5000, int(case["n"] * (1.0, 0.3, 2.5, 0.1)[b % 4])) + (b % 3)
            w = _kick_work(n, mesh if b % 2 == 0 else small[b // 2 % 3], case["form"])
            out = {k: out[k] + w[k] for k in out}
        return out
    if case["kind"] == "field":
        return _kick_work(case["n"], mesh, case["form"], moved=64)
    w = _kick_work(case["n"], mesh, case["form"])
    if case["kind"] == "track":  # kick, transport (a read and a write of the rows) and moments (a read) per step
        k = _steps(case)
        return {"bytes": k * (w["bytes"] + 144 * case["n"]), "flops": k * (w["flops"] + 100 * case["n"])}
    return w


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _igf(mesh, h):
    x, y, z = (h[a] * torch.arange(mesh[a] + 1, dtype=torch.float64, device="cuda") - h[a] / 2 for a in range(3))
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
    r = torch.sqrt(x * x + y * y + z * z)
    ig = (-x * x * 0.5 * torch.atan(y * z / (x * r)) + y * z * torch.log(x + r)
          - y * y * 0.5 * torch.atan(z * x / (y * r)) + z * x * torch.log(y + r)
          - z * z * 0.5 * torch.atan(x * y / (z * r)) + x * y * torch.log(z + r))
    for a in range(3):
        ig = torch.diff(ig, dim=a)
    return ig


def _potential(q, h):
    mesh = q.shape
    g = _igf(mesh, h)
    for a in range(3):  # the mirrored lags behind the octant
        g = torch.cat((g, torch.flip(g.narrow(a, 1, mesh[a] - 1), (a,))), dim=a)
    s = tuple(2 * m - 1 for m in mesh)
    phi = torch.fft.irfftn(torch.fft.rfftn(q, s) * torch.fft.rfftn(g), s)
    return phi[:mesh[0], :mesh[1], :mesh[2]] / (4 * math.pi * EPS0 * h[0] * h[1] * h[2])


def _sample(F, c):
    """Trilinear samples at [N, 3] grid coordinates, 0 outside the grid."""
    top = torch.tensor([m - 1 for m in F.shape], dtype=torch.float64, device="cuda")
    ok = ((c >= 0) & (c <= top)).all(1)
    i = torch.minimum(torch.floor(c.clamp_min(0)), top - 1).long()
    t = c - i
    flat, (_, ny, nz) = F.reshape(-1), F.shape
    out = torch.zeros(c.shape[0], dtype=torch.float64, device="cuda")
    for a in (0, 1):
        for b in (0, 1):
            for d in (0, 1):
                w = (t[:, 0] if a else 1 - t[:, 0]) * (t[:, 1] if b else 1 - t[:, 1]) * (t[:, 2] if d else 1 - t[:, 2])
                at = ((i[:, 0] + a) * ny + i[:, 1] + b) * nz + i[:, 2] + d
                out += torch.where(ok, flat[at.clamp(0, flat.numel() - 1)] * w, torch.zeros_like(w))
    return out


def _field(X, q, gamma, mesh):
    """Field at the positions X [N, 3] (z already scaled by gamma)."""
    nm = torch.tensor(mesh, dtype=torch.float64, device="cuda")
    lo, hi = X.min(0).values, X.max(0).values
    h = (hi - lo) / (nm - 3)
    mid = (q @ (X / h)) / q.sum()
    off = torch.floor(lo / h - mid) + mid
    G = X / h - off
    cell = (torch.floor(G) + 1).long()
    key = (cell[:, 0] * mesh[1] + cell[:, 1]) * mesh[2] + cell[:, 2]
    grid = torch.zeros(mesh[0] * mesh[1] * mesh[2], dtype=torch.float64, device="cuda").index_add_(0, key, q)
    hs = [float(v) for v in h]
    phi = _potential(grid.reshape(mesh), hs)
    E = torch.zeros((X.shape[0], 3), dtype=torch.float64, device="cuda")
    for a in range(3):
        F = torch.zeros_like(phi)
        F.narrow(a, 0, mesh[a] - 1).copy_(-torch.diff(phi, dim=a) / hs[a])
        shift = torch.full((3,), 0.5, dtype=torch.float64, device="cuda")
        shift[a] = 0.0
        E[:, a] = _sample(F, G + shift) * (gamma if a < 2 else 1.0)
    return E


def _kick(rp, q, energy, dz, mesh):
    """The kick on rp [6, N], as new particles."""
    gr = energy * 1e9 / M_E_EV
    br = math.sqrt(1 - gr ** -2)
    pr = M_E_EV * math.sqrt(gr * gr - 1)
    x, xq, y, yq, tau, d = rp
    gamma = (br * d + 1) * gr
    beta = torch.sqrt(1 - gamma ** -2)
    pz = torch.sqrt((gamma * beta / (gr * br)) ** 2 - xq * xq - yq * yq)
    u = torch.stack((xq / pz, yq / pz, torch.ones_like(pz)))
    u = u / torch.linalg.norm(u, dim=0)
    lab = torch.stack((x - u[0] * beta * tau, y - u[1] * beta * tau, -u[2] * beta * tau))
    p = u * gamma * beta * M_E_EV
    t3 = p.mean(1)
    pav = torch.linalg.norm(t3)
    t3 = t3 / pav
    t1 = torch.linalg.cross(torch.tensor([0., 1., 0.], dtype=torch.float64, device="cuda"), t3)
    t1 = t1 / torch.linalg.norm(t1)
    T = torch.stack((t1, torch.linalg.cross(t3, t1), t3), dim=1)
    g0 = float(torch.sqrt((pav / M_E_EV) ** 2 + 1))
    X = lab.T @ T
    X[:, 2] *= g0
    E = _field(X, q, g0, mesh)
    cdt = dz / br
    P = p.T @ T
    P[:, :2] += cdt * g0 ** -2 * E[:, :2]
    P[:, 2] += cdt * E[:, 2]
    p = (P @ T.T).T
    s = (p * p).sum(0)
    gamma = torch.sqrt(1 + s / M_E_EV ** 2)
    beta = torch.sqrt(1 - gamma ** -2)
    u = p / torch.sqrt(s)
    c = -lab[2] / (beta * u[2])
    return torch.stack((lab[0] + beta * u[0] * c, p[0] / pr, lab[1] + beta * u[1] * c, p[1] / pr, c,
                        (gamma / gr - 1) / br))


def _section(k1, length, energy):
    """First-order matrix of a drift or quadrupole."""
    R = np.eye(6)
    for i, k in ((0, k1), (2, -k1)):
        w = math.sqrt(abs(k))
        c, s = (1.0, length) if k == 0 else (math.cos(w * length), math.sin(w * length) / w) if k > 0 else (
            math.cosh(w * length), math.sinh(w * length) / w)
        R[i:i + 2, i:i + 2] = [[c, s], [-k * s, c]]
    g = energy * 1e9 / M_E_EV
    R[4, 5] = -length / (g * g - 1)
    return R


def _exact_track(case, seed):
    rp, q = _beam(case["n"], seed, case["sx"], case["st"], case["charge"])
    mesh, energy = (case["nx"], case["ny"], case["nz"]), case["energy"]
    edges, z = [], 0.0
    for _ in range(case["cells"]):
        for length, k1 in ((0.2, 1.2), (1.0, 0.0), (0.2, -1.2), (1.0, 0.0)):
            edges.append((z, z + length, k1))
            z += length
    total, at = z, 0.0
    while total - at > 1e-10:
        to = min(at + case["dz"], total)
        R = np.eye(6)
        for a, b, k1 in edges:
            if min(b, to) - max(a, at) > 1e-10:
                R = _section(k1, min(b, to) - max(a, at), energy) @ R
        rp = torch.from_numpy(R).cuda() @ rp
        rp = _kick(rp, q, energy, to - at, mesh)
        at = to
    return [rp, None]


def exact(case, seed):
    mesh = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "batch":
        return [_kick(rp, q, energy, case["dz"], m) for n, m, energy, rp, q in _members(case, seed)]
    if case["kind"] == "field":
        X, Q, gamma = _field_inputs(case, seed)
        X[:, 2] *= gamma
        return [X, _field(torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda(), gamma, mesh)]
    if case["kind"] == "track":
        return _exact_track(case, seed) if case["order"] == 1 else None
    rp, q = _beam(case["n"], seed, case["sx"], case["st"], case["charge"])
    out = _kick(rp, q, case["energy"], case["dz"], mesh)
    return out if case["kind"] == "kick" else out.cpu().numpy()
