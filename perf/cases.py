"""Measured cases of the lattice Yang-Mills hot path, through the Python mirror of the C ABI.

A pass is a segment of a user's run: a number of steps (leapfrog, Langevin, gradient flow, Gauss
restore) of a lattice or of an ensemble, the measurement that such a run takes with them, and the
state, read back into page-locked host arrays with ``download``.  FP32 storage holds 32-bit values,
so the state of an FP32 lattice is returned as float32, that of an FP64 lattice as float64.

A case is a dict of plain values:
  what     "leapfrog" | "langevin" | "flow" | "restore" | "ensemble"
  nc       2 or 3; bits 32 or 64 (storage); nx, ny, nz the extents
  steps    steps (sweeps, iterations) of a pass; every: steps between two measurements
  members  trajectories of an ensemble (half SU(2), half SU(3), L = 16, 24, 32, 48 in turn)
  sweep    "checkerboard" or "simultaneous" (flow)
"""
import math

import numpy as np
import torch

import topologicalcymsolver_gb300 as tcym

NM = {2: 4, 3: 18}  # doubles per link in the host layout
NA = {2: 3, 3: 8}   # algebra components
DT = 0.05           # leapfrog
DT_LANGEVIN, GAMMA, TEMPERATURE = 0.02, 1.0, 0.6
DTAU = 0.02         # flow
LINK_WIDTH = 0.3    # start: U = exp(i theta^a t^a), theta ~ N(0, 0.3^2)
FIELD_VARIANCE = 0.3  # E ~ N(0, 0.3), the lower end of the trajectories' temperatures
ENSEMBLE_L = (16, 24, 32, 48)

_context = None


def _ctx():
    """The one library context of the process, as a program keeps it."""
    global _context
    if _context is None:
        _context = tcym.Context(0)
    return _context


def _case(name, what, nc, bits, shape, steps, every=0, sweep="", members=0):
    return {"name": name, "what": what, "nc": nc, "bits": bits, "nx": shape[0], "ny": shape[1], "nz": shape[2],
            "steps": steps, "every": every, "sweep": sweep, "members": members}


def listed():
    return [
        # the plain drop-in at the reference's own size, all observables every 10 steps
        _case("su2_16_fp64_series", "leapfrog", 2, 64, (16, 16, 16), 20, 10),
        # one small trajectory stepped alone: launches and latency
        _case("su3_24_leapfrog", "leapfrog", 3, 32, (24, 24, 24), 80, 20),
        # a served Langevin request: N_CS every 20 steps
        _case("su2_32_langevin", "langevin", 2, 32, (32, 32, 32), 80, 20),
        # the Langevin production run: N_CS integrated along the trajectory
        _case("su3_64_langevin", "langevin", 3, 32, (64, 64, 64), 80, 10),
        # cooling of a 96^3 configuration: observables every 10 checkerboard sweeps
        _case("su2_96_cooling", "flow", 2, 32, (96, 96, 96), 60, 10, "checkerboard"),
        # smoothing before a topology measurement: the reference's simultaneous flow
        _case("su3_64_flow", "flow", 3, 32, (64, 64, 64), 120, 20, "simultaneous"),
        # a large SU(3) trajectory
        _case("su3_96_leapfrog", "leapfrog", 3, 32, (96, 96, 96), 80, 20),
        # SU(2) at the largest served size
        _case("su2_128_leapfrog", "leapfrog", 2, 32, (128, 128, 128), 80, 20),
        # the plain FP64 path of SU(3)
        _case("su3_48_fp64", "leapfrog", 3, 64, (48, 48, 48), 20, 10),
        # ragged extents, odd nz
        _case("su3_33x20x27_odd", "leapfrog", 3, 32, (33, 20, 27), 80, 20),
        # many trajectories of mixed groups and sizes advanced together, N_CS every 20 steps
        _case("ensemble_32", "ensemble", 0, 32, (0, 0, 0), 80, 20, "", 32),
        # preparation of a request: Gauss's law restored on a fresh field
        _case("su3_64_restore", "restore", 3, 32, (64, 64, 64), 60),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["leapfrog", "leapfrog", "langevin", "flow", "flow_cb", "restore", "ensemble", "fp64"])
    if kind == "ensemble":
        c = _case("", "ensemble", 0, 32, (0, 0, 0), rng.randrange(40, 81), rng.choice([10, 20]), "",
                  rng.randrange(4, 33))
        del c["name"]
        return c
    nc = rng.choice([2, 3])
    top = 56 if kind == "fp64" else (96 if nc == 3 else 120)
    n = [int(round(math.exp(rng.uniform(math.log(14), math.log(top))))) for _ in range(3)]
    if rng.random() < 0.5:  # most lattices in use are cubes
        n = [n[0]] * 3
    if kind == "flow_cb":
        n = [x + x % 2 for x in n]
    steps = rng.randrange(10, 21) if kind == "fp64" else rng.randrange(40, 81)
    every = rng.choice([10, 20])
    what, bits, sweep = kind, 32, ""
    if kind == "fp64":
        what, bits = rng.choice(["leapfrog", "langevin"]), 64
    elif kind == "flow":
        sweep = "simultaneous"
    elif kind == "flow_cb":
        what, sweep = "flow", "checkerboard"
    elif kind == "restore":
        bits, every = rng.choice([32, 32, 64]), 0
        if bits == 64:
            n = [min(x, 48) for x in n]
    c = _case("", what, nc, bits, n, steps, every, sweep)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _generators(nc, dev):
    """t^a, Hermitian, tr(t^a t^b) = delta^ab / 2, in the library's order."""
    t = torch.zeros(NA[nc], nc, nc, dtype=torch.complex128)
    k = 0
    for j in range(1, nc):
        for i in range(j):
            t[k, i, j] = t[k, j, i] = 0.5
            t[k + 1, i, j], t[k + 1, j, i] = -0.5j, 0.5j
            k += 2
            if i == 0 and j == 1:
                t[2, 0, 0], t[2, 1, 1] = 0.5, -0.5
                k = 3
    if nc == 3:
        s = 0.5 / math.sqrt(3.0)
        t[7, 0, 0], t[7, 1, 1], t[7, 2, 2] = s, s, -2 * s
    return t.to(dev)


def _device():
    return torch.device("cuda", 0)


def _to_host_layout(u, nc):
    """(..., nc, nc) complex links as the host layout's NM[nc] doubles."""
    if nc == 2:
        return torch.stack([u[..., 0, 1].imag, u[..., 0, 1].real, u[..., 0, 0].imag, u[..., 0, 0].real], -1)
    return torch.view_as_real(u.transpose(-1, -2).contiguous()).reshape(*u.shape[:-2], 18)


def _from_host_layout(a, nc):
    if nc == 2:
        q0, q1, q2, q3 = a.unbind(-1)
        row0 = torch.stack([torch.complex(q3, q2), torch.complex(q1, q0)], -1)
        row1 = torch.stack([torch.complex(-q1, q0), torch.complex(q3, -q2)], -1)
        return torch.stack([row0, row1], -2)
    return torch.view_as_complex(a.reshape(*a.shape[:-1], 9, 2)).reshape(*a.shape[:-1], 3, 3).transpose(-1, -2)


def _mul(a, b):
    """Matrix product of the last two dimensions."""
    n = a.shape[-1]
    out = a[..., :, 0:1] * b[..., 0:1, :]
    for k in range(1, n):
        out.addcmul_(a[..., :, k:k + 1], b[..., k:k + 1, :])
    return out


def _dag(a):
    return a.transpose(-1, -2).conj()


def _expi(theta, t):
    """exp(i theta^a t^a): Taylor series of the quarter argument, squared twice."""
    h = 0.25j * torch.tensordot(theta.to(torch.complex128), t, 1)
    one = torch.eye(t.shape[-1], dtype=torch.complex128, device=theta.device)
    out = one + h / 14
    for k in range(13, 0, -1):
        out = one + _mul(h, out) / k
    for _ in range(2):
        out = _mul(out, out)
    return out


def _start(nc, volume, seed, bits, zero_field=False):
    """Links and fields of `volume` sites in the host layouts, on the GPU, to the storage's precision."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    t = _generators(nc, dev)
    U = torch.empty(volume, 3, NM[nc], dtype=torch.float64, device=dev)
    for a in range(0, volume, 1 << 18):
        n = min(volume, a + (1 << 18)) - a
        theta = LINK_WIDTH * torch.randn(n, 3, NA[nc], dtype=torch.float64, device=dev, generator=g)
        U[a:a + n] = _to_host_layout(_expi(theta, t), nc)
    if zero_field:
        E = torch.zeros(volume, 3, NA[nc], dtype=torch.float64, device=dev)
    else:
        E = math.sqrt(FIELD_VARIANCE) * torch.randn(volume, 3, NA[nc], dtype=torch.float64, device=dev, generator=g)
    return (U, E) if bits == 64 else (U.float().double(), E.float().double())


def _inputs(case, nc, volume, seed):
    return _start(nc, volume, 7919 * int(seed) + nc, case["bits"], case["what"] == "langevin")


def _shapes(case):
    """(nc, extents) of every lattice of the case."""
    if case["what"] == "ensemble":
        return [(2 + i % 2, (ENSEMBLE_L[i // 2 % 4],) * 3) for i in range(case["members"])]
    return [(case["nc"], (case["nx"], case["ny"], case["nz"]))]


class _HostState:
    """Page-locked host arrays of one or more lattices of one group, one after the other, and
    (FP32 storage) their 32-bit values."""

    def __init__(self, nc, volumes, bits):
        self.nc, self.bits, self.at = nc, bits, np.concatenate([[0], np.cumsum(volumes)])
        n = int(self.at[-1])
        self.U, self.E = tcym.pinned_empty((n, 3, NM[nc])), tcym.pinned_empty((n, 3, NA[nc]))
        if bits == 32:
            self.U32, self.E32 = (torch.empty(x.shape, dtype=torch.float32) for x in (self.U, self.E))

    def arrays(self, i):
        a, b = int(self.at[i]), int(self.at[i + 1])
        return self.U[a:b], self.E[a:b]

    def values(self, u=True):
        if self.bits == 64:
            return ([self.U] if u else []) + [self.E]
        if u:
            self.U32.copy_(torch.from_numpy(self.U))
        self.E32.copy_(torch.from_numpy(self.E))
        return ([self.U32] if u else []) + [self.E32]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.seed, s.step = case, int(seed), 0
    prec = tcym.FP32 if case["bits"] == 32 else tcym.FP64
    shapes = _shapes(case)
    s.host = {nc: _HostState(nc, [int(np.prod(n)) for c, n in shapes if c == nc], case["bits"])
              for nc in sorted({c for c, _ in shapes})}
    for nc, h in s.host.items():
        U, E = _inputs(case, nc, int(h.at[-1]), seed)
        torch.from_numpy(h.U).copy_(U)
        torch.from_numpy(h.E).copy_(E)
    s.lats, s.slot, used = [], [], {2: 0, 3: 0}
    for nc, n in shapes:
        lat = tcym.Lattice(_ctx(), nc, n, prec)
        s.slot.append(used[nc])
        used[nc] += 1
        lat.upload(*s.host[nc].arrays(s.slot[-1]))
        s.lats.append(lat)
    if case["what"] == "langevin":
        s.lats[0].ncs_track(case["every"])
        s.lats[0].ncs_reset()
    if case["what"] == "ensemble":
        s.ens = tcym.Ensemble(_ctx())
        for lat in s.lats:
            lat.ncs_reset()
            s.ens.add(lat, DT)
    if case["what"] == "restore":
        s.E0 = tcym.pinned_empty(s.host[case["nc"]].E.shape)  # the field before the restore
        s.E0[...] = s.host[case["nc"]].E
    return s


# -------------------------------------------------------------------- a pass
def _numbers(values, bits):
    return np.array(values, dtype=np.float32 if bits == 32 else np.float64)


def _observables(lat):
    o = lat.observables()
    return [o.T00, o.electric, o.magnetic, *o.esqr, *o.bsqr, o.gauss_rms, o.gauss_absmax, o.edotb]


def run(s):
    case, lat = s.case, s.lats[0]
    what, steps, every, bits = case["what"], case["steps"], case["every"], case["bits"]
    series = []
    if what == "ensemble":
        for a in range(0, steps, every):
            n = min(every, steps - a)
            s.ens.step(n)
            edotb, ncs = s.ens.measure(n)
            series.append([edotb, ncs])
        for (nc, _), slot, member in zip(_shapes(case), s.slot, s.lats):
            member.download(*s.host[nc].arrays(slot))
        return {"series": _numbers(series, bits), "state": [s.host[nc].values() for nc in sorted(s.host)]}
    host = s.host[case["nc"]]
    if what == "restore":
        lat.upload(None, s.E0)
        lat.gauss_restore(1e-14, steps)
        lat.download(*host.arrays(0))
        return {"field": host.values(u=False)}
    if what == "langevin":
        lat.langevin(DT_LANGEVIN, GAMMA, TEMPERATURE, s.seed, s.step, steps)
        s.step += steps
        series = [lat.ncs()]
    else:
        for a in range(0, steps, every):
            n = min(every, steps - a)
            if what == "flow":
                lat.flow(DTAU, n, tcym.FLOW_CHECKERBOARD if case["sweep"] == "checkerboard" else tcym.FLOW_SIMULTANEOUS)
            else:
                lat.leapfrog(DT, n)
            series.append(_observables(lat))
    lat.download(*host.arrays(0))
    return {"series": _numbers(series, bits), "state": host.values()}


# --------------------------------------------------------------- what it costs
def work(case):
    """Bytes: the stored links and fields (FP32: 16 + 12 and 48 + 32 bytes a link, FP64: 32 + 24 and
    144 + 64) read and written once by each step or sweep, read once by each measurement, and the state
    read out once as doubles; a restore's iteration reads the links and updates the fields three times.
    Flops: a step's 18 group products a site (SU(3) 198, SU(2) 28 operations each), a third more for the
    exponentials; a measurement's 42; an iteration's 3 x 12."""
    total = {"bytes": 0.0, "flops": 0.0}
    for nc, n in _shapes(case):
        sites = float(np.prod(n))
        u = {(2, 32): 16, (2, 64): 32, (3, 32): 48, (3, 64): 144}[nc, case["bits"]]
        e = {(2, 32): 12, (2, 64): 24, (3, 32): 32, (3, 64): 64}[nc, case["bits"]]
        product = {2: 28, 3: 198}[nc]
        out = 8 * (NM[nc] + NA[nc])
        if case["what"] == "restore":
            total["bytes"] += 3 * sites * (3 * case["steps"] * (u + 2 * e) + out + 8 * NA[nc])
            total["flops"] += 36 * case["steps"] * sites * product
            continue
        measured = -(-case["steps"] // case["every"]) if case["what"] != "langevin" else case["steps"] // case["every"]
        rw = 2 * u if case["sweep"] == "checkerboard" else 2 * (u + e)
        total["bytes"] += 3 * sites * (case["steps"] * rw + measured * (u + e) + out)
        total["flops"] += sites * product * (24 * case["steps"] + 42 * measured)
    return total


# ------------------------------------------------- the same in plain torch, 64 bits
def _at(a, mu, k=1):
    """The field a (..., nz, ny, nx, i, j) at x + k mu."""
    return torch.roll(a, -k, -3 - mu)


def _proj(v, t):
    """Re tr(i t^a v)."""
    return -torch.einsum("aij,...ji->...a", t, v).imag


def _transported_back(u, e, mu, t):
    """Components of U_mu^dag E_mu U_mu at x - mu, as seen from x."""
    h = torch.tensordot(e.to(torch.complex128), t, 1)
    w = _at(_mul(_mul(_dag(u), h), u), mu, -1)
    return 2 * torch.einsum("aij,...ji->...a", t, w).real


def _staples(U, mu):
    out = 0
    for nu in range(3):
        if nu != mu:
            out = out + _mul(_mul(_at(U[nu], mu), _dag(_at(U[mu], nu))), _dag(U[nu]))
            out = out + _at(_mul(_mul(_dag(_at(U[nu], mu)), _dag(U[mu])), U[nu]), nu, -1)
    return out


def _force(U, mu, t):
    return _proj(_mul(U[mu], _staples(U, mu)), t)


def _gauss(U, E, t):
    return sum(E[mu] - _transported_back(U[mu], E[mu], mu, t) for mu in range(3))


def _edotb(U, E, t):
    """Clover E.B summed over each lattice, and the three plaquettes' 4 Re tr(1 - P)."""
    out, b2 = 0, []
    for mu in range(3):
        j, k = (mu + 1) % 3, (mu + 2) % 3
        x, y = U[j], U[k]
        xk, yj = _at(x, k), _at(y, j)  # U_j(x+k), U_k(x+j)
        q = _mul(_mul(x, yj), _mul(_dag(xk), _dag(y)))
        b2.append(4 * (x.shape[-1] - torch.diagonal(q, dim1=-2, dim2=-1).sum(-1).real))
        q = q + _at(_mul(_mul(yj, _dag(xk)), _mul(_dag(y), x)), j, -1)
        q = q + _at(_mul(_mul(_dag(y), x), _mul(yj, _dag(xk))), k, -1)
        q = q + _at(_at(_mul(_mul(_dag(xk), _dag(y)), _mul(x, yj)), j, -1), k, -1)
        e = 0.5 * (E[mu] + _transported_back(U[mu], E[mu], mu, t))
        out = out + (e * 2 * _proj(0.25 * q, t)).sum((-4, -3, -2, -1))
    return out, b2


def _exact_observables(U, E, t):
    edotb, b2 = _edotb(U, E, t)
    g = _gauss(U, E, t)
    esqr = [float((e * e).sum(-1).mean()) for e in E]
    bsqr = [float(b.mean()) for b in b2]
    return [0.5 * (sum(esqr) + sum(bsqr)), 0.5 * sum(esqr), 0.5 * sum(bsqr), *esqr, *bsqr,
            float((g * g).mean().sqrt()), float(g.abs().max()), float(edotb.sum())]


def _philox(c, key):
    """Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF
    k0, k1 = key & mask, (key >> 32) & mask

    def product(m, x):
        lo, hi = m * (x & 0xFFFF), m * (x >> 16)
        mid = hi + (lo >> 16)
        return (mid >> 16) & mask, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    for _ in range(10):
        hi0, lo0 = product(0xD2511F53, c[0])
        hi1, lo1 = product(0xCD9E8D57, c[2])
        c = [hi1 ^ c[1] ^ k0, lo1, hi0 ^ c[3] ^ k1, lo0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _noise(volume, mu, na, seed, step):
    """The library's documented noise stream: counter (site, step, 0, mu << 8 | j), key the seed;
    Box-Muller pairs for the components 2j and 2j + 1."""
    site = torch.arange(volume, dtype=torch.int64, device=_device())
    z = []
    for j in range((na + 1) // 2):
        c = _philox([site, torch.full_like(site, step), torch.zeros_like(site),
                     torch.full_like(site, (mu << 8) | j)], seed)
        r = torch.sqrt(-2 * torch.log((c[0].double() + 1) * 2.0 ** -32))
        phi = 2 * math.pi * (c[1].double() * 2.0 ** -32)
        z += [r * torch.cos(phi), r * torch.sin(phi)]
    return torch.stack(z[:na], -1)


def _exact_step(case, U, E, t, seed, step):
    what = case["what"]
    if case["sweep"] == "checkerboard":
        n = U[0].shape[-5:-2]
        z, y, x = torch.meshgrid(*(torch.arange(k, device=U[0].device) for k in n), indexing="ij")
        for parity in (0, 1):
            here = ((x + y + z) % 2 == parity)[..., None, None]
            for mu in range(3):
                new = _mul(_expi(2 * DTAU * _force(U, mu, t), t), U[mu])
                U[mu] = torch.where(here, new, U[mu])
        return U, E
    dt = {"flow": DTAU, "langevin": DT_LANGEVIN}.get(what, DT)
    f = [_force(U, mu, t) for mu in range(3)]
    for mu in range(3):
        if what == "flow":
            E[mu] = -2 * f[mu]
        elif what == "langevin":
            xi = _noise(E[mu][..., 0].numel(), mu, E[mu].shape[-1], seed, step).reshape(E[mu].shape)
            E[mu] = E[mu] - 2 * dt * f[mu] - GAMMA * dt * E[mu] + math.sqrt(GAMMA * dt * 2 * TEMPERATURE) * xi
        else:
            E[mu] = E[mu] - 2 * dt * f[mu]
        U[mu] = _mul(_expi(-dt * E[mu], t), U[mu])
    return U, E


def _split(nc, n, U, E):
    """Host-layout arrays of equal lattices, one after the other, as lists over mu of fields
    (lattice, nz, ny, nx, ...)."""
    shape = (-1, n[2], n[1], n[0])
    u = _from_host_layout(U, nc).contiguous().reshape(*shape, 3, nc, nc)
    e = E.reshape(*shape, 3, NA[nc])
    return [u[..., mu, :, :].contiguous() for mu in range(3)], [e[..., mu, :].contiguous() for mu in range(3)]


def _join(nc, U, E):
    u = _to_host_layout(torch.stack(U, -3), nc)
    return u.reshape(-1, 3, NM[nc]), torch.stack(E, -2).reshape(-1, 3, NA[nc])


def exact(case, seed):
    """The first pass in 64 bits.  None where it would take over about 15 seconds (SU(3) 96^3, 80 steps: 6)."""
    shapes = _shapes(case)
    sites = sum(float(np.prod(n)) * (1 if nc == 3 else 0.4) for nc, n in shapes)
    if sites * case["steps"] * (3 if case["sweep"] == "checkerboard" else 1) > 1e8:
        return None
    dev, steps, every = _device(), case["steps"], case["every"]
    if case["what"] == "ensemble":
        at, parts = {2: 0, 3: 0}, {}
        start = {nc: _inputs(case, nc, sum(int(np.prod(n)) for c, n in shapes if c == nc), seed)
                 for nc in sorted({c for c, _ in shapes})}
        for i, (nc, n) in enumerate(shapes):
            parts.setdefault((nc, n), []).append((i, at[nc]))
            at[nc] += int(np.prod(n))
        series = np.zeros((-(-steps // every), 2, len(shapes)))
        for (nc, n), where in parts.items():
            t, v = _generators(nc, dev), int(np.prod(n))
            rows = torch.cat([torch.arange(a, a + v, device=dev) for _, a in where])
            U, E = _split(nc, n, start[nc][0][rows], start[nc][1][rows])
            ncs, index = 0, [i for i, _ in where]
            for k, a in enumerate(range(0, steps, every)):
                m = min(every, steps - a)
                for _ in range(m):
                    U, E = _exact_step(case, U, E, t, 0, 0)
                edotb = _edotb(U, E, t)[0]
                ncs = ncs + DT * m * edotb / (8 * math.pi ** 2)
                series[k, 0, index], series[k, 1, index] = edotb.cpu().numpy(), ncs.cpu().numpy()
            start[nc][0][rows], start[nc][1][rows] = _join(nc, U, E)
        return {"series": series, "state": [list(start[nc]) for nc in sorted(start)]}
    nc, n = shapes[0]
    t = _generators(nc, dev)
    U, E = _split(nc, n, *_inputs(case, nc, int(np.prod(n)), seed))
    series = []
    if case["what"] == "restore":
        for _ in range(steps):
            for g in (7 / 24, 7 / 48, 7 / 72):
                G = _gauss(U, E, t)
                H = torch.tensordot(G.to(torch.complex128), t, 1)
                for mu in range(3):
                    w = _mul(_mul(U[mu], _at(H, mu)), _dag(U[mu]))
                    E[mu] = E[mu] - g * (G - 2 * torch.einsum("aij,...ji->...a", t, w).real)
        return {"field": [_join(nc, U, E)[1]]}
    ncs = 0.0
    for k in range(steps):
        U, E = _exact_step(case, U, E, t, int(seed), k)
        if case["what"] == "langevin":
            if (k + 1) % every == 0:
                ncs += DT_LANGEVIN * every * float(_edotb(U, E, t)[0].sum()) / (8 * math.pi ** 2)
        elif (k + 1) % every == 0 or k + 1 == steps:
            series.append(_exact_observables(U, E, t))
    if case["what"] == "langevin":
        series = [ncs]
    return {"series": np.array(series), "state": list(_join(nc, U, E))}
