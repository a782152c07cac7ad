"""Workloads whose time and results describe this framework in use.

Three kinds of case, each through public entry points:

* ``fix``    -- the batched engine (``GaugeFixer``): import one or more lattices, run a gauge-fixing
  schedule on them, export the fixed fields.  The context, with its launch shapes tuned, is kept
  from call to call, as a program that fixes many configurations keeps it.
* ``driver`` -- a driver loop on the plugin classes (``LandauKernelsSU3`` ... ``GaugeFixingStats``), in
  place on one field in the reference layout.
* ``site``   -- the quality of a field, per site and averaged, as a diagnostics program asks for it.

Fields are synthetic: links near 1 (strength ``eps``) under a Haar-random gauge transformation, or
Haar-random links, drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from su3_ma_gauge_gpu_b200 import (CommonKernelsSU3, CoulombKernelsSU3, GaugeFixingStats, LandauKernelsSU3,
                                   MAGKernelsSU3, U1xU1KernelsSU3)
from su3_ma_gauge_gpu_b200.engine import GaugeFixer, Schedule

KERNELS = {"landau": LandauKernelsSU3, "coulomb": CoulombKernelsSU3, "mag": MAGKernelsSU3, "u1xu1": U1xU1KernelsSU3}
RNG_SEED = 7          # Philox key word of the random updates
OMEGA = 1.7           # overrelaxation parameter
SR_PROBABILITY = 0.7  # stochastic relaxation


def listed():
    fix = dict(kind="fix", mixed="no", host=False, eps=0.3, random_trafo=False, sa=0, sa_max=1.0, micro_every=1,
               check=20, reproject=100)
    return [
        # one sweep and its check on a lattice of a few thousand links: launches and host calls
        dict(name="landau_4x8_driver", kind="driver", gauge="landau", size="4x4x4x8", real=64, eps=0.3,
             steps="or or stats", temperature=0.5),
        # the 8^4 plain double-precision fix from Haar-random links, first 400 sweeps of it
        dict(fix, name="plain8_fix", gauge="landau", sizes="8x8x8x8", eps=0.0, sweeps=400),
        # one configuration from host memory and back, double precision, an uneven lattice
        dict(fix, name="landau_host_fix", gauge="landau", sizes="20x10x14x18", host=True, sweeps=41),
        # Gribov copies of uneven lattices in one batch, each from its own random gauge
        dict(fix, name="gribov_fix", gauge="landau", sizes="12x12x12x12*6 16x16x16x16*6 40x20x20x20*4", mixed="refine",
             random_trafo=True, sweeps=41),
        # the 32^4 mixed-precision Landau fix, its first 61 sweeps
        dict(fix, name="landau32_refine_fix", gauge="landau", sizes="32x32x32x32", mixed="refine", sweeps=61),
        # Coulomb, all timeslices batched: a short annealing with microcanonical steps, then overrelaxation
        dict(fix, name="coulomb48_refine_fix", gauge="coulomb", sizes="16x48x48x48", mixed="refine", sa=6,
             micro_every=3, sweeps=21),
        # maximal Abelian gauge, the largest lattice: a short geometric annealing, then overrelaxation
        dict(fix, name="mag48_refine_fix", gauge="mag", sizes="48x48x48x48", mixed="refine", eps=0.5, sa=8, sa_max=1.4,
             sweeps=21),
        # the reference driver's loop in double precision: sweeps, reprojection, check
        dict(name="landau32_driver", kind="driver", gauge="landau", size="32x32x32x32", real=64, eps=0.3,
             steps="or or or or micro project stats", temperature=0.5),
        # the MAG driver's phases in double precision on an uneven lattice
        dict(name="mag_driver", kind="driver", gauge="mag", size="22x14x18x10", real=64, eps=0.5,
             steps="random sa micro sa sr or or project stats", temperature=0.7),
        # a single-precision driver: heat bath with microcanonical steps
        dict(name="landau32_sa_driver_fp32", kind="driver", gauge="landau", size="32x32x32x32", real=32, eps=0.3,
             steps="sa micro sa micro or stats", temperature=0.4),
        # a Coulomb timeslice in single precision, as the slice-by-slice driver sweeps it
        dict(name="coulomb_slice_driver_fp32", kind="driver", gauge="coulomb", size="1x32x24x20", real=32, eps=0.3,
             steps="or or or or project stats", temperature=0.5),
        # quality of a loaded configuration, per site and averaged
        dict(name="site_quality", kind="site", gauge="mag", size="24x24x24x24", real=64, eps=0.3),
    ]


def _even(rng, lo, hi):
    """An even extent between lo and hi, spread over its logarithm."""
    return 2 * max(1, round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))


def _text(size):
    return "x".join(str(v) for v in size)


def draw(rng):
    gauge = rng.choice(("landau", "coulomb", "mag", "u1xu1"))
    kind = rng.choice(("fix", "fix", "driver", "driver", "site"))
    eps = round(rng.uniform(0.2, 0.5), 3)
    while True:
        # Coulomb timeslices need a multiple of 16 sites, which three even extents do not always give
        size = [_even(rng, 4, 40) for _ in range(4)]
        if gauge != "coulomb" or size[1] * size[2] * size[3] % 16 == 0:
            break
    if kind == "fix":
        mixed = rng.choice(("no", "yes", "refine"))
        copies = rng.choice((1, 1, 1, 2, 3)) if math.prod(size) <= 500_000 else 1
        return dict(kind="fix", gauge=gauge, sizes=_text(size) + "*%d" % copies, mixed=mixed, host=rng.random() < 0.2,
                    eps=eps, random_trafo=rng.random() < 0.3, sa=rng.choice((0, 0, 2, 5)),
                    sa_max=round(rng.uniform(0.3, 1.4), 3), micro_every=rng.choice((1, 2, 3)), check=rng.choice((10, 20)),
                    reproject=rng.choice((30, 100)), sweeps=rng.randrange(11, 42))
    real = rng.choice((32, 64))
    if gauge == "coulomb":
        size[0] = 1
    if kind == "site":
        return dict(kind="site", gauge=gauge, size=_text(size), real=real, eps=eps)
    rules = ["or", "or", "or", "micro", "sa"] + (["sr"] if gauge == "mag" else [])
    steps = [rng.choice(rules) for _ in range(rng.randrange(2, 6))] + rng.choice(([], ["project"])) + ["stats"]
    return dict(kind="driver", gauge=gauge, size=_text(size), real=real, eps=eps, steps=" ".join(steps),
                temperature=round(rng.uniform(0.1, 1.0), 3))


def _size(text):
    return tuple(int(v) for v in text.split("x"))


def _lattices(case):
    out = []
    for part in case["sizes"].split():
        size, _, count = part.partition("*")
        out += [_size(size)] * int(count or 1)
    return out


# ---- synthetic fields ----------------------------------------------------------------------------
# A field is a complex tensor [4, 3, 3, V] in the parity-split site order of the reference layout:
# site l = ((t*Nx + x)*Ny + y)*Nz + z at index l//2, + V/2 for odd t + x + y + z.

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _coordinates(size, device):
    """Coordinates of every site in split order, [4, V]."""
    nt, nx, ny, nz = size
    V = math.prod(size)
    h = torch.arange(V // 2, device=device)
    l = torch.cat([2 * h, 2 * h])
    z, y, x, t = l % nz, l // nz % ny, l // (nz * ny) % nx, l // (nz * ny * nx)
    odd = torch.cat([torch.zeros_like(h), torch.ones_like(h)])
    return torch.stack([t, x, y, z + ((t + x + y + z) % 2 != odd)])


def _index(size, c):
    nt, nx, ny, nz = size
    l = ((c[0] * nx + c[1]) * ny + c[2]) * nz + c[3]
    return l // 2 + (c.sum(dim=0) % 2) * (math.prod(size) // 2)


def _neighbours(size, step, device):
    """Index of x + step * mu for every site x and direction mu."""
    c = _coordinates(size, device)
    out = []
    for mu in range(4):
        d = c.clone()
        d[mu] = (d[mu] + step) % size[mu]
        out.append(_index(size, d))
    return out


def _third_row(a):
    """Row 2 of SU(3) matrices [..., 3, 3, V] from rows 0 and 1: conj(row0 x row1), normalised."""
    r0, r1 = a[..., 0, :, :], a[..., 1, :, :]
    c = (torch.roll(r0, -1, -2) * torch.roll(r1, -2, -2) - torch.roll(r0, -2, -2) * torch.roll(r1, -1, -2)).conj()
    return c / c.abs().square().sum(dim=-2, keepdim=True).sqrt()


def _unitary(a):
    """SU(3) from [3, 3, V]: Gram-Schmidt of rows 0 and 1, row 2 from them."""
    r0 = a[0] / a[0].abs().square().sum(dim=0).sqrt()
    r1 = a[1] - (a[1] * r0.conj()).sum(dim=0) * r0
    r1 = r1 / r1.abs().square().sum(dim=0).sqrt()
    out = torch.stack([r0, r1, torch.empty_like(r0)])
    out[2] = _third_row(out)
    return out


def _mul(a, b, adjoint=False):
    """a b, or a b^dagger, of [3, 3, V] matrices."""
    rows = []
    for i in range(3):
        rows.append(torch.stack([sum(a[i, k] * (b[j, k].conj() if adjoint else b[k, j]) for k in range(3))
                                 for j in range(3)]))
    return torch.stack(rows)


def _gaussian(shape, gen):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device=gen.device, dtype=torch.float64))


def _near_one(V, eps, gen):
    a = _gaussian((3, 3, V), gen)
    ih = 1j * eps * 0.5 * (a + a.conj().transpose(0, 1))
    m = ih + 0.5 * _mul(ih, ih)
    for i in range(3):
        m[i, i] += 1.0
    return _unitary(m)


def _field(size, eps, seed):
    """Links near 1 (Haar-random ones for eps = 0) under a Haar-random gauge transformation, [4, 3, 3, V]."""
    gen = torch.Generator(device=_device()).manual_seed(seed)
    V = math.prod(size)
    g = _unitary(_gaussian((3, 3, V), gen))
    out = torch.empty((4, 3, 3, V), dtype=torch.complex128, device=gen.device)
    for mu, up in enumerate(_neighbours(size, 1, gen.device)):
        u = _near_one(V, eps, gen) if eps else _unitary(_gaussian((3, 3, V), gen))
        out[mu] = _mul(_mul(g, u), g[:, :, up], adjoint=True)
    return out


def _to_layout(u, dtype):
    """[4, 3, 3, V] -> the reference layout's array of 72 V reals."""
    return torch.view_as_real(u).permute(0, 1, 2, 4, 3).to(dtype).reshape(-1)


def _from_layout(r, V):
    return torch.view_as_complex(r.double().reshape(4, 3, 3, 2, V).permute(0, 1, 2, 4, 3).contiguous())


def _timeslices(u, size):
    """The field as the array of its Nt timeslices, [Nt][4, 3, 3, Vs], each in its own split order."""
    device = u.device
    slice_size = (1,) + tuple(size[1:])
    c = _coordinates(slice_size, device)
    out = []
    for t in range(size[0]):
        ct = c.clone()
        ct[0] = t
        out.append(u[..., _index(size, ct)])
    return out


def _dtype(real):
    return torch.float64 if real == 64 else torch.float32


def _fix_input(case, size, seed):
    u = _field(size, case["eps"], seed)
    if case["gauge"] == "coulomb":
        return torch.cat([_to_layout(s, torch.float64) for s in _timeslices(u, size)])
    return _to_layout(u, torch.float64)


def _driver_input(case, seed):
    """The field of a driver case, and for Coulomb slices that of timeslice t - 1, else None."""
    size, dtype = _size(case["size"]), _dtype(case["real"])
    up = _to_layout(_field(size, case["eps"], seed), dtype)
    return up, _to_layout(_field(size, case["eps"], seed + 1_000_003), dtype) if case["gauge"] == "coulomb" else None


# ---- the cases -----------------------------------------------------------------------------------

def prepare(case, seed):
    precision = "double" if case.get("real", 64) == 64 else "float"
    if case["kind"] == "fix":
        sizes = _lattices(case)
        fields = [_fix_input(case, s, seed + 17 * k) for k, s in enumerate(sizes)]
        outs = [torch.empty_like(f) for f in fields]
        fixer = GaugeFixer(sizes, gauge=case["gauge"], mixed={"no": False, "yes": True, "refine": "refine"}[case["mixed"]])
        for k, f in enumerate(fields):
            fixer.load(k, f)
        fixer.autotune()
        if case["host"]:  # page-locked host arrays, as a program that streams configurations keeps them
            fields = [f.cpu().pin_memory().numpy() for f in fields]
            outs = [torch.empty(f.shape, dtype=torch.float64).pin_memory().numpy() for f in fields]
        schedule = Schedule(random_trafo=int(case["random_trafo"]), seed=RNG_SEED, sa_steps=case["sa"], sa_min=0.01,
                            sa_max=case["sa_max"], sa_geometric=int(case["gauge"] == "mag"), micro_updates=1,
                            micro_every=case["micro_every"], or_max_iter=case["sweeps"], or_parameter=OMEGA,
                            precision=1e-12, switch_theta=1e-9, check_precision=case["check"],
                            reproject=case["reproject"])
        return dict(case=case, fixer=fixer, fields=fields, outs=outs, schedule=schedule)
    size = _size(case["size"])
    up, down = _driver_input(case, seed)
    kernels = KERNELS[case["gauge"]](size, precision)
    stats = GaugeFixingStats(up, size, KERNELS[case["gauge"]], "AVERAGE", precision)
    state = dict(case=case, kernels=kernels, stats=stats, up=up, down=down)
    if case["kind"] == "site":
        V = math.prod(size)
        state["gff"], state["theta"] = (torch.empty(V, dtype=torch.float64, device=up.device) for _ in range(2))
    else:
        state["common"] = CommonKernelsSU3(size, precision)
    return state


def _run_driver(state):
    case, k, up, down = state["case"], state["kernels"], state["up"], state["down"]
    field = (up, down) if down is not None else (up,)
    counter = 0
    for step in case["steps"].split():
        if step == "project":
            state["common"].projectSU3(0, 0, up)
        elif step == "stats":
            state["stats"].generateGaugeQuality()
        else:
            for parity in (0, 1):
                if step == "or":
                    k.orStep(0, 0, *field, None, parity, OMEGA)
                elif step == "micro":
                    k.microStep(0, 0, *field, None, parity)
                elif step == "sa":
                    k.saStep(0, 0, *field, None, parity, case["temperature"], RNG_SEED, counter)
                elif step == "sr":
                    k.srStep(0, 0, *field, None, parity, SR_PROBABILITY, RNG_SEED, counter)
                else:
                    k.randomTrafo(0, 0, *field, None, parity, RNG_SEED, counter)
                counter += step in ("sa", "sr", "random")
    out = dict(up=up, gff=state["stats"].getCurrentGff(), theta=state["stats"].getCurrentA())
    return out if down is None else dict(out, down=down)


def run(state):
    kind = state["case"]["kind"]
    if kind == "fix":
        fixer = state["fixer"]
        for k, f in enumerate(state["fields"]):
            fixer.load(k, f)
        reports = fixer.fix(state["schedule"])
        for k, f in enumerate(state["outs"]):
            fixer.store(k, f)
        return dict(fields=state["outs"], gff=np.array([r.gff for r in reports]),
                    theta=np.array([r.theta for r in reports]))
    if kind == "site":
        state["kernels"].generateGaugeQualityPerSite(0, 0, state["up"], state["gff"], state["theta"])
        state["stats"].generateGaugeQuality()
        return dict(gff=state["gff"], theta=state["theta"], mean_gff=state["stats"].getCurrentGff(),
                    mean_theta=state["stats"].getCurrentA())
    return _run_driver(state)


def work(case):
    """Bytes: the field read once and written once per sweep or reprojection (12 reals per link move,
    18 where row 2 is written), read once per check, 12 in and 18 out at import and export.
    Operations: 2274 per site update (an overrelaxation update's), 1000 per site for a check."""
    if case["kind"] == "fix":
        links = 4 * sum(math.prod(s) for s in _lattices(case))
        real = 8 if case["mixed"] == "no" else 4
        sweeps = case["sweeps"] + int(case["random_trafo"]) + case["sa"] + case["sa"] // case["micro_every"]
        checks = 1 + math.ceil((case["sweeps"] - 1) / case["check"])
        return dict(bytes=links * (sweeps * 24 * real + checks * 12 * real + 30 * 8),
                    flops=links / 4 * (2274 * sweeps + 1000 * checks))
    links, real = 4 * math.prod(_size(case["size"])), case["real"] // 8
    if case["kind"] == "site":
        return dict(bytes=links * 12 * real * 2 + links / 4 * 16, flops=2 * links / 4 * 1000)
    steps = case["steps"].split()
    sweeps = sum(s not in ("project", "stats") for s in steps)
    return dict(bytes=links * real * (24 * sweeps + 30 * steps.count("project") + 12 * steps.count("stats")),
                flops=links / 4 * (2274 * sweeps + 1000 * steps.count("stats")))


# ---- the same in 64 bits with torch ---------------------------------------------------------------

def _philox(x0, counter, key0, seed):
    """Philox4x32-10 of counter (x0, counter, 0x12345678, 0xabcdef09) and key (key0, seed), on int64 tensors."""
    mask = 0xFFFFFFFF

    def product(a, x):
        low, high = x * (a & 0xFFFF), x * (a >> 16)
        return (high + (low >> 16)) >> 16, (low + ((high & 0xFFFF) << 16)) & mask

    c = [x0, torch.full_like(x0, counter), torch.full_like(x0, 0x12345678), torch.full_like(x0, 0xABCDEF09)]
    k0, k1 = key0, seed
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        hi0, lo0 = product(0xD2511F53, c[0])
        hi1, lo1 = product(0xCD9E8D57, c[2])
        c = [hi1 ^ c[1] ^ k0, lo1, hi0 ^ c[3] ^ k1, lo0]
    return c


class _Draws:
    """The uniform numbers of every site of a parity: draw n of a site comes from Philox block
    1 + n / (numbers per block), last word first."""

    def __init__(self, sites, real, seed, counter, device):
        h = torch.arange(sites, device=device)
        self.tid, self.real, self.seed, self.counter = (h >> 5) * 256 + (h & 31), real, seed, counter
        self.n = torch.zeros_like(h)

    def next(self, at=None):
        n = self.n if at is None else self.n[at]
        tid = self.tid if at is None else self.tid[at]
        per = 4 if self.real == 32 else 2
        w = _philox(1 + n // per, self.counter, tid, self.seed)
        if self.real == 32:
            v = torch.stack(w[::-1]).gather(0, (n % 4)[None])[0]
            u = (1 + (v >> 8)).double() * float.fromhex("0x1.fffffep-25")
        else:
            first = n % 2 == 0
            hi, lo = torch.where(first, w[3], w[1]), torch.where(first, w[2], w[0])
            u = (1 + ((hi << 21) | (lo >> 11))).double() * float.fromhex("0x1.fffffffffffffp-54")
        if at is None:
            self.n = self.n + 1
        else:
            self.n[at] += 1
        return u


def _norm(a):
    return a.square().sum(dim=0).sqrt()


def _heat_bath(a, temperature, draws):
    """Kennedy-Pendleton heat bath of the SU(2) element a [4, N]."""
    norm = _norm(a)
    e = torch.stack([a[0], -a[1], -a[2], -a[3]]) / norm
    p0 = float(np.float32(temperature)) / norm
    delta = torch.zeros_like(p0)
    at = torch.arange(p0.numel(), device=p0.device)

    def above(at):
        r = draws.next(at)
        while True:
            low = torch.nonzero(r < 0.0001)[:, 0]
            if not low.numel():
                return r
            r[low] = draws.next(at[low])

    while at.numel():
        r1 = -torch.log(above(at)) * p0[at]
        r2 = -torch.log(above(at)) * p0[at]
        r3 = torch.cos(2 * math.pi * draws.next(at)).square()
        d = r2 + r1 * r3
        r4 = draws.next(at)
        delta[at] = d
        at = at[r4 * r4 > 1.0 - 0.5 * d]
    a0 = 1.0 - delta
    cos_theta = 2.0 * draws.next() - 1.0
    sin_theta, sin_alpha = (1.0 - cos_theta ** 2).sqrt(), (1.0 - a0 ** 2).sqrt()
    phi = 2.0 * math.pi * draws.next()
    a1, a2, a3 = sin_alpha * sin_theta * torch.cos(phi), sin_alpha * sin_theta * torch.sin(phi), sin_alpha * cos_theta
    return torch.stack([a0 * e[0] + a3 * e[3] + a2 * e[2] + e[1] * a1, a2 * e[3] + a1 * e[0] - a3 * e[2] - e[1] * a0,
                        a3 * e[1] - a0 * e[2] + a2 * e[0] - a1 * e[3], e[0] * a3 - e[3] * a0 + a1 * e[2] - a2 * e[1]])


def _update(rule, a, parameter, draws):
    v2, a02 = a[1:].square().sum(dim=0), a[0] ** 2
    if rule == "or":
        b = (float(np.float32(parameter)) * a02 + v2) / (a02 + v2)
        return torch.cat([a[:1], b * a[1:]]) / (a02 + b * b * v2).sqrt()
    if rule == "micro":
        return torch.cat([((a02 - v2) / (a02 + v2))[None], 2.0 * a[0] / (a02 + v2) * a[1:]])
    if rule == "sa":
        return _heat_bath(a, parameter, draws)
    if rule == "sr":
        square = torch.cat([(a02 - v2)[None], 2.0 * a[0] * a[1:]])
        a = torch.where(draws.next() < float(np.float32(parameter)), square, a)
        return a / _norm(a)
    alpha, phi, cos_theta = math.pi * draws.next(), 2.0 * math.pi * draws.next(), 2.0 * draws.next() - 1.0
    s = (1.0 - cos_theta ** 2).sqrt() * torch.sin(alpha)
    return torch.stack([torch.cos(alpha), s * torch.cos(phi), s * torch.sin(phi), torch.sin(alpha) * cos_theta])


def _coupling(gauge, up, dn, i, j):
    """The SU(2) quaternion (i, j) of the links up, dn [n, 3, 3, N] of a site's directions."""
    if gauge == "mag":
        a = up[:, [i, i, j, j], [i, j, i, j]]
        b = dn[:, [i, i, j, j], [i, j, i, j]]
        sign = torch.tensor([1.0, -1.0, -1.0, 1.0], device=up.device)[None, :, None]
        D = ((a.abs().square() + b.abs().square()) * sign).sum(dim=(0, 1))
        c = (a[:, 0] * a[:, 2].conj() - a[:, 1] * a[:, 3].conj()).sum(dim=0)
        d = (b[:, 0].conj() * b[:, 1] - b[:, 2].conj() * b[:, 3]).sum(dim=0)
        w1, w2 = 2.0 * (c.imag + d.imag), 2.0 * (c.real + d.real)
        return torch.stack([D + (D * D + w1 * w1 + w2 * w2).sqrt(), w1, w2, torch.zeros_like(D)])
    q = torch.zeros(4, up.shape[-1], dtype=torch.float64, device=up.device)
    for m, s in ((up, -1.0), (dn, 1.0)):
        m = m.sum(dim=0)
        q += torch.stack([m[i, i].real + m[j, j].real, s * (m[i, j].imag + m[j, i].imag),
                          s * (m[i, j].real - m[j, i].real), s * (m[i, i].imag - m[j, j].imag)])
    if gauge == "u1xu1":
        q[1:3] = 0
    return q


def _pass(gauge, rule, u, size, parity, parameter, draws, down=None):
    """One parity pass in place on u [4, 3, 3, V] (rows 0 and 1 of each link; row 2 is rebuilt from them).
    down: for Coulomb, the field that holds the temporal links of timeslice t - 1."""
    V = math.prod(size)
    s = torch.arange(V // 2, device=u.device) + parity * (V // 2)
    nb = _neighbours(size, -1, u.device)
    links = []
    for mu in range(4):
        here = u[mu][:, :, s]
        below = (down if down is not None and mu == 0 else u)[mu][:, :, s if mu == 0 and gauge == "coulomb" else nb[mu][s]]
        links.append((here, below))
    up, dn = torch.stack([a for a, _ in links]), torch.stack([b for _, b in links])
    del links
    up[:, 2], dn[:, 2] = _third_row(up), _third_row(dn)
    first = 1 if gauge == "coulomb" else 0
    for i, j in ((0, 2), (1, 2), (0, 1)):
        g = _update(rule, _coupling(gauge, up[first:], dn[first:], i, j), parameter, draws)
        if gauge in ("u1xu1", "mag"):
            g[[1, 2] if gauge == "u1xu1" else [3]] = 0
            g = g / _norm(g)
        g00, g01 = torch.complex(g[0], g[3]), torch.complex(g[2], g[1])
        ri, rj = up[:, i].clone(), up[:, j].clone()
        up[:, i], up[:, j] = g00 * ri + g01 * rj, g00.conj() * rj - g01.conj() * ri
        ci, cj = dn[:, :, i].clone(), dn[:, :, j].clone()
        dn[:, :, i], dn[:, :, j] = g00.conj() * ci + g01.conj() * cj, g00 * cj - g01 * ci
    for mu in range(4):
        u[mu][:2, :, s] = up[mu, :2]
        if mu == 0 and gauge == "coulomb":
            if down is not None:
                down[0][:2, :, s] = dn[0, :2]
        else:
            u[mu][:2, :, nb[mu][s]] = dn[mu, :2]


def _project(u):
    for mu in range(4):
        u[mu] = _unitary(u[mu])


def _site_quality(gauge, u, size):
    """Functional and theta of every site."""
    u = u.clone()
    u[:, 2] = _third_row(u)
    nb = _neighbours(size, -1, u.device)
    first = 1 if gauge == "coulomb" else 0
    if gauge == "mag":
        gff = sum(u[mu, j, j].abs().square() for mu in range(4) for j in range(3))
        theta = 0
        for i, j in ((0, 1), (0, 2), (1, 2)):
            X = 0
            for mu in range(4):
                a, d = u[mu], u[mu][:, :, nb[mu]]
                X = X + a[i, i] * a[j, i].conj() - a[i, j] * a[j, j].conj()
                X = X + d[i, i].conj() * d[i, j] - d[j, i].conj() * d[j, j]
            theta = theta + X.abs()
        return gff, theta
    gff = sum(u[mu, j, j].real for mu in range(first, 4) for j in range(3))
    A = sum(u[mu] - u[mu][:, :, nb[mu]] for mu in range(first, 4))
    trace = (A[0, 0] + A[1, 1] + A[2, 2]) / 3.0
    for j in range(3):
        A[j, j] -= trace
    return gff, (A - A.conj().transpose(0, 1)).abs().square().sum(dim=(0, 1))


def _quality(gauge, u, size):
    gff, theta = _site_quality(gauge, u, size)
    return float(gff.mean()) / (9.0 if gauge == "coulomb" else 12.0), float(theta.mean()) / 3.0


def exact(case, seed):
    gauge = case["gauge"]
    if case["kind"] == "fix":
        # the heat bath of a single-precision field accepts by single-precision numbers; a Coulomb
        # lattice's timeslices and long runs on large lattices would take too long here
        if (case["sa"] and case["mixed"] != "no") or gauge == "coulomb" or \
                sum(math.prod(s) for s in _lattices(case)) * (case["sweeps"] + 4 * case["sa"]) > 1e8:
            return None
        fields, gffs, thetas = [], [], []
        for k, size in enumerate(_lattices(case)):
            u = _from_layout(_fix_input(case, size, seed + 17 * k), math.prod(size))
            gff, theta = _exact_fix(case, u, size, k)
            fields.append(_to_layout(u, torch.float64))
            gffs.append(gff)
            thetas.append(theta)
        if case["host"]:
            fields = [f.cpu().numpy() for f in fields]
        return dict(fields=fields, gff=np.array(gffs), theta=np.array(thetas))
    size = _size(case["size"])
    V = math.prod(size)
    up, down = _driver_input(case, seed)
    u = _from_layout(up, V)
    if case["kind"] == "site":
        gff, theta = _site_quality(gauge, u, size)
        mean = _quality(gauge, u, size)
        return dict(gff=gff, theta=theta, mean_gff=mean[0], mean_theta=mean[1])
    if case["real"] == 32 and "sa" in case["steps"].split():
        return None
    d = _from_layout(down, V) if down is not None else None
    counter, quality = 0, (0.0, 0.0)
    for step in case["steps"].split():
        if step == "project":
            _project(u)
        elif step == "stats":
            quality = _quality(gauge, u, size)
        else:
            parameter = {"or": OMEGA, "sa": case["temperature"], "sr": SR_PROBABILITY}.get(step, 0.0)
            for parity in (0, 1):
                _pass(gauge, step, u, size, parity, parameter, _Draws(V // 2, case["real"], RNG_SEED, counter, u.device), d)
                counter += step in ("sa", "sr", "random")
    out = dict(up=_to_layout(u, up.dtype), gff=quality[0], theta=quality[1])
    return out if d is None else dict(out, down=_to_layout(d, up.dtype))


def _exact_fix(case, u, size, k):
    """The schedule of a fix case on instance k, in place; functional and theta at its last check."""
    gauge, real, counter = case["gauge"], 64 if case["mixed"] == "no" else 32, 0
    V = math.prod(size)

    def sweep(rule, parameter):
        nonlocal counter
        for parity in (0, 1):
            draws = _Draws(V // 2, real, RNG_SEED + k, counter + parity, u.device)
            _pass(gauge, rule, u, size, parity, parameter, draws)
        counter += 2 if rule in ("sa", "random") else 0

    if case["random_trafo"]:
        sweep("random", 0.0)
    t, n = np.float32(case["sa_max"]), case["sa"]
    step = (t - np.float32(0.01)) / np.float32(max(n, 1))
    for i in range(n):
        geometric = case["sa_max"] * (0.01 / case["sa_max"]) ** (i / max(n - 1, 1))
        sweep("sa", geometric if gauge == "mag" else float(t))
        t = np.float32(t - step)
        if i % case["micro_every"] == case["micro_every"] - 1:
            sweep("micro", 0.0)
    for _ in range(case["sweeps"]):
        sweep("or", OMEGA)
    quality = _quality(gauge, u, size)
    _project(u)
    return quality
