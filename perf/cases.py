"""What a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of the qcb package, on lattices that it
prepares on the device: heatbath sweeps with the plaquette, the reference's frozen-block
schedule, the Wilson flow with its (t, Q, E) records, link smearing, measurements alone,
batches of lattices, the request server and event chains.  The inputs are SU(3) fields drawn
with torch from the seed alone: each link is near the identity (mean plaquette about 0.6, the
value of a thermalised field at beta = 6), then the field is transformed by a random gauge.

A field in single precision gives its measurements as float32, a field in double precision as
float64.  The links come back as a view of the library's own device storage (its padding, which
stays zero, included).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ecmc-qncb_b200"))

import qcb  # noqa: E402

EPS = 0.02  # the driver's flow step


def listed():
    return [
        # the plain run: a small FP64 lattice, every sweep followed by its plaquette; launches and latency
        {"name": "sweep_8_fp64", "kind": "heatbath", "dims": "8x8x8x8", "prec": "fp64", "nr": 18, "beta": 6.0,
         "sweeps": 1, "hits": 1},
        # generation at the benchmark's size in its storage, the plaquette every five sweeps
        {"name": "sweeps_32_fp32r12", "kind": "heatbath", "dims": "32x32x32x32", "prec": "fp32", "nr": 12,
         "beta": 6.0, "sweeps": 5, "hits": 1},
        # the same in the default storage (double precision, all 18 reals)
        {"name": "sweeps_32_fp64", "kind": "heatbath", "dims": "32x32x32x32", "prec": "fp64", "nr": 18,
         "beta": 6.0, "sweeps": 2, "hits": 1},
        # the reference's schedule (frozen block faces after a random shift) on an uneven lattice, full FP32 links
        {"name": "frozen_ragged_fp32", "kind": "frozen", "dims": "12x18x24x30", "prec": "fp32", "nr": 18,
         "beta": 5.85, "sweeps": 2, "hits": 2, "l_core": 6},
        # link smearing: RK3 steps in place, then Q and E, in double precision
        {"name": "smear_16_fp64", "kind": "smear", "dims": "16x16x16x32", "prec": "fp64", "nr": 18, "steps": 5},
        # the topology measurement of the benchmark: a record every ten RK3 steps
        {"name": "flow_32_fp32r12", "kind": "flow", "dims": "32x32x32x32", "prec": "fp32", "nr": 12, "groups": 2,
         "rk": 10},
        # the largest lattice, Q and E before every RK3 step
        {"name": "flow_64_fp32r12", "kind": "flow", "dims": "64x64x64x64", "prec": "fp32", "nr": 12, "groups": 2,
         "rk": 1},
        # measurements of a stored configuration: plaquette, Q and E, no flow
        {"name": "measure_ragged_fp64", "kind": "measure", "dims": "20x24x28x36", "prec": "fp64", "nr": 18},
        # many small lattices at several couplings as one captured plan
        {"name": "batch_fp32r12", "kind": "batch", "prec": "fp32", "nr": 12, "n": 24, "lmin": 8, "lmax": 24,
         "sweeps": 6, "groups": 2, "rk": 5, "hits": 1, "pick": 3},
        # event chains on a small lattice: 256 chains, far fewer than the chip can hold
        {"name": "chains_16_fp64", "kind": "chains", "dims": "16x16x16x16", "prec": "fp64", "nr": 18, "beta": 6.0,
         "l_core": 4, "theta": 100.0, "calls": 2},
        # event chains on a large one: 20736 chains
        {"name": "chains_48_fp64", "kind": "chains", "dims": "48x48x48x48", "prec": "fp64", "nr": 18, "beta": 6.0,
         "l_core": 4, "theta": 100.0, "calls": 1},
        # the request server: sweeps jobs and flow jobs of mixed sizes together
        {"name": "serve_fp32r12", "kind": "serve", "prec": "fp32", "nr": 12, "n": 8, "lmin": 8, "lmax": 24,
         "units": 8, "pick": 5},
    ]


def _even(rng, lo, hi):
    return 2 * rng.randint(lo // 2, hi // 2)


def _log_even(rng, lo, hi):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, 2 * round(v / 2)))


def draw(rng):
    kind = rng.choice(["heatbath", "heatbath", "frozen", "smear", "flow", "flow", "measure", "batch", "chains", "serve"])
    prec, nr = rng.choice([("fp64", 18), ("fp32", 12), ("fp32", 12), ("fp32", 18), ("fp64", 12)])
    side = _log_even(rng, 6, 30)
    dims = "x".join(str(max(4, side + 2 * rng.randint(-2, 2))) for _ in range(4))
    beta = rng.choice([5.7, 5.85, 6.0, 6.2, 6.3])
    c = {"kind": kind, "prec": prec, "nr": nr}
    if kind == "heatbath":
        c.update(dims=dims, beta=beta, sweeps=rng.randint(1, 4), hits=rng.choice([1, 1, 2]))
    elif kind == "frozen":
        l_core = rng.choice([4, 6, 8])
        c.update(dims="x".join(str(l_core * rng.randint(1, max(1, 28 // l_core))) for _ in range(4)), beta=beta,
                 sweeps=rng.randint(1, 3), hits=rng.choice([1, 2]), l_core=l_core)
    elif kind == "smear":
        c.update(dims=dims, steps=rng.randint(1, 6))
    elif kind == "flow":
        c.update(dims=dims, groups=rng.randint(1, 3), rk=rng.randint(1, 5))
    elif kind == "measure":
        c.update(dims=dims)
    elif kind == "batch":
        c.update(prec="fp32", n=rng.randint(2, 24), lmin=4, lmax=_even(rng, 6, 20), sweeps=rng.choice([0, 2, 4]),
                 groups=rng.randint(1, 2), rk=rng.randint(1, 4), hits=1, pick=rng.randint(0, 1 << 20))
    elif kind == "chains":
        l_core = rng.choice([4, 4, 6])
        c.update(prec="fp64", nr=18, dims="x".join(str(l_core * rng.randint(1, 24 // l_core)) for _ in range(4)),
                 beta=beta, l_core=l_core, theta=rng.choice([40.0, 100.0]), calls=rng.randint(1, 2))
    else:
        c.update(prec="fp32", n=rng.randint(2, 10), lmin=4, lmax=_even(rng, 8, 20), units=rng.randint(2, 8),
                 pick=rng.randint(0, 1 << 20))
    return c


# ---- shapes ---------------------------------------------------------------------------------


def _dims(c):
    return tuple(int(v) for v in c["dims"].split("x"))


def _volume(d):
    return d[0] * d[1] * d[2] * d[3]


def _sizes(c):
    """Extents of the lattices of a batch or of the server's jobs."""
    import random

    rng = random.Random(1000003 * c["pick"] + c["n"])
    out = []
    for _ in range(c["n"]):
        side = _even(rng, c["lmin"], c["lmax"])
        out.append((side, side, side, side) if rng.random() < 0.7 else (side, side, max(4, side - 2), side + 2))
    return out


def _betas(n):
    return [(5.7, 5.85, 6.0, 6.2)[k % 4] for k in range(n)]


# ---- inputs ---------------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cross_row(r0, r1):
    """conj(r0 x r1): the third row of an SU(3) matrix."""
    return torch.linalg.cross(r0, r1, dim=-1).conj().resolve_conj()


def _su3(m):
    """SU(3) from rows 0 and 1 of m by Gram-Schmidt."""
    r0 = m[..., 0, :]
    r0 = r0 / r0.abs().square().sum(-1, keepdim=True).sqrt()
    r1 = m[..., 1, :]
    r1 = r1 - (r0.conj() * r1).sum(-1, keepdim=True) * r0
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([r0, r1, _cross_row(r0, r1)], dim=-2)


def _mm(a, b):
    return a[..., :, 0:1] * b[..., 0:1, :] + a[..., :, 1:2] * b[..., 1:2, :] + a[..., :, 2:3] * b[..., 2:3, :]


def _adj(a):
    return a.transpose(-1, -2).conj()


AXIS = (3, 2, 1, 0)  # of directions x, y, z, t in a (Lt, Lz, Ly, Lx, ...) tensor


def _at(f, *steps):
    """f(x + steps), steps = (direction, distance) pairs."""
    for d, s in steps:
        f = torch.roll(f, -s, AXIS[d])
    return f


def _directions(dims, seed):
    """U_mu(x) for mu = 0 .. 3, one after the other, each (Lt, Lz, Ly, Lx, 3, 3) complex128."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed) % (1 << 62) + 1)
    shape = tuple(reversed(dims)) + (3, 3)

    def normal():
        return torch.randn(shape + (2,), generator=gen, device=_device(), dtype=torch.float32).to(torch.float64)

    g = _su3(torch.view_as_complex(normal()))
    one = torch.eye(3, dtype=torch.complex128, device=_device())
    for mu in range(4):
        u = _su3(one + 0.22 * torch.view_as_complex(normal()))
        yield _mm(_mm(g, u), _adj(_at(g, (mu, 1))))


def _packed(u, nr):
    """(2, nr, Vh) reals of direction u in the library's order: both parities, checkerboard sites."""
    t, z, y, x = u.shape[:4]
    dev = u.device
    q = (torch.arange(t, device=dev)[:, None, None] + torch.arange(z, device=dev)[None, :, None]
         + torch.arange(y, device=dev)[None, None, :]) & 1
    pairs = u.reshape(t, z, y, x // 2, 2, 9)
    out = []
    for par in (0, 1):
        odd = ((par + q) & 1).bool()[..., None, None]
        v = torch.where(odd, pairs[..., 1, :], pairs[..., 0, :]).reshape(-1, 9)
        out.append(torch.view_as_real(v).reshape(-1, 18)[:, :nr].transpose(0, 1))
    return torch.stack(out)


def _rounded(u, prec, nr):
    """The link that the storage holds of u, in double precision."""
    if prec == "fp32":
        u = u.to(torch.complex64).to(torch.complex128)
    if nr == 12:
        u = torch.cat([u[..., :2, :], _cross_row(u[..., 0, :], u[..., 1, :])[..., None, :]], dim=-2)
    return u


class _Array:
    """A tensor over the field's storage; it keeps the field, so that the memory outlives the tensor."""

    def __init__(self, field, ptr, shape, typestr):
        self.field = field
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _storage(prec, nr):
    """Reals of one chunk of the storage."""
    return 4 if (prec == "fp32" and nr == 12) else 2


def _view(field, prec, nr):
    ptr, stride, nchunk, chunk = field.device_links()
    w = _storage(prec, nr)
    return torch.as_tensor(_Array(field, ptr, (4, 2, nchunk, stride, w), "<f8" if prec == "fp64" else "<f4"))


def _fill(view, dims, seed, nr):
    """Writes a field's links into a (4, 2, chunks, stride, w) tensor."""
    vh, w = _volume(dims) // 2, view.shape[-1]
    for mu, u in enumerate(_directions(dims, seed)):
        p = _packed(u, nr)
        view[mu, :, :, :vh, :] = p.reshape(2, nr // w, w, vh).transpose(2, 3).to(view.dtype)


_CONTEXT = []


def _context():
    """The program's one context."""
    if not _CONTEXT:
        _CONTEXT.append(qcb.Context(0))
    return _CONTEXT[0]


def _field(dims, prec, nr, seed):
    ctx = _context()
    f = qcb.GaugeField(ctx, dims, prec, nr)
    ctx.sync()
    v = _view(f, prec, nr)
    _fill(v, dims, seed, nr)
    torch.cuda.synchronize()
    return f, v


def prepare(case, seed):
    c = case
    s = {"case": c, "ctx": _context(), "out": np.float32 if c["prec"] == "fp32" else np.float64}
    if c["kind"] in ("batch", "serve"):
        s["fields"], s["links"] = [], []
        for k, d in enumerate(_sizes(c)):
            f, v = _field(d, c["prec"], c["nr"], 64 * seed + k)
            s["fields"].append(f)
            s["links"].append(v)
        s["sweep"] = 0
        s["seeds"] = [seed + 7 * k for k in range(c["n"])]
        if c["kind"] == "batch":
            s["batch"] = qcb.Batch(s["ctx"], s["fields"])
        else:
            s["server"] = qcb.Server(s["ctx"], c["prec"], c["nr"], hbm_budget=2 << 30)
        return s
    dims = _dims(c)
    s["field"], s["links"] = _field(dims, c["prec"], c["nr"], 64 * seed)
    if c["kind"] in ("heatbath", "frozen"):
        hp = qcb.io.default_params()
        hp.beta, hp.N_samples, hp.N_sweeps, hp.N_hits = c["beta"], 1, c["sweeps"], c["hits"]
        s["hp"], s["rng"] = hp, qcb.PhiloxStream(seed=seed)
    if c["kind"] == "frozen":
        s["shift"] = tuple((seed >> (3 * k)) % c["l_core"] for k in range(4))
    if c["kind"] == "chains":
        p = dict(beta=c["beta"], theta_sample=c["theta"], theta_refresh_site=0.493 * c["theta"],
                 theta_refresh_R=0.147 * c["theta"], epsilon_set=0.15, poisson=False, l_core=c["l_core"])
        s["chains"] = qcb.EventChains(s["field"], p, seed)
        s["shifts"] = [[(seed + 3 * k + d) % c["l_core"] for d in range(4)] for k in range(c["calls"])]
    return s


# ---- one pass -------------------------------------------------------------------------------


def _flow_steps(field, eps, n):
    qcb._lib.check(qcb._lib.lib().qcb_flow_steps(field.h, eps, n))


def run(state):
    s, c, out = state, state["case"], state["out"]
    kind = c["kind"]
    if kind == "heatbath":
        p = qcb.heatbathcb.samples_plaquette(s["field"], s["hp"], s["rng"])
        return {"plaquette": out(p), "links": s["links"]}
    if kind == "frozen":
        s["field"].heatbath_frozen(c["beta"], c["sweeps"], c["hits"], s["rng"].seed, s["rng"].sweep, c["l_core"],
                                   s["shift"])
        s["rng"].sweep += c["sweeps"]
        p = qcb.observables.mean_plaquette_global(s["field"])
        return {"plaquette": out(p), "links": s["links"]}
    if kind == "smear":
        _flow_steps(s["field"], EPS, c["steps"])
        q, e = qcb.observables.topo_q_e_clover_global(s["field"])
        return {"qe": np.array([q, e], out), "links": s["links"]}
    if kind == "flow":
        rec = qcb.observables.topo_charge_flowed(s["field"], qcb.GradientFlow(EPS), c["groups"], c["rk"])
        return {"records": rec.astype(out)}
    if kind == "measure":
        p = qcb.observables.mean_plaquette_global(s["field"])
        q, e = qcb.observables.topo_q_e_clover_global(s["field"])
        return {"plaquette": out(p), "qe": np.array([q, e], out)}
    if kind == "batch":
        p, rec, _ = s["batch"].run(_betas(c["n"]), s["seeds"], [s["sweep"]] * c["n"], c["sweeps"], c["hits"], EPS,
                                   c["groups"], c["rk"])
        s["sweep"] += c["sweeps"]
        return {"plaquette": p.astype(out), "records": rec.astype(out), "links": s["links"]}
    if kind == "chains":
        s["chains"].sample_n(s["shifts"])
        counts = s["chains"].counters(reset=True)
        p = qcb.observables.mean_plaquette_global(s["field"])
        return {"counts": np.array(counts, np.int64), "plaquette": out(p), "links": s["links"]}
    # serve: every other job flows a copy of its lattice, the others sweep theirs
    ids = []
    for k, f in enumerate(s["fields"]):
        if k % 2:
            ids.append(s["server"].submit_flow(f, EPS, c["units"] + k % 3))
        else:
            ids.append(s["server"].submit_sweeps(f, _betas(c["n"])[k], c["units"] + k % 3, s["seeds"][k], s["sweep"]))
    s["sweep"] += c["units"] + 2
    s["server"].drain(60.0)
    got = {r.id: r for r in s["server"].poll()}
    flows = [[got[i].t, got[i].q, got[i].e] for i in ids[1::2]]
    return {"flow": np.array(flows, out), "plaquette": np.array([got[i].plaquette for i in ids[::2]], out),
            "links": s["links"][::2]}


# ---- what a pass cannot do without ----------------------------------------------------------

PRODUCT = 198  # operations of a 3x3 complex product


def work(case):
    c = case
    real = 8 if c["prec"] == "fp64" else 4
    link, alg = real * c["nr"], real * 8

    # a heatbath sweep: each of 4V updates needs its staple, (6 x 2 products), and its link;
    # a pass over half the links of one direction reads the 8 half-fields and writes one
    def sweeps(v, n, hits):
        return n * 4 * v * 9 * link, n * 4 * v * (12 * PRODUCT + hits * 3 * 150)

    # an RK3 step: three stages, each reads and writes the links; the accumulator twice each way;
    # three products for each plaquette, an exponential and two products for each link
    def steps(v, n):
        return n * v * (24 * link + 16 * alg), n * v * 3 * (6 * 3 * PRODUCT + 4 * (2 * PRODUCT + 400))

    def plaquette(v):
        return v * 4 * link, v * 6 * 2 * PRODUCT

    # Q and E read the links once; three products for each plaquette, four leaves for each plane
    def clover(v):
        return v * 4 * link, v * 6 * 5 * PRODUCT

    parts = []
    if c["kind"] in ("batch", "serve"):
        vs = [_volume(d) for d in _sizes(c)]
        for k, v in enumerate(vs):
            if c["kind"] == "batch":
                parts += [sweeps(v, c["sweeps"], c["hits"]), plaquette(v), steps(v, c["groups"] * c["rk"])]
                parts += [clover(v)] * (c["groups"] + 1)
            elif k % 2:
                parts += [steps(v, c["units"] + k % 3), clover(v)]
            else:
                parts += [sweeps(v, c["units"] + k % 3, 1), plaquette(v)]
    else:
        v = _volume(_dims(c))
        if c["kind"] == "heatbath":
            parts += [sweeps(v, c["sweeps"], c["hits"]), plaquette(v)]
        elif c["kind"] == "frozen":  # the links on the block faces stay
            moved = v * (1.0 - 1.0 / c["l_core"]) ** 3
            parts += [sweeps(moved, c["sweeps"], c["hits"]), plaquette(v)]
        elif c["kind"] == "smear":
            parts += [steps(v, c["steps"]), clover(v)]
        elif c["kind"] == "flow":
            # the record is taken before each group; the last group's result is not measured
            parts += [steps(v, c["groups"] * c["rk"])] + [clover(v)] * c["groups"]
        elif c["kind"] == "measure":
            parts += [plaquette(v), clover(v)]
        else:
            # event chains: about 3.15 events for each unit of angle, 6.5 k operations and the
            # 19 links around the active one for each; the lattice read and written once
            events = 3.15 * c["theta"] * c["calls"] * v / c["l_core"] ** 4
            parts += [(2 * v * 4 * link + events * 19 * 144, events * 6582), plaquette(v)]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ---- 64-bit values --------------------------------------------------------------------------


def _staple(u, mu):
    a = 0
    for nu in range(4):
        if nu == mu:
            continue
        a = a + _mm(_mm(_at(u[nu], (mu, 1)), _adj(_at(u[mu], (nu, 1)))), _adj(u[nu]))
        down = _at(u[nu], (nu, -1))
        a = a + _mm(_adj(_mm(_at(u[mu], (nu, -1)), _at(u[nu], (mu, 1), (nu, -1)))), down)
    return a


def _traceless(m):
    m = 0.5 * (m - _adj(m))
    tr = (m[..., 0, 0] + m[..., 1, 1] + m[..., 2, 2]) / 3.0
    return m - tr[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)


def _exp(x):
    one = torch.eye(3, dtype=x.dtype, device=x.device)
    e = one.expand(x.shape)
    for n in range(18, 0, -1):
        e = one + _mm(x, e) / n
    return e


def _rk3(u, eps):
    def force(w):
        return [-_traceless(_mm(w[mu], _staple(w, mu))) for mu in range(4)]

    z0 = force(u)
    u = [_mm(_exp(0.25 * eps * z0[m]), u[m]) for m in range(4)]
    z1 = force(u)
    acc = [8.0 / 9.0 * z1[m] - 17.0 / 36.0 * z0[m] for m in range(4)]
    u = [_mm(_exp(eps * acc[m]), u[m]) for m in range(4)]
    z2 = force(u)
    return [_mm(_exp(0.75 * eps * z2[m] - eps * acc[m]), u[m]) for m in range(4)]


def _plane_trace(u, mu, nu):
    p = _mm(_mm(u[mu], _at(u[nu], (mu, 1))), _adj(_mm(u[nu], _at(u[mu], (nu, 1)))))
    return (p[..., 0, 0] + p[..., 1, 1] + p[..., 2, 2]).real


def _mean_plaquette(u, dims):
    s = sum(_plane_trace(u, mu, nu).sum() for mu in range(4) for nu in range(mu + 1, 4))
    return float(s) / (18.0 * _volume(dims))


def _clover(u, dims):
    """(Q, E)."""
    f = {}
    for mu in range(4):
        for nu in range(mu + 1, 4):
            c = _mm(_mm(u[mu], _at(u[nu], (mu, 1))), _adj(_mm(u[nu], _at(u[mu], (nu, 1)))))
            side = _adj(_mm(_at(u[nu], (mu, -1)), _at(u[mu], (mu, -1), (nu, 1))))
            c = c + _mm(_mm(u[nu], side), _at(u[mu], (mu, -1)))
            low = _adj(_mm(_at(u[nu], (mu, -1), (nu, -1)), _at(u[mu], (mu, -1))))
            c = c + _mm(low, _mm(_at(u[mu], (mu, -1), (nu, -1)), _at(u[nu], (nu, -1))))
            turn = _mm(_at(u[mu], (nu, -1)), _at(u[nu], (mu, 1), (nu, -1)))
            c = c + _mm(_mm(_adj(_at(u[nu], (nu, -1))), turn), _adj(u[mu]))
            f[mu, nu] = 0.125 * (c - _adj(c))

    def dot(a, b):
        return (a * b.transpose(-1, -2)).sum((-1, -2)).real

    q = dot(f[0, 1], f[2, 3]) - dot(f[0, 2], f[1, 3]) + dot(f[0, 3], f[1, 2])
    e = sum(v.abs().square().sum() for v in f.values())
    return float(q.sum()) / (4.0 * math.pi ** 2), 0.5 * float(e) / _volume(dims)


def _philox(c, k0, k1):
    """Philox4x32-10 of four int64 tensors that hold 32-bit words."""
    low = 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & low) ^ c[1] ^ k0, p1 & low, ((p0 >> 32) & low) ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    return [(w.to(torch.float64) + 0.5) * 2.0 ** -32 for w in c]


def _kennedy_pendleton(alpha, link, sweep, sub, k0, k1):
    n = alpha.numel()
    a0 = torch.zeros(n, dtype=torch.float64, device=alpha.device)
    todo = torch.arange(n, device=alpha.device)
    for attempt in range(4096):
        if todo.numel() == 0:
            break
        ids = link[todo]
        d, r1, r2, r3 = _philox([ids, torch.full_like(ids, sweep), torch.full_like(ids, sub),
                                 torch.full_like(ids, attempt)], k0, k1)
        lam = -0.5 / alpha[todo] * (torch.log(r1) + torch.cos(2.0 * math.pi * r2) ** 2 * torch.log(r3))
        ok = d * d <= 1.0 - lam
        a0[todo[ok]] = 1.0 - 2.0 * lam[ok]
        todo = todo[~ok]
    w = _philox([link, torch.full_like(link, sweep), torch.full_like(link, sub), torch.full_like(link, 0xFFFFFFFF)],
                k0, k1)
    ct = 2.0 * w[1] - 1.0
    st, r = torch.sqrt((1.0 - ct * ct).clamp(min=0)), torch.sqrt((1.0 - a0 * a0).clamp(min=0))
    return a0, r * st * torch.cos(2 * math.pi * w[0]), r * st * torch.sin(2 * math.pi * w[0]), r * ct


def _heatbath(u, dims, beta, n_sweeps, hits, seed, frozen=None):
    """n_sweeps checkerboard sweeps of u; frozen = (l_core, shift) leaves the block faces."""
    dev = u[0].device
    grid = torch.meshgrid(*[torch.arange(n, device=dev) for n in reversed(dims)], indexing="ij")
    x = list(reversed(grid))
    site = x[0] + dims[0] * (x[1] + dims[1] * (x[2] + dims[2] * x[3]))
    parity = (x[0] + x[1] + x[2] + x[3]) & 1
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for sweep in range(n_sweeps):
        for mu in range(4):
            for par in (0, 1):
                on = parity == par
                if frozen:
                    for d in range(4):
                        if d != mu:
                            on = on & ((x[d] + frozen[1][d]) % frozen[0] != 0)
                a, w = _staple(u, mu)[on], u[mu][on]
                link = site[on] + mu * _volume(dims)
                for h in range(hits):
                    for sub, (i, j) in enumerate(((0, 1), (1, 2), (0, 2))):
                        m = _mm(w, a)
                        v = [0.5 * (m[:, i, i] + m[:, j, j]).real, 0.5 * (m[:, i, j] + m[:, j, i]).imag,
                             0.5 * (m[:, i, j] - m[:, j, i]).real, 0.5 * (m[:, i, i] - m[:, j, j]).imag]
                        k = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2 + v[3] ** 2)
                        v = [t / k for t in v]
                        p = _kennedy_pendleton(2.0 * beta * k / 3.0, link, sweep, 4 * h + sub, k0, k1)
                        q = [p[0] * v[0] + p[1] * v[1] + p[2] * v[2] + p[3] * v[3],
                             -p[0] * v[1] + p[1] * v[0] - p[2] * v[3] + p[3] * v[2],
                             -p[0] * v[2] + p[1] * v[3] + p[2] * v[0] - p[3] * v[1],
                             -p[0] * v[3] - p[1] * v[2] + p[2] * v[1] + p[3] * v[0]]
                        top = torch.complex(q[0], q[3])[:, None], torch.complex(q[2], q[1])[:, None]
                        bottom = torch.complex(-q[2], q[1])[:, None], torch.complex(q[0], -q[3])[:, None]
                        wi, wj = w[:, i].clone(), w[:, j].clone()
                        w = w.clone()
                        w[:, i], w[:, j] = top[0] * wi + top[1] * wj, bottom[0] * wi + bottom[1] * wj
                u = list(u)
                u[mu] = u[mu].clone()
                u[mu][on] = w
    return u


def _layout(u, dims, prec, nr):
    """u as the library stores it, in 64 bits."""
    vh, w = _volume(dims) // 2, _storage(prec, nr)
    out = torch.zeros((4, 2, nr // w, (vh + 63) // 64 * 64, w), dtype=torch.float64, device=u[0].device)
    for mu in range(4):
        out[mu, :, :, :vh, :] = _packed(u[mu], nr).reshape(2, nr // w, w, vh).transpose(2, 3)
    return out


def _records(u, dims, groups, rk, last):
    rec = []
    for g in range(groups + (1 if last else 0)):
        rec.append((g * rk * EPS,) + _clover(u, dims))
        if g < groups:
            for _ in range(rk):
                u = _rk3(u, EPS)
    return rec


def exact(case, seed):
    """run()'s outputs for these inputs in 64 bits.  None: lattices that would take too long, event
    chains (a serial chain of thousands of events for each block), and what follows from the
    accept/reject decisions of single-precision draws, which have no 64-bit value."""
    c = case
    kind, prec, nr = c["kind"], c["prec"], c["nr"]
    if kind == "chains":
        return None

    def start(dims, s):
        return [_rounded(u, prec, nr) for u in _directions(dims, s)]

    if kind == "batch":
        sizes = _sizes(c)
        if c["sweeps"] or sum(map(_volume, sizes)) > 1 << 20:
            return None
        fields = [start(d, 64 * seed + k) for k, d in enumerate(sizes)]
        return {"plaquette": np.array([_mean_plaquette(u, d) for u, d in zip(fields, sizes)]),
                "records": np.array([_records(u, d, c["groups"], c["rk"], True) for u, d in zip(fields, sizes)]),
                "links": [_layout(u, d, prec, nr) for u, d in zip(fields, sizes)]}
    if kind == "serve":
        rec = []
        for k, d in enumerate(_sizes(c)):
            if k % 2:
                u = start(d, 64 * seed + k)
                n = c["units"] + k % 3
                for _ in range(n):
                    u = _rk3(u, EPS)
                rec.append((n * EPS,) + _clover(u, d))
        return {"flow": np.array(rec), "plaquette": None, "links": None}
    dims = _dims(c)
    v = _volume(dims)
    if v > 1 << 21:
        return None
    if kind in ("heatbath", "frozen"):
        if prec == "fp32":
            return None
        frozen = None
        if kind == "frozen":
            frozen = (c["l_core"], tuple((seed >> (3 * k)) % c["l_core"] for k in range(4)))
        u = _heatbath(start(dims, 64 * seed), dims, c["beta"], c["sweeps"], c["hits"], seed, frozen)
        return {"plaquette": np.float64(_mean_plaquette(u, dims)), "links": _layout(u, dims, prec, nr)}
    u = start(dims, 64 * seed)
    if kind == "smear":
        for _ in range(c["steps"]):
            u = _rk3(u, EPS)
        return {"qe": np.array(_clover(u, dims)), "links": _layout(u, dims, prec, nr)}
    if kind == "flow":
        return {"records": np.array(_records(u, dims, c["groups"], c["rk"], False)).reshape(-1)}
    return {"plaquette": np.float64(_mean_plaquette(u, dims)), "qe": np.array(_clover(u, dims))}
