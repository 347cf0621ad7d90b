"""The work that a user of this library has it do, as cases that can be timed.

Each case is one call (or the two or three calls of one step) through the
public Python entry points, on inputs of the kind the unbinding meets in a
simulation: NFW subhaloes with Jeans velocities and unbound contaminants in a
periodic box, sizes from the steep power law dN/dlnN ~ N^-0.9, all generated on
the GPU from a seed.  The kinds:

  unbind    Unbinder.unbind_batch_device: one subhalo, or a batch of them, with
            the arrays on the device; FP32 or FP64 walk; the exact tree or the
            reference's sampled potentials (max_sample); periodic box or not
  energies  Unbinder.binding_energies: one energy pass over one subhalo held in
            host arrays (the call a C++ host program makes)
  gradient  adjoint.BindingEnergy: E_tot of a batch's particle sets, forward and
            backward
  step      TrackingStep.load_snapshot + run: the particle-ID table of a new
            snapshot, the members re-resolved and gathered, the batch unbound, the
            profile and shape of every subhalo
  table     a particle-ID table alone: fill and look up (mapped or flat)
"""
import collections
import ctypes
import math

import numpy as np
import torch

from hbtplus_gb300 import _lib
from hbtplus_gb300 import synthetic
from hbtplus_gb300.adjoint import BindingEnergy
from hbtplus_gb300.index import FlatIndexTable, MappedIndexTable
from hbtplus_gb300.step import TrackingStep
from hbtplus_gb300.unbind import Unbinder

G = synthetic.G_MPC_KMS
MASS = 1e-4
SLOPE = -0.9
PARTICLE_BYTES = 40   # id 8, pos 12, vel 12, mass 4, type 4
RESULT_BYTES = ctypes.sizeof(_lib.hbtu_result)
PROPS_BYTES = ctypes.sizeof(_lib.hbtu_props)
STATE_BYTES = ctypes.sizeof(_lib.hbtu_state)
FLOPS = 14            # one potential contribution: 3 sub, 5 r^2, 4 rsqrt, 2 update


def _unbind(name=None, nsub=1, nmin=20, nmax=20, contaminants=0.2, theta=0.45, max_sample=0,
            fp64=False, periodic=True, clumps=0):
    c = dict(kind="unbind", nsub=nsub, nmin=nmin, nmax=nmax, contaminants=contaminants,
             theta=theta, max_sample=max_sample, fp64=fp64, periodic=periodic, clumps=clumps)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's own calling pattern: Subhalo_t::Unbind for one subhalo at
        # a time, most of them of a few hundred particles (latency)
        _unbind("unbind one of 317", nsub=1, nmin=317, nmax=317),
        # an isolated subhalo of 1e5 particles and 10% contaminants
        _unbind("unbind one of 1.1e5", nsub=1, nmin=100000, nmax=100000, contaminants=0.1),
        # a large host with 300 embedded clumps, 2.7e7 particles: tree throughput
        _unbind("unbind a host of 2.7e7", nsub=1, nmin=20000000, nmax=20000000,
                contaminants=0.05, clumps=300),
        # all subhaloes of one nesting level in one call: the size law over four decades
        _unbind("unbind 2000", nsub=2000, nmin=20, nmax=200000),
        # the same with the reference's default of sampled potentials
        _unbind("unbind 2000 sampled", nsub=2000, nmin=20, nmax=200000, max_sample=1000),
        # the bulk of a halo catalogue: many subhaloes near the resolution limit
        _unbind("unbind 20000 small", nsub=20000, nmin=20, nmax=500),
        # the reference's arithmetic bit for bit, for comparison with its outputs
        _unbind("unbind 400 fp64", nsub=400, nmin=20, nmax=20000, fp64=True),
        # one pass of energies and potentials for a host program's arrays
        dict(name="energies of 5e4, host arrays", kind="energies", n=50000, theta=0.45,
             periodic=True),
        # tidal diagnostics over the batch's particle sets, forward and backward
        dict(name="gradient 2000", kind="gradient", nsub=2000, nmin=20, nmax=200000, theta=0.45),
        # the same for one subhalo of 1e6 particles
        dict(name="gradient one of 1e6", kind="gradient", nsub=1, nmin=1000000, nmax=1000000,
             theta=0.45),
        # a tracking step between two snapshots: 20,000 subhaloes, 3e7 particles
        dict(name="tracking step", kind="step", nsub=20000, nmin=20, nmax=200000, ntot=30000000,
             flat=False),
        # IDs of a zoom snapshot through the dense table
        dict(name="flat table of 3e6", kind="table", flat=True, n=3000001, m=1000003),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "batch", "batch", "sampled", "fp64", "energies", "gradient", "step",
                       "table"])
    if kind == "one":
        n = _log_uniform(rng, 20, 2000000)
        return _unbind(nsub=1, nmin=n, nmax=n, contaminants=round(rng.uniform(0.05, 0.3), 3),
                       theta=rng.choice([0.3, 0.45, 0.45, 0.7]), periodic=rng.random() < 0.8)
    if kind in ("batch", "sampled"):
        return _unbind(nsub=_log_uniform(rng, 8, 20000), nmin=20,
                       nmax=_log_uniform(rng, 200, 200000),
                       contaminants=round(rng.uniform(0.05, 0.3), 3),
                       theta=rng.choice([0.3, 0.45, 0.45, 0.7]),
                       max_sample=rng.choice([300, 1000, 1000]) if kind == "sampled" else 0,
                       periodic=rng.random() < 0.8)
    if kind == "fp64":
        return _unbind(nsub=_log_uniform(rng, 1, 1000), nmin=20, nmax=_log_uniform(rng, 200, 20000),
                       contaminants=round(rng.uniform(0.05, 0.3), 3), fp64=True,
                       periodic=rng.random() < 0.8)
    if kind == "energies":
        return dict(kind="energies", n=_log_uniform(rng, 30, 200000),
                    theta=rng.choice([0.3, 0.45, 0.7]), periodic=rng.random() < 0.8)
    if kind == "gradient":
        if rng.random() < 0.5:
            n = _log_uniform(rng, 1000, 2000000)
            return dict(kind="gradient", nsub=1, nmin=n, nmax=n, theta=0.45)
        return dict(kind="gradient", nsub=_log_uniform(rng, 4, 4000), nmin=20,
                    nmax=_log_uniform(rng, 200, 200000), theta=0.45)
    if kind == "step":
        nsub = _log_uniform(rng, 300, 20000)
        return dict(kind="step", nsub=nsub, nmin=20, nmax=_log_uniform(rng, 2000, 200000),
                    ntot=nsub * rng.randrange(600, 1500), flat=rng.random() < 0.3)
    n = _log_uniform(rng, 1000, 20000000)
    return dict(kind="table", flat=rng.random() < 0.5, n=n, m=max(1, n // rng.randrange(1, 9)))


# ---------------------------------------------------------------- sizes (a case's own, for every seed)
def _sizes(nsub, nmin, nmax):
    """nsub sizes at the mid-quantiles of dN/dlnN ~ N^SLOPE on [nmin, nmax]."""
    u = (np.arange(nsub) + 0.5) / nsub
    a, b = SLOPE * math.log(nmin), SLOPE * math.log(nmax)
    n = np.exp(np.log(np.exp(a) + u * (np.exp(b) - np.exp(a))) / SLOPE)
    return np.maximum(np.floor(n + 1e-6).astype(np.int64), int(nmin))


def _clump_sizes(k):
    return np.exp(np.linspace(math.log(1e3), math.log(1e5), k)).astype(np.int64)


def _contaminants(n, frac):
    return np.rint(frac * np.asarray(n)).astype(np.int64)


def _counts(case):
    n = _sizes(case["nsub"], case["nmin"], case["nmax"])
    if case.get("clumps"):
        n = n + _clump_sizes(case["clumps"]).sum()
    return n + _contaminants(n, case.get("contaminants", 0.2))


def _interactions(n):
    """Contributions that one target's walk sums in an NFW subhalo of n particles at an
    opening angle of 0.45 (counted on the library's walks: about 6 log2(n)^2)."""
    n = np.asarray(n, np.float64)
    return np.minimum(n, 6.0 * np.log2(np.maximum(n, 2.0)) ** 2)


def work(case):
    kind = case["kind"]
    if kind == "table":
        return {"bytes": 16.0 * case["n"] + 16.0 * case["m"], "flops": 0.0}
    if kind == "energies":
        n = case["n"]
        return {"bytes": float(n) * (36 + 12), "flops": FLOPS * float(n * _interactions(n))}
    if kind == "gradient":
        n = _sizes(case["nsub"], case["nmin"], case["nmax"])
        return {"bytes": float(n.sum()) * (28 + 28) + 8.0 * len(n),
                "flops": 3 * FLOPS * float((n * _interactions(n)).sum())}
    n = _counts(case)
    if kind == "step":
        n = np.maximum(1, np.rint(0.9 * n))
    trees = np.minimum(n, case["max_sample"]) if case.get("max_sample") else n
    w = {"bytes": float(n.sum()) * (PARTICLE_BYTES + 12) + len(n) * (STATE_BYTES + RESULT_BYTES),
         "flops": FLOPS * float((n * _interactions(trees)).sum())}
    if kind == "step":
        w["bytes"] += case["ntot"] * float(PARTICLE_BYTES) + n.sum() * 16.0 + len(n) * PROPS_BYTES
    return w


# ---------------------------------------------------------------- inputs
_tables = {}


def _nfw(c, ngrid=2048):
    """Radius grid x = r/rs, enclosed-mass fraction, isotropic Jeans sigma^2 and
    potential (units of G M / rs) of a truncated NFW halo of concentration c."""
    if c not in _tables:
        def m(x):
            return np.log1p(x) - x / (1 + x)
        x = np.geomspace(1e-6 * c, c, ngrid)
        f = m(x) / (x ** 3 * (1 + x) ** 2)
        seg = 0.5 * (f[1:] + f[:-1]) * np.diff(x)
        tail = np.concatenate([np.cumsum(seg[::-1])[::-1], [0.0]])
        _tables[c] = (x, m(x) / m(c), x * (1 + x) ** 2 * tail / m(c),
                      -(m(x) / x + 1 / (1 + x) - 1 / (1 + c)) / m(c))
    return [torch.as_tensor(t, device="cuda") for t in _tables[c]]


def _interp(x, xp, fp):
    i = torch.searchsorted(xp, x).clamp(1, len(xp) - 1)
    t = ((x - xp[i - 1]) / (xp[i] - xp[i - 1])).clamp(0, 1)
    return fp[i - 1] + t * (fp[i] - fp[i - 1])


def _directions(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


CONCENTRATIONS = np.linspace(5.0, 20.0, 16)


def _halo(g, n, r200, conc):
    """Positions and velocities of one class of NFW subhaloes: particles of subhaloes of one
    concentration; n: particles in its subhalo and r200, both per particle."""
    x, menc, sig2, _ = _nfw(conc)
    u = torch.rand(len(n), generator=g, device="cuda", dtype=torch.float64)
    xr = _interp(u, menc, x)
    rs = r200 / conc
    sig = (_interp(xr, x, sig2).clamp_min(0) * G * MASS * n / rs).sqrt()
    return (_directions(g, len(n)) * (xr * rs)[:, None],
            torch.randn(len(n), 3, generator=g, device="cuda", dtype=torch.float64) * sig[:, None])


def _contaminant(g, n, r200, conc):
    """Unbound particles: uniform in a sphere of 2 r200 at three times the escape speed."""
    x, _, _, phi = _nfw(conc)
    rs = r200 / conc
    r = 2 * r200 * torch.rand(len(n), generator=g, device="cuda", dtype=torch.float64) ** (1 / 3)
    xc = r / rs
    p = torch.where(xc <= conc, _interp(xc, x, phi) * G * MASS * n / rs, -G * MASS * n / r)
    return (_directions(g, len(n)) * r[:, None],
            _directions(g, len(n)) * (3 * (2 * p.abs()).sqrt())[:, None])


def _clump_set(g, case, r200, conc):
    """Plummer clumps on the host's profile: positions and velocities of all of them."""
    sizes = torch.as_tensor(_clump_sizes(case["clumps"]), device="cuda")
    host = torch.full((len(sizes),), float(case["nmin"]), device="cuda", dtype=torch.float64)
    cpos, cvel = _halo(g, host, torch.full_like(host, r200), conc)
    k = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
    a = 0.01
    u = torch.rand(len(k), generator=g, device="cuda", dtype=torch.float64) * (100 / 101.) ** 1.5
    r = a / (u.clamp_min(1e-12) ** (-2 / 3) - 1).sqrt()
    sig = (G * MASS * sizes[k] / (6 * (r * r + a * a).sqrt())).sqrt()
    return (cpos[k] + _directions(g, len(k)) * r[:, None],
            cvel[k] + torch.randn(len(k), 3, generator=g, device="cuda",
                                  dtype=torch.float64) * sig[:, None])


def _population(case, seed, box, contaminants):
    """A batch of subhaloes on the device: arrays per particle (subhalo by subhalo, the particle
    nearest the centre first), offsets, and the frames the unbinding starts from."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    size = _sizes(case["nsub"], case["nmin"], case["nmax"])[rng.permutation(case["nsub"])]
    clumps = bool(case.get("clumps"))
    conc = (np.full(1, CONCENTRATIONS[0]) if clumps else
            CONCENTRATIONS[rng.integers(len(CONCENTRATIONS), size=len(size))])
    r200 = 0.2 * (size / 1e5) ** (1 / 3)
    if clumps:
        r200 = np.full(1, 1.0)  # the host's, as in the repository's 2e7-particle workload
    center = rng.uniform(0, box, size=(len(size), 3))
    face = rng.uniform(size=len(size)) < 0.05  # some straddle a face of the box
    center[face, 0] = (rng.uniform(-1, 1, size=face.sum()) * r200[face]) % box
    bulk = rng.normal(scale=300.0, size=(len(size), 3))
    if not case.get("periodic", True):
        center = box / 4 + center / 2
    extra = _clump_sizes(case["clumps"]).sum() if clumps else 0
    cont = _contaminants(size + extra, contaminants)
    pos, vel, sub = [], [], []
    for c in np.unique(conc):
        for counts, make in ((size, _halo), (cont, _contaminant)):
            s = np.flatnonzero(conc == c)
            s = s[counts[s] > 0]
            k = torch.repeat_interleave(torch.as_tensor(s, device="cuda"),
                                        torch.as_tensor(counts[s], device="cuda"))
            n = torch.as_tensor((size + extra).astype(np.float64), device="cuda")[k]
            p, v = make(g, n, torch.as_tensor(r200, device="cuda")[k], float(c))
            pos.append(p)
            vel.append(v)
            sub.append(k)
    if clumps:
        p, v = _clump_set(g, case, float(r200[0]), float(conc[0]))
        pos.append(p)
        vel.append(v)
        sub.append(torch.zeros(len(p), dtype=torch.int64, device="cuda"))
    pos, vel, sub = torch.cat(pos), torch.cat(vel), torch.cat(sub)
    mix = torch.randperm(len(sub), generator=g, device="cuda")
    mix = mix[torch.sort(sub[mix], stable=True).indices]
    pos, vel, sub = pos[mix], vel[mix], sub[mix]
    total = size + extra + cont
    off = np.concatenate([[0], np.cumsum(total)]).astype(np.int64)
    # the particle nearest the centre goes first: the last snapshot's most-bound one
    r2 = (pos * pos).sum(1)
    least = torch.full((len(size),), math.inf, device="cuda", dtype=torch.float64)
    least.scatter_reduce_(0, sub, r2, "amin")
    at = torch.full((len(size),), 1 << 62, device="cuda", dtype=torch.int64)
    index = torch.arange(len(sub), device="cuda")
    at.scatter_reduce_(0, sub, torch.where(r2 == least[sub], index, 1 << 62), "amin")
    first = torch.as_tensor(off[:-1], device="cuda")
    for a in (pos, vel):
        a[first], a[at] = a[at].clone(), a[first].clone()
    cen = torch.as_tensor(center, device="cuda")
    pos = torch.remainder(pos + cen[sub], box).float()
    pos[pos >= box] = 0.0
    vel = (vel + torch.as_tensor(bulk, device="cuda")[sub]).float()
    dev = dict(id=torch.randperm(len(sub), generator=g, device="cuda"), pos=pos.contiguous(),
               vel=vel.contiguous(), mass=torch.full((len(sub),), MASS, device="cuda"),
               type=torch.ones(len(sub), dtype=torch.int32, device="cuda"))
    frames = dict(ref_pos=center.astype(np.float32), ref_vel=bulk.astype(np.float32),
                  mostbound_pos=dev["pos"][first].cpu().numpy(),
                  mostbound_vel=dev["vel"][first].cpu().numpy(),
                  mostbound_id=dev["id"][first].cpu().numpy())
    return g, dev, off, sub, frames


def _states(frames):
    n = len(frames["mostbound_id"])
    sts = (_lib.hbtu_state * max(n, 1))()
    a = np.frombuffer(sts, dtype=np.dtype(_lib.hbtu_state))
    for k in ("ref_pos", "ref_vel", "mostbound_pos", "mostbound_vel", "mostbound_id"):
        a[k][:n] = frames[k]
    return sts


_handles = collections.OrderedDict()


def _program(case, box):
    """The handle a program keeps for all its calls with the same parameters."""
    par = synthetic.default_params(open_angle=case.get("theta", 0.45), box_size=box,
                                   max_sample_size=case.get("max_sample", 0),
                                   periodic=int(case.get("periodic", True)))
    key = (tuple(sorted(par.items())), bool(case.get("fp64")), case.get("kind"), case.get("flat"))
    if key not in _handles:
        _handles.clear()  # one program at a time (a state holds on to its own)
        ub = Unbinder(par, precision=int(bool(case.get("fp64"))))
        ub.set_stream(torch.cuda.current_stream().cuda_stream)
        more = None
        if case["kind"] == "step":
            more = TrackingStep(ub, flat=case["flat"])
        elif case["kind"] == "table":
            more = (FlatIndexTable if case["flat"] else MappedIndexTable)(ub)
        _handles[key] = (ub, more)
    return _handles[key]


def _outputs(n, nsub):
    return dict(order=torch.empty(n, dtype=torch.int64, device="cuda"),
                energy=torch.empty(n, dtype=torch.float32, device="cuda"),
                res=torch.empty(nsub * RESULT_BYTES, dtype=torch.uint8, device="cuda"))


def prepare(case, seed):
    kind = case["kind"]
    box = 200.0 if kind == "step" else 100.0
    ub, more = _program(case, box)
    st = dict(case=case, ub=ub)
    if kind == "unbind":
        g, dev, off, sub, frames = _population(case, seed, box, case["contaminants"])
        st |= dict(dev=dev, off=off, frames=frames, states=_states(frames),
                   out=_outputs(int(off[-1]), len(off) - 1))
    elif kind == "energies":
        one = dict(case, nsub=1, nmin=case["n"], nmax=case["n"])
        g, dev, off, sub, frames = _population(one, seed, box, 0.0)
        st |= {k: dev[k].cpu().numpy() for k in ("id", "pos", "vel", "mass")}
        st |= dict(ref_pos=frames["ref_pos"][0], ref_vel=frames["ref_vel"][0])
    elif kind == "gradient":
        g, dev, off, sub, frames = _population(case, seed, box, 0.0)
        st |= dict(off=off, ref_pos=frames["ref_pos"], ref_vel=frames["ref_vel"])
        st |= {k: dev[k].requires_grad_() for k in ("pos", "vel", "mass")}
    elif kind == "step":
        g, dev, off, sub, frames = _population(case, seed, box, 0.2)
        nin, nbg = int(off[-1]), max(0, case["ntot"] - int(off[-1]))
        more_pos = torch.rand(nbg, 3, generator=g, device="cuda") * box
        more_vel = 300 * torch.randn(nbg, 3, generator=g, device="cuda")
        ids = torch.randperm(nin + nbg, generator=g, device="cuda") * 3 + 1
        # the last snapshot's membership: each subhalo without its outer tenth
        d = dev["pos"].double() - torch.as_tensor(frames["ref_pos"], device="cuda").double()[sub]
        r2 = (d - box * torch.round(d / box)).square().sum(1)
        first = torch.as_tensor(off[:-1], device="cuda")
        r2[first] = -1.0
        by_r = torch.sort(r2, stable=True).indices
        by_r = by_r[torch.sort(sub[by_r], stable=True).indices]
        keep_n = np.maximum(1, np.rint(0.9 * np.diff(off)).astype(np.int64))
        rank = torch.arange(nin, device="cuda") - first[sub]
        kept = by_r[rank < torch.as_tensor(keep_n, device="cuda")[sub]]
        kept = torch.sort(kept).values  # in list order; the first particle stays first
        pos = torch.cat([dev["pos"], more_pos])
        vel = torch.cat([dev["vel"], more_vel])
        pos = torch.remainder(pos + vel * 1e-4, box)
        pos[pos >= box] = 0.0
        mix = torch.randperm(nin + nbg, generator=g, device="cuda")
        frames["mostbound_id"] = ids[first].cpu().numpy()
        st |= dict(step=more, snap=[ids[mix], pos[mix].contiguous(), vel[mix].contiguous(),
                                    torch.full((nin + nbg,), MASS, device="cuda"),
                                    torch.ones(nin + nbg, dtype=torch.int32, device="cuda")],
                   member=ids[kept].contiguous(), states=_states(frames),
                   off=np.concatenate([[0], np.cumsum(keep_n)]).astype(np.int64))
    else:
        g = torch.Generator("cuda").manual_seed(int(seed))
        span = 3 * case["n"] // 2
        keys = torch.randperm(span, generator=g, device="cuda")[:case["n"]] * (1 if case["flat"] else 5) + 11
        pick = torch.randint(case["n"], (case["m"],), generator=g, device="cuda")
        query = keys[pick]
        query[::10] += 1  # some are not in the table (or are another key's)
        st |= dict(table=more, keys=keys, values=torch.arange(case["n"], device="cuda"),
                   query=query, found=torch.empty(case["m"], dtype=torch.int64, device="cuda"))
    return st


def _result_views(res, nsub):
    """hbtu_result records as the fields a program reads: views of the buffer."""
    f, w, q = (res.view(t).view(nsub, -1) for t in (torch.float32, torch.int32, torch.int64))
    return dict(nbound=q[:, 0], mbound=f[:, 2], ref_pos=f[:, 3:6], ref_vel=f[:, 6:9],
                mostbound=f[:, 9:15], specific=f[:, 15:20], nbound_type=q[:, 10:16],
                mbound_type=f[:, 32:38], flags=w[:, 38:42], counts=q[:, 21:23], status=w[:, 46])


def run(st):
    kind = st["case"]["kind"]
    if kind == "unbind":
        out = st["out"]
        st["ub"].unbind_batch_device(st["dev"], st["off"], st["states"], out)
        return dict(order=out["order"], energy=out["energy"],
                    res=_result_views(out["res"], len(st["off"]) - 1))
    if kind == "energies":
        energy, pot = st["ub"].binding_energies(st["pos"], st["vel"], st["mass"], st["ref_pos"],
                                                st["ref_vel"], ids=st["id"])
        return dict(energy=energy, potential=pot)
    if kind == "gradient":
        E = BindingEnergy.apply(st["pos"], st["vel"], st["mass"], st["ub"], st["off"],
                                st["ref_pos"], st["ref_vel"])
        gp, gv, gm = torch.autograd.grad(E.sum(), (st["pos"], st["vel"], st["mass"]))
        return dict(E=E, grad_pos=gp, grad_vel=gv, grad_mass=gm)
    if kind == "step":
        st["step"].load_snapshot(*st["snap"])
        out, index = st["step"].run(st["off"], st["member"], st["states"],
                                    properties=dict(snapshot_index=7))
        props = np.frombuffer(out["props"], dtype=np.dtype(_lib.hbtu_props))
        return dict(index=index, order=out["order"], energy=out["energy"],
                    res=_result_views(out["res"], len(st["off"]) - 1),
                    props={k: props[k] for k in props.dtype.names})
    st["table"].fill_device(st["keys"], st["values"], null_index=-1)
    st["table"].lookup_device(st["query"], st["found"])
    return st["found"]


# ---------------------------------------------------------------- the same in 64 bits, by direct sums
H_SOFT = 2.8 * float(np.float32(0.002))
MOST_PAIRS = 4e10  # a few seconds of pairwise sums in 64 bits


def _wrap(d, box, periodic):
    return d - box * torch.round(d / box) if periodic else d


def _pairwise(x, m, box, periodic, targets=None, grad=False):
    """Softened potentials (and their gradients) of particles x[targets] from all others."""
    n = len(x)
    t = torch.arange(n, device="cuda") if targets is None else targets
    phi = torch.empty(len(t), dtype=torch.float64, device="cuda")
    gr = torch.empty(len(t), 3, dtype=torch.float64, device="cuda") if grad else None
    for i in range(0, len(t), max(1, 100_000_000 // max(n, 1))):
        k = t[i:i + max(1, 100_000_000 // max(n, 1))]
        d = [_wrap(x[None, :, j] - x[k, None, j], box, periodic) for j in range(3)]
        r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt_()
        r[torch.arange(len(k), device="cuda"), k] = math.inf  # not from itself
        f = -1 / r
        near = torch.nonzero(r < H_SOFT, as_tuple=True)
        u = r[near] / H_SOFT
        us = u.clamp_min(1e-30)
        f[near] = torch.where(u < 0.5, -2.8 + u * u * (16 / 3 + u * u * (6.4 * u - 9.6)),
                              -3.2 + 1 / (15 * us) + u * u * (
                                  32 / 3 + u * (-16 + u * (9.6 - 32 / 15 * u)))) / H_SOFT
        phi[i:i + len(k)] = f @ m
        if grad:
            w = 1 / (r * r * r)
            w[near] = torch.where(u < 0.5, 32 / 3 + u * u * (32 * u - 38.4),
                                  -1 / (15 * us ** 3) + 64 / 3 + u * (
                                      -48 + u * (38.4 - 32 / 3 * u))) / H_SOFT ** 3
            for j in range(3):
                gr[i:i + len(k), j] = -((w * d[j]) @ m)
    return (G32 * phi, G32 * gr) if grad else G32 * phi


G32 = float(np.float32(G))
HUBBLE = 100.0


def _unbind_exact(x, v, m, ref_pos, ref_vel, box, periodic):
    """The unbinding loop of one subhalo in 64 bits: a full pass by direct sums each time.
    Returns the energies by list position and (mbound, ref_pos, ref_vel, specific)."""
    n = len(x)
    energy = torch.full((n,), math.nan, dtype=torch.float64, device="cuda")
    cur, xr, vr = torch.arange(n, device="cuda"), ref_pos, ref_vel
    while True:
        dv = v[cur] - vr + HUBBLE * _wrap(x[cur] - xr, box, periodic)
        E = 0.5 * (dv * dv).sum(1) + _pairwise(x[cur], m[cur], box, periodic)
        bound = E < 0
        nb = int(bound.sum())
        if nb < 20:  # disrupted: the last most-bound particle alone is left
            neg = torch.nonzero(bound)
            energy.fill_(math.nan)
            energy[0] = E[neg[-1, 0]] if nb else E[0]
            return energy, None
        energy[nb:len(cur)] = torch.sort(E[~bound]).values
        last, cur, Eb = len(cur), cur[bound], E[bound]
        M = m[cur].sum()
        vr = (m[cur, None] * v[cur]).sum(0) / M
        o = x[cur[0]]
        xr = o + (m[cur, None] * _wrap(x[cur] - o, box, periodic)).sum(0) / M
        if nb >= last * 0.995:
            break
    energy[:nb] = torch.sort(Eb).values
    dx = _wrap(x[cur] - xr, box, periodic)
    dv = v[cur] - vr + HUBBLE * dx
    K = 0.5 * (m[cur] * (dv * dv).sum(1)).sum() / M
    L = (m[cur, None] * torch.linalg.cross(dx, dv)).sum(0) / M
    return energy, (M, xr, vr, torch.cat([((m[cur] * Eb).sum() / M - K)[None], K[None], L]))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "table") or case.get("max_sample"):
        return None
    box, periodic = 100.0, bool(case.get("periodic", True))
    if kind == "energies":
        if float(case["n"]) ** 2 > MOST_PAIRS:
            return None
        one = dict(case, nsub=1, nmin=case["n"], nmax=case["n"])
        g, dev, off, sub, frames = _population(one, seed, box, 0.0)
        x, v, m = (dev[k].double() for k in ("pos", "vel", "mass"))
        f = {k: torch.as_tensor(frames[k][0], device="cuda").double() for k in ("ref_pos", "ref_vel")}
        pot = _pairwise(x, m, box, periodic)
        dv = v - f["ref_vel"] + HUBBLE * _wrap(x - f["ref_pos"], box, periodic)
        return dict(energy=0.5 * (dv * dv).sum(1) + pot, potential=pot)
    n = (_sizes(case["nsub"], case["nmin"], case["nmax"]) if kind == "gradient" else _counts(case))
    if (n.astype(np.float64) ** 2).sum() > MOST_PAIRS or len(n) > 1000:
        return None
    if kind == "gradient":
        g, dev, off, sub, frames = _population(case, seed, box, 0.0)
    else:
        g, dev, off, sub, frames = _population(case, seed, box, case["contaminants"])
    x, v, m = (dev[k].double() for k in ("pos", "vel", "mass"))
    rp, rv = (torch.as_tensor(frames[k], device="cuda").double() for k in ("ref_pos", "ref_vel"))
    if kind == "gradient":
        got = [[], [], [], []]
        for s in range(len(n)):
            a = slice(int(off[s]), int(off[s + 1]))
            dv = v[a] - rv[s] + HUBBLE * _wrap(x[a] - rp[s], box, True)
            phi, gr = _pairwise(x[a], m[a], box, True, grad=True)
            k2 = (dv * dv).sum(1)
            for q, y in zip(got, ((0.5 * m[a] * (k2 + phi)).sum()[None],
                                  m[a, None] * (HUBBLE * dv + gr), m[a, None] * dv, 0.5 * k2 + phi)):
                q.append(y)
        return dict(zip(("E", "grad_pos", "grad_vel", "grad_mass"), map(torch.cat, got)))
    energy, per = [], []
    for s in range(len(n)):
        a = slice(int(off[s]), int(off[s + 1]))
        e, r = _unbind_exact(x[a], v[a], m[a], rp[s], rv[s], box, periodic)
        if r is None:
            first = int(off[s])
            r = (m[first], x[first], v[first], torch.zeros(5, dtype=torch.float64, device="cuda"))
        energy.append(e)
        per.append(r)
    mb, xr, vr, sp = (torch.stack(q) for q in zip(*per))
    res = dict.fromkeys(_result_views(torch.empty(RESULT_BYTES, dtype=torch.uint8), 1))
    return dict(order=None, energy=torch.cat(energy),
                res=res | dict(mbound=mb, ref_pos=xr, ref_vel=vr, specific=sp))
