"""The work that programs have this library do, as timed cases.

A case names an entry point, a lattice and the options that matter to it:

  operator   one application of the Dirac operator or of its Schur form
             (Staggered.D, .stagD2ee) to a field on the device;
  vectors    stagDN, the operator on several fields at once (deflation,
             several sources of one propagator);
  solve      solveEE / solve at the three inner precisions, on device fields
             and on host arrays in QEX's order;
  shifts     cgm_ee, the shifted systems of a rational term for several
             right-hand sides;
  batch      solve_batched, many small lattices at once (an ensemble);
  smear      the HISQ links of a thin gauge field;
  chain      the chain rule back through that smearing;
  force      the HISQ fermion force of one molecular-dynamics step: smearing,
             solve, outer products and chain rule;
  gauge      the gauge part of a trajectory: forces, momentum and link updates,
             and the Hamiltonian at its end.

Lattices are those of the tests and of bench.py (8^4 to 32^4, 8^3 x 16,
24^3 x 48) and ragged ones with unequal even sides; draw() spreads them over
the same ranges.  Solves ask for |r|^2 <= 1e-24 |b|^2, as the tests' tighter
solves do, so that a solution is the same to about 1e-10 whichever inner
precision found it.

Gauge fields are exp(eps T)-like SU(3) matrices (warm starts), fat links 0.8
SU(3) plus Gaussian noise of 0.2, long links SU(3), all with the staggered
phases and the antiperiodic time boundary folded in; sources are Gaussian.
"""
import functools
import math

import numpy as np
import torch

from qex_b200 import _lib as L
from qex_b200 import md, smear, stag

DEV = "cuda"
C128 = torch.complex128
R2REQ = 1e-24
SLOPPY = {"none": L.SLOPPY_NONE, "single": L.SLOPPY_SINGLE, "half": L.SLOPPY_HALF}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def case(name, kind, dims, **options):
    c = {"kind": kind, "dims": "x".join(str(d) for d in dims), **options}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest call: a test or a tuning run on a toy lattice, all latency
        case("operator-naive-8", "operator", (8, 8, 8, 8), links="naive", fn="stagD2ee"),
        # a measurement code's D on a lattice whose sides are no powers of two
        case("operator-ragged", "operator", (12, 10, 14, 18), links="fat_naik", fn="D"),
        # the Schur operator where links stream from memory: the inside of every large solve
        case("operator-32", "operator", (32, 32, 32, 32), links="fat_naik", fn="stagD2ee"),
        # eight sources of a propagator on a production-shaped lattice
        case("vectors-24x48", "vectors", (24, 24, 24, 48), links="fat_naik", n=8),
        # a QEX host's solve: host arrays in and out, a lattice of the size of its examples
        case("solve-host-8x16", "solve", (8, 8, 8, 16), links="naive", fn="solve", mass=0.1, inner="none", mem="host"),
        # the mixed-precision solve of a large lattice
        case("solve-half-32", "solve", (32, 32, 32, 32), links="fat_naik", fn="solveEE", mass=0.05, inner="half",
             mem="device"),
        # a rational term: six poles for eight pseudofermions
        case("shifts-16", "shifts", (16, 16, 16, 16), links="fat_naik", mass=0.05, shifts=6, rhs=8),
        # an ensemble of small lattices of four shapes
        case("batch-16", "batch", (8, 8, 8, 16), lattices=16, mass=0.1),
        # HISQ links of a new configuration
        case("smear-32", "smear", (32, 32, 32, 32), lepage=0.0),
        # the chain rule alone, ragged
        case("chain-ragged", "chain", (12, 20, 14, 18), lepage=0.0),
        # one fermion force of a trajectory
        case("force-16", "force", (16, 16, 16, 16), mass=0.05, inner="half"),
        # the gauge part of a trajectory, tree-level Symanzik action
        case("gauge-symanzik-24", "gauge", (24, 24, 24, 24), beta=5.6, c1=-1.0 / 12.0, steps=2),
    ]


#: The volumes of each kind: from the smallest lattice that is used for it to the listed one.
VOLUMES = {
    "operator": (4 ** 4, 32 ** 4),
    "vectors": (8 ** 4, 24 ** 3 * 48),
    "solve": (8 ** 4, 24 ** 4),
    "shifts": (8 ** 4, 16 ** 4),
    "batch": (4 ** 4, 8 ** 3 * 16),
    "smear": (8 ** 4, 32 ** 4),
    "chain": (8 ** 4, 24 ** 4),
    "force": (8 ** 4, 16 ** 4),
    "gauge": (8 ** 4, 24 ** 4),
}


def log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw_dims(rng, lo, hi):
    """Four even sides >= 4 with a product in [lo, hi], its logarithm uniform; time is the longest more often than not."""
    for _ in range(1000):
        side = log_between(rng, lo, hi) ** 0.25
        dims = [max(4, 2 * round(0.5 * side * math.exp(rng.gauss(0.0, 0.25)))) for _ in range(4)]
        if lo <= math.prod(dims) <= hi:
            if rng.random() < 0.5:
                dims.sort()
            return tuple(dims)
    return (8, 8, 8, 8)


def draw(rng):
    kind = rng.choice(sorted(VOLUMES))
    dims = draw_dims(rng, *VOLUMES[kind])
    links = rng.choice(["naive", "fat_naik"])
    mass = round(log_between(rng, 0.05, 0.2), 4)
    lepage = rng.choice([0.0, 1.0])
    if kind == "operator":
        return case(None, kind, dims, links=links, fn=rng.choice(["D", "stagD2ee"]))
    if kind == "vectors":
        return case(None, kind, dims, links=links, n=rng.randint(1, 8))
    if kind == "solve":
        return case(None, kind, dims, links=links, fn=rng.choice(["solve", "solveEE"]), mass=mass,
                    inner=rng.choice(sorted(SLOPPY)), mem=rng.choice(["host", "device", "device"]))
    if kind == "shifts":
        return case(None, kind, dims, links=links, mass=mass, shifts=rng.randint(1, 6), rhs=rng.randint(1, 8))
    if kind == "batch":
        return case(None, kind, dims, lattices=rng.randint(2, 16), mass=mass)
    if kind in ("smear", "chain"):
        return case(None, kind, dims, lepage=lepage)
    if kind == "force":
        return case(None, kind, dims, mass=mass, inner=rng.choice(["none", "half"]))
    return case(None, kind, dims, beta=round(rng.uniform(5.0, 7.0), 3), c1=rng.choice([0.0, -1.0 / 12.0, -0.331]),
                steps=rng.randint(1, 2))


# ---------------------------------------------------------------------------
# geometry: QEX's checkerboard order (even sites first), signs of the links
# ---------------------------------------------------------------------------

def dims_of(c):
    return tuple(int(d) for d in c["dims"].split("x"))


def volume(dims):
    return math.prod(dims)


@functools.lru_cache(maxsize=64)
def coordinates(dims):
    """(4, V) coordinates of the sites in checkerboard order, and the order's place of each lexicographic site."""
    V = volume(dims)
    lex = torch.arange(V, device=DEV)
    x, t = [], lex
    for d in dims:
        x.append(t % d)
        t = t // d
    x = torch.stack(x)
    place = (lex + (x.sum(0) & 1) * V) // 2
    out = torch.empty_like(x)
    out[:, place] = x
    return out, place


def sign(dims, mu, hop):
    """Staggered phase of direction mu, and -1 where a hop crosses the antiperiodic time boundary."""
    x, _ = coordinates(dims)
    odd = (x[3], x[0] + x[3], x[0] + x[1] + x[3], torch.zeros_like(x[0]))[mu] & 1
    s = 1.0 - 2.0 * odd.double()
    return torch.where(x[3] + hop >= dims[3], -s, s) if mu == 3 else s


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def gaussian(shape, gen):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=gen, device=DEV, dtype=torch.float64))


def warm_su3(n, V, eps, gen):
    """n SU(3) link fields (n, 3, 3, V) near the identity: 1 + h + h^2/2 with h = eps times a Gaussian element of
    su(3), its rows made orthonormal and the last one the conjugate cross product."""
    a = gaussian((n, 3, 3, V), gen)
    h = 0.25 * eps * (a - a.conj().transpose(1, 2)) * math.sqrt(2.0)
    tr = (h[:, 0, 0] + h[:, 1, 1] + h[:, 2, 2]) / 3.0
    for i in range(3):
        h[:, i, i] -= tr
    u = h.clone()
    for k in range(3):
        u += 0.5 * h[:, :, k, None, :] * h[:, None, k, :, :]
    for i in range(3):
        u[:, i, i] += 1.0
    r0 = u[:, 0] / (u[:, 0].abs() ** 2).sum(1, keepdim=True).sqrt()
    r1 = u[:, 1] - (r0.conj() * u[:, 1]).sum(1, keepdim=True) * r0
    r1 = r1 / (r1.abs() ** 2).sum(1, keepdim=True).sqrt()
    r2 = torch.linalg.cross(r0, r1, dim=1).conj()
    return torch.stack([r0, r1, r2], dim=1)


def momenta(V, gen):
    """Traceless anti-Hermitian Gaussian momenta with <|P|^2> = 8 per link."""
    a = gaussian((4, 3, 3, V), gen)
    p = 0.5 * (a - a.conj().transpose(1, 2))
    tr = (p[:, 0, 0] + p[:, 1, 1] + p[:, 2, 2]) / 3.0
    for i in range(3):
        p[:, i, i] -= tr
    return p


def thin_links(dims, gen, eps=0.3):
    """Phased thin links (4, 3, 3, V), as they go into the smearing."""
    u = warm_su3(4, volume(dims), eps, gen)
    for mu in range(4):
        u[mu] *= sign(dims, mu, 1)
    return u


def link_list(dims, links, gen, eps=0.3):
    """Phased link list: four naive fields, or eight fat and long ones in turn."""
    if links == "naive":
        return thin_links(dims, gen, eps)
    V = volume(dims)
    g = torch.empty((8, 3, 3, V), dtype=C128, device=DEV)
    g[0::2] = 0.8 * warm_su3(4, V, eps, gen) + 0.2 * gaussian((4, 3, 3, V), gen)
    g[1::2] = warm_su3(4, V, eps, gen)
    for k in range(8):
        g[k] *= sign(dims, k // 2, 1 + 2 * (k % 2))
    return g


def even_source(V, gen):
    b = gaussian((3, V), gen)
    b[:, V // 2:] = 0
    return b


def shift_values(n):
    """n poles spaced evenly in their logarithm from 1e-4 to 1."""
    return [1e-4 if n == 1 else 10.0 ** (-4.0 + 4.0 * k / (n - 1)) for k in range(n)]


def batch_members(c):
    """Lattice sides and masses of a batch: four shapes around the given one, masses by a factor of two around the
    given one."""
    d = dims_of(c)
    shapes = [d, (d[0], d[1], d[2], d[0]), (d[0], d[0], d[0], d[0]), (d[3], d[1], d[2], d[3])]
    return [(shapes[j % 4], c["mass"] * 2.0 ** (((5 * j) % 7 - 3) / 6.0)) for j in range(c["lattices"])]


def host(t):
    """A device vector (3, V) as the host array (V, 3)."""
    return np.ascontiguousarray(t.cpu().numpy().T)


def inputs(c, seed):
    """The fields of a case, in the library's device layout."""
    gen, dims = generator(seed), dims_of(c)
    V, kind = volume(dims), c["kind"]
    if kind in ("operator", "vectors", "solve", "shifts"):
        d = {"links": link_list(dims, c["links"], gen)}
        if kind == "operator":
            d["x"] = gaussian((3, V), gen)
        elif kind == "vectors":
            d["x"] = [gaussian((3, V), gen) for _ in range(c["n"])]
        elif kind == "solve":
            d["x"] = gaussian((3, V), gen) if c["fn"] == "solve" else even_source(V, gen)
        else:
            d["x"] = [even_source(V, gen) for _ in range(c["rhs"])]
        return d
    if kind == "batch":
        return {"members": [{"dims": dj, "mass": mj, "links": link_list(dj, "naive", gen, 0.1 + 0.05 * (j % 9)),
                             "x": even_source(volume(dj), gen)} for j, (dj, mj) in enumerate(batch_members(c))]}
    if kind == "gauge":
        return {"links": warm_su3(4, V, 0.3, gen), "p": momenta(V, gen)}
    d = {"links": thin_links(dims, gen)}
    if kind == "chain":
        d["fat"], d["long"] = gaussian((4, 3, 3, V), gen), gaussian((4, 3, 3, V), gen)
    if kind == "force":
        d["x"] = even_source(V, gen)
    return d


# ---------------------------------------------------------------------------
# what a program holds, and one pass
# ---------------------------------------------------------------------------

def params(inner):
    return stag.SolverParams(r2req=R2REQ, sloppySolve=SLOPPY[inner])


def prepare(c, seed):
    d, dims, kind = inputs(c, seed), dims_of(c), c["kind"]
    s = {"case": c}
    if kind == "batch":
        s["lay"] = [stag.Layout(m["dims"]) for m in d["members"]]
        s["op"] = [stag.Staggered(lay, m["links"]) for lay, m in zip(s["lay"], d["members"])]
        s["b"] = [m["x"] for m in d["members"]]
        s["x"] = [torch.zeros_like(b) for b in s["b"]]
        s["mass"] = [m["mass"] for m in d["members"]]
        return s
    lay = s["lay"] = stag.Layout(dims)
    if kind in ("operator", "vectors", "solve", "shifts"):
        s["op"] = stag.Staggered(lay, d["links"])
        s["x"] = d["x"]
    if kind == "operator":
        s["r"] = torch.zeros_like(s["x"])
    elif kind == "vectors":
        s["r"] = [torch.zeros_like(x) for x in s["x"]]
    elif kind == "solve":
        if c["mem"] == "host":
            s["x"] = host(s["x"])
        s["r"] = np.zeros_like(s["x"]) if c["mem"] == "host" else torch.zeros_like(s["x"])
    elif kind == "shifts":
        s["r"] = [[torch.zeros_like(x) for _ in range(c["shifts"])] for x in s["x"]]
    elif kind == "gauge":
        s["u"], s["p"] = d["links"], d["p"]
        s["md"] = md.MD(lay, md.GaugeAction(lay, c["beta"], c["c1"]))
    else:
        s["u"] = d["links"]
        s["sm"] = smear.Smear(lay)
        s["coef"] = smear.newHISQ(c.get("lepage", 0.0), 1.0)
        s["r"] = [torch.zeros_like(s["u"]) for _ in range(2 if kind == "smear" else 1)]
        if kind == "chain":
            s["fat"], s["long"] = d["fat"], d["long"]
        if kind == "force":
            s["phi"] = d["x"]
            one = torch.eye(3, dtype=C128, device=DEV).reshape(1, 3, 3, 1).expand(8, 3, 3, lay.V).contiguous()
            s["op"] = stag.Staggered(lay, one, s["coef"].naik)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "operator":
        if c["fn"] == "D":
            s["op"].D(s["r"], s["x"], 0.1)
        else:
            s["op"].stagD2ee(s["r"], s["x"], 0.01)
        return s["r"]
    if kind == "vectors":
        s["op"].stagDN(L.EVEN, s["r"], s["x"], 0.1)
        return s["r"]
    if kind == "solve":
        solver = s["op"].solve if c["fn"] == "solve" else s["op"].solveEE
        solver(s["r"], s["x"], c["mass"], params(c["inner"]))
        return s["r"]
    if kind == "shifts":
        s["op"].cgm_ee(c["mass"], shift_values(c["shifts"]), s["x"], s["r"], params("single"))
        return s["r"]
    if kind == "batch":
        stag.solve_batched(s["op"], s["x"], s["b"], s["mass"], params("none"))
        return s["x"]
    if kind == "smear":
        s["sm"].smear(s["coef"], s["u"], *s["r"])
        return s["r"]
    if kind == "chain":
        s["sm"].smearDeriv(s["coef"], s["u"], s["fat"], s["long"], s["r"][0])
        return s["r"]
    if kind == "force":
        s["sm"].force(s["op"], s["coef"], s["u"], s["r"][0], s["phi"], c["mass"], params(c["inner"]))
        return s["r"]
    # a trajectory keeps its start for the accept/reject step
    u, p = s["u"].clone(), s["p"].clone()
    s["md"].leapfrog(u, p, 0.05 * c["steps"], c["steps"])
    return [u, p, s["md"].hamiltonian(u, p)]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

MATMUL = 9 * (3 * 8 - 2)  # a 3x3 complex product


def iterations(mass):
    """Of CG to R2REQ: half the root of the condition number times log(2/eps), with the largest eigenvalue 21 that the
    iteration counts of these fields show."""
    return 0.5 * math.sqrt(21.0 / (4.0 * mass * mass)) * math.log(2.0 / math.sqrt(R2REQ))


def operator_work(V, links, sites, real=8, fields=1):
    """Of one sweep over `sites` output sites of one parity: links of both ends once, the field once in and once out."""
    n = 4 if links == "naive" else 8
    flops = (570 if links == "naive" else 1146) * sites * fields
    long = 12 if links != "naive" and real < 8 else 18
    link = 4 * 18 + (4 * long if n == 8 else 0)
    return {"bytes": real * (2 * link * sites + 6 * fields * (V - sites) + 6 * fields * sites), "flops": flops}


def solve_work(V, links, mass, real):
    """Two half sweeps and the vector updates of each iteration (x, r, p read and written, A p read)."""
    its, half = iterations(mass), operator_work(V, links, V // 2, real)
    return {"bytes": its * (2 * half["bytes"] + 7 * 6 * real * (V // 2)), "flops": its * (2 * half["flops"] + 36 * V // 2)}


def smear_flops(V):
    """Both fat7 levels as QEX counts them, and the long links."""
    return V * (2 * 61632 + 4 * 2 * MATMUL)


def work(c):
    kind = c["kind"]
    V = volume(dims_of(c))
    field, link = 48 * V, 144 * V
    if kind == "operator":
        if c["fn"] == "D":
            n = 4 if c["links"] == "naive" else 8
            return {"bytes": n * link + 2 * field, "flops": V * (570 if n == 4 else 1146)}
        w = operator_work(V, c["links"], V // 2)  # the second sweep's links are the first's
        return {"bytes": w["bytes"], "flops": 2 * w["flops"]}
    if kind == "vectors":
        w = operator_work(V, c["links"], V // 2, 8, c["n"])
        return {"bytes": w["bytes"] + c["n"] * field // 2, "flops": w["flops"]}
    if kind == "solve":
        return solve_work(V, c["links"], c["mass"], {"none": 8, "single": 4, "half": 2}[c["inner"]])
    if kind == "shifts":
        its = iterations(math.sqrt(c["mass"] ** 2 + 0.25e-4))
        half = operator_work(V, c["links"], V // 2, 4, c["rhs"])
        vectors = 24 * (V // 2) * c["rhs"] * (3 + 4 * c["shifts"])
        return {"bytes": its * (2 * half["bytes"] + vectors), "flops": 2 * its * half["flops"]}
    if kind == "batch":
        each = [solve_work(volume(d), "naive", m, 8) for d, m in batch_members(c)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "smear":
        return {"bytes": 12 * link, "flops": smear_flops(V)}
    if kind == "chain":
        return {"bytes": 16 * link, "flops": 3 * smear_flops(V)}
    if kind == "force":
        w = solve_work(V, "fat_naik", c["mass"], 2 if c["inner"] == "half" else 8)
        return {"bytes": w["bytes"] + 8 * link + field, "flops": w["flops"] + 4 * smear_flops(V)}
    forces, paths = c["steps"] + 1, 6 * 2 + (18 * 4 if c["c1"] else 0) + 1
    return {"bytes": link * (forces * (8 + 8) + c["steps"] * 12 + 8),
            "flops": 4 * V * MATMUL * (forces * paths + 10 * c["steps"])}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits: fields as (sites in four dimensions, ...), neighbours by roll
# ---------------------------------------------------------------------------

def to_grid(dims, t, inner):
    """(..., inner axes, V) in checkerboard order -> (..., L3, L2, L1, L0, inner axes)."""
    _, place = coordinates(dims)
    t = t.index_select(-1, place)
    lead = t.ndim - 1 - inner
    t = t.reshape(t.shape[:-1] + tuple(reversed(dims)))
    order = list(range(lead)) + list(range(lead + inner, lead + inner + 4)) + list(range(lead, lead + inner))
    return t.permute(order).contiguous()


def from_grid(dims, t, inner):
    lead = t.ndim - 4 - inner
    order = list(range(lead)) + list(range(lead + 4, lead + 4 + inner)) + list(range(lead, lead + 4))
    t = t.permute(order).reshape([t.shape[i] for i in order[:lead + inner]] + [volume(dims)])
    _, place = coordinates(dims)
    out = torch.empty_like(t)
    out[..., place] = t
    return out


def ahead(t, mu, n=1, inner=2):
    """The field's value n sites further along mu."""
    return torch.roll(t, -n, dims=t.ndim - inner - 1 - mu)


def dag(m):
    return m.conj().transpose(-1, -2)


def grid_links(dims, u):
    return [to_grid(dims, u[k], 2) for k in range(u.shape[0])]


def two_d(g, x):
    """2D x for vectors (..., sites, 3)."""
    out = torch.zeros_like(x)
    for k, u in enumerate(g):
        mu, hop = (k // 2, 1 + 2 * (k % 2)) if len(g) == 8 else (k, 1)
        out += (u @ ahead(x, mu, hop, 1).unsqueeze(-1)).squeeze(-1)
        out -= ahead((dag(u) @ x.unsqueeze(-1)).squeeze(-1), mu, -hop, 1)
    return out


def parity_mask(dims, parity=0):
    x = torch.zeros((3, volume(dims)), dtype=C128, device=DEV)
    half = volume(dims) // 2
    x[:, parity * half:(parity + 1) * half] = 1
    return to_grid(dims, x, 1)


def conjugate_gradient(apply, b, batch_dims=0):
    """A x = b to rounding, systems along the leading dimensions independent."""
    axes = tuple(range(batch_dims, b.ndim))

    def dot(a, c):
        return (a.conj() * c).real.sum(axes, keepdim=True)

    x, r = torch.zeros_like(b), b.clone()
    p, r2 = r.clone(), dot(b, b)
    stop = 1e-29 * r2
    for i in range(20000):
        ap = apply(p)
        alpha = r2 / dot(p, ap).clamp_min(1e-300)
        x += alpha * p
        r -= alpha * ap
        new = dot(r, r)
        if i % 16 == 0 and bool((new <= stop).all()):
            break
        p = r + (new / r2.clamp_min(1e-300)) * p
        r2 = new
    return x


def solve_even(dims, g, b, m2, batch_dims=0):
    """(4 m2 - (2D)_eo (2D)_oe) x = b on even sites."""
    even = parity_mask(dims)
    return conjugate_gradient(lambda p: even * (4.0 * m2 * p - two_d(g, two_d(g, p))), even * b, batch_dims)


def staple(u, f, mu, nu):
    """Of the field f, whose links point along mu, on both sides along nu."""
    up = u[nu] @ ahead(f, nu) @ dag(ahead(u[nu], mu))
    down = dag(u[nu]) @ f @ ahead(u[nu], mu)
    return up + ahead(down, nu, -1)


def fat7(u, one, c3, c5, c7, cl):
    out = []
    for mu in range(4):
        acc = (one - 6.0 * cl) * u[mu]
        for nu in range(4):
            if nu == mu:
                continue
            s3 = staple(u, u[mu], mu, nu)
            acc = acc + c3 * s3
            if cl:
                acc = acc + cl * staple(u, s3, mu, nu)
            for rho in range(4):
                if rho in (mu, nu):
                    continue
                s5 = staple(u, s3, mu, rho)
                acc = acc + c5 * s5 + c7 * staple(u, s5, mu, 6 - mu - nu - rho)
        out.append(acc)
    return out


def unitary(x):
    """x (x^dag x)^(-1/2) by Newton's iteration for the polar factor."""
    for _ in range(9):
        x = 0.5 * (x + dag(torch.linalg.inv(x)))
    return x


def hisq(u, lepage):
    """Fat and long links with HISQ's coefficients (naik 1)."""
    def coefficients(f, naik):
        return (1.0 + 3.0 * f + naik) / 8.0, -1.0 / 16, 1.0 / 64, -1.0 / 384, -f / 16.0

    w = [unitary(x) for x in fat7(u, *coefficients(lepage, 0.0))]
    fat = fat7(w, *coefficients(2.0 - lepage, 1.0))
    long = [-1.0 / 24 * (w[mu] @ ahead(w[mu], mu) @ ahead(w[mu], mu, 2)) for mu in range(4)]
    return fat, long


def traceless_antihermitian(m):
    a = 0.5 * (m - dag(m))
    return a - torch.diagonal(a, dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3.0 * torch.eye(3, dtype=C128, device=DEV)


def gradient(scalar, u):
    """f with d scalar = sum Re Tr dU^dag f, for each field."""
    return torch.autograd.grad(scalar, u)


def real_inner(a, b):
    return sum((x.conj() * y).real.sum() for x, y in zip(a, b))


def gauge_action(u, beta, c1):
    """-(1/3) times the weighted sums of Re Tr over plaquettes and 2x1 rectangles."""
    total = 0.0
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            if nu < mu:
                loop = u[mu] @ ahead(u[nu], mu) @ dag(u[nu] @ ahead(u[mu], nu))
                total = total + (1.0 - 8.0 * c1) * beta * loop.diagonal(dim1=-2, dim2=-1).real.sum()
            if c1:
                two = u[mu] @ ahead(u[mu], mu)
                loop = two @ ahead(u[nu], mu, 2) @ dag(u[nu] @ ahead(two, nu))
                total = total + c1 * beta * loop.diagonal(dim1=-2, dim2=-1).real.sum()
    return -total / 3.0


def gauge_trajectory(dims, c, u, p):
    def force(v):
        with torch.enable_grad():
            w = [x.detach().requires_grad_(True) for x in v]
            f = gradient(gauge_action(w, c["beta"], c["c1"]), w)
        # the momentum's change is minus the action's derivative along it
        return [traceless_antihermitian(fx @ dag(x)) for fx, x in zip(f, v)]

    eps = 0.05
    kick = [0.5 * eps] + [eps] * (c["steps"] - 1) + [0.5 * eps]
    for k, e in enumerate(kick):
        if k:
            u = [torch.linalg.matrix_exp(eps * q) @ x for q, x in zip(p, u)]
        p = [q - e * f for q, f in zip(p, force(u))]
    kinetic = 0.5 * sum((q.abs() ** 2).sum() for q in p) - 16.0 * volume(dims)
    return [torch.stack([from_grid(dims, x, 2) for x in u]), torch.stack([from_grid(dims, x, 2) for x in p]),
            float(kinetic + gauge_action(u, c["beta"], c["c1"]))]


def hisq_chain(dims, u, lepage, fat, long):
    """d/du of sum Re Tr (fat^dag fat(u) + long^dag long(u))."""
    with torch.enable_grad():
        w = [x.detach().requires_grad_(True) for x in u]
        f, n = hisq(w, lepage)
        return gradient(real_inner(fat, f) + real_inner(long, n), w)


def exact(c, seed):
    kind, dims = c["kind"], dims_of(c)
    V = volume(dims)
    if V > {"solve": 16 ** 3 * 32, "chain": 24 ** 4, "gauge": 24 ** 4}.get(kind, 1 << 30):
        return None  # too long, or too much held for the derivative
    with torch.no_grad():
        d = inputs(c, seed)
        if kind == "batch":
            out = []
            for m in d["members"]:
                g = grid_links(m["dims"], m["links"])
                out.append(from_grid(m["dims"], solve_even(m["dims"], g, to_grid(m["dims"], m["x"], 1),
                                                           m["mass"] ** 2), 1))
            return out
        g = grid_links(dims, d["links"])
        if kind == "operator":
            x = to_grid(dims, d["x"], 1)
            if c["fn"] == "D":
                return from_grid(dims, 0.1 * x + 0.5 * two_d(g, x), 1)
            even = parity_mask(dims)
            x = even * x
            return from_grid(dims, even * (0.04 * x - two_d(g, two_d(g, x))), 1)
        if kind == "vectors":
            even = parity_mask(dims)
            return [from_grid(dims, even * (0.1 * x + two_d(g, x)), 1)
                    for x in (to_grid(dims, t, 1) for t in d["x"])]
        if kind == "solve":
            b, m = to_grid(dims, d["x"], 1), c["mass"]
            if c["fn"] == "solveEE":
                x = solve_even(dims, g, b, m * m)
            else:
                # D x = b: x_e from the Schur form of D^dag b, then x_o = (b_o - D_oe x_e) / m
                even = parity_mask(dims)
                x = 4.0 * solve_even(dims, g, m * b - 0.5 * two_d(g, b), m * m)
                x = x + (1.0 - even) * (b - 0.5 * two_d(g, x)) / m
            x = from_grid(dims, x, 1)
            return host(x) if c["mem"] == "host" else x
        if kind == "shifts":
            b = torch.stack([to_grid(dims, t, 1) for t in d["x"]])
            per = [solve_even(dims, g, b, c["mass"] ** 2 + 0.25 * s, 1) for s in shift_values(c["shifts"])]
            return [[from_grid(dims, y[j], 1) for y in per] for j in range(c["rhs"])]
        if kind == "gauge":
            return gauge_trajectory(dims, c, g, grid_links(dims, d["p"]))
        if kind == "smear":
            fat, long = hisq(g, c["lepage"])
            return [torch.stack([from_grid(dims, x, 2) for x in f]) for f in (fat, long)]
        if kind == "chain":
            f = hisq_chain(dims, g, c["lepage"], grid_links(dims, d["fat"]), grid_links(dims, d["long"]))
            return [torch.stack([from_grid(dims, x, 2) for x in f])]
        # force: psi = (4 y, (2D)_oe 4 y), its outer products (odd sites negated) through the chain rule
        fat, long = hisq(g, 0.0)
        ops = [x for pair in zip(fat, long) for x in pair]
        psi = 4.0 * solve_even(dims, ops, to_grid(dims, d["x"], 1), c["mass"] ** 2)
        psi = psi + two_d(ops, psi)
        flip = (2.0 * parity_mask(dims) - 1.0).unsqueeze(-1)
        outer = [[flip * psi.unsqueeze(-1) @ ahead(psi, mu, hop, 1).conj().unsqueeze(-2) for mu in range(4)]
                 for hop in (1, 3)]
        f = hisq_chain(dims, g, 0.0, *outer)
        return [torch.stack([from_grid(dims, traceless_antihermitian(fx @ dag(x)), 2) for fx, x in zip(f, g)])]
