"""The workloads this framework is timed on, and their values in 64 bits.

A case names one path through the public entry points (``context.Context`` on
device arrays, ``descriptor`` on host arrays) with its sizes and definition:

* ``step``        descriptor, then the force vector-Jacobian product, on a
                  neighbour list that is on the GPU -- a molecular-dynamics or
                  training step
* ``descriptor``  the descriptor alone (energies, clustering, data selection)
* ``md``          positions in: neighbour list, descriptor, forces
* ``host``        ``get_soap`` and ``soap_contract`` on host arrays, as a caller
                  of soap_turbo makes them
* ``cart``        the FP64 form with ``soap_cart_der`` written out, and its
                  contraction
* ``hessian``     the central-atom Hessian contracted with weight vectors

Structures are random periodic cubes.  With several species the sites
are the atoms of the second one, with one species they are all atoms.
"""
import math

import numpy as np
import torch

from soap_turbo_b200 import descriptor as drop_in
from soap_turbo_b200 import synthetic
from soap_turbo_b200.context import Context

RCUT, RSOFT, NF, SIGMA = 5.0, 4.5, 4.0, 0.5  # synthetic.Hyper's defaults, Angstrom
FRACTIONS = {1: (1.0,), 2: (0.5, 0.5), 3: (0.4, 0.4, 0.2)}
DENSITY = {1: 0.11, 2: 0.10, 3: 0.10}  # atoms per cubic Angstrom


def _case(path, basis, alpha, l_max, atoms, sigma_scaling=0.0, n_vec=0):
    return {"path": path, "basis": basis, "alpha": alpha, "l_max": l_max, "atoms": atoms,
            "sigma_scaling": sigma_scaling, "n_vec": n_vec}


def listed():
    return [
        # one small cell per call: active learning, an optimiser's inner loop
        _case("step", "poly3", "8", 8, 64) | {"name": "step_1species_64"},
        # the three-species structure of the benchmark: a production step
        _case("step", "poly3gauss", "8,8,8", 8, 4096) | {"name": "step_3species_4096"},
        # a large single-species cell, uncompressed descriptor
        _case("step", "poly3", "8", 8, 16384) | {"name": "step_1species_16384"},
        # a high-resolution basis with distance-dependent sigmas, ragged sizes
        _case("step", "poly3gauss", "9,7", 10, 777, 0.05) | {"name": "step_high_resolution_777"},
        # the third basis, which expands each pair in closed form
        _case("step", "poly3operator", "7,6", 7, 1500) | {"name": "step_operator_1500"},
        # descriptors of a large structure without forces
        _case("descriptor", "poly3gauss", "8,8,8", 8, 32768) | {"name": "descriptor_3species_32768"},
        # a step from positions: the neighbour list is rebuilt on the GPU
        _case("md", "poly3gauss", "8,8,8", 8, 4096) | {"name": "md_3species_4096"},
        # the reference's own calls on host arrays
        _case("host", "poly3gauss", "8,8,8", 8, 4096) | {"name": "host_3species_4096"},
        # callers that read soap_cart_der itself: compressed, and a small cell uncompressed
        _case("cart", "poly3gauss", "8,8,8", 8, 1024) | {"name": "cart_3species_1024"},
        _case("cart", "poly3", "8", 8, 100) | {"name": "cart_1species_100"},
        # second derivatives: one weight vector on the benchmark structure, several on a small cell
        _case("hessian", "poly3gauss", "8,8,8", 8, 4096, 0.0, 1) | {"name": "hessian_3species_4096"},
        _case("hessian", "poly3", "6", 6, 150, 0.0, 5) | {"name": "hessian_1species_150"},
    ]


def draw(rng):
    path = rng.choice(["step", "step", "step", "descriptor", "md", "host", "cart", "hessian"])
    most = {"step": 12000, "descriptor": 24000, "md": 8000, "host": 6000, "cart": 1000, "hessian": 3000}[path]
    atoms = int(round(math.exp(rng.uniform(math.log(50), math.log(most)))))
    bases = ["poly3", "poly3gauss"] if path == "hessian" else ["poly3", "poly3gauss", "poly3operator"]
    basis = rng.choice(bases)
    alpha = ",".join(str(rng.randint(4, 8)) for _ in range(rng.randint(1, 3)))
    sigma_scaling = rng.choice([0.0, 0.0, 0.05])
    if rng.random() < 0.3:
        alpha = rng.choice(["8", "8,8", "8,8,8"])  # the usual definitions
    l_max = rng.choice([4, 6, 7, 8, 8])
    if rng.random() < 0.15:  # beyond the usual resolution, on smaller structures
        l_max, atoms = rng.randint(9, 10), min(atoms, 700)
    n_vec = rng.randint(1, 3) if path == "hessian" else 0
    return _case(path, basis, alpha, l_max, atoms, sigma_scaling, n_vec)


# ------------------------------------------------------------------ the inputs
def _alpha(case):
    return [int(a) for a in case["alpha"].split(",")]


def _hyper(case):
    al = _alpha(case)
    return synthetic.Hyper(alpha_max=al, l_max=case["l_max"], basis=case["basis"],
                           atom_sigma_r_scaling=case["sigma_scaling"], atom_sigma_t_scaling=case["sigma_scaling"],
                           compress_mode="trivial" if len(al) > 1 else "None")


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _near(pos, box, sites, reach_of):
    """(site index, atom, displacement) of every image of every atom closer
    than reach_of, the site itself not counted."""
    images = 0 if box >= 2.0 * reach_of else math.ceil(reach_of / box)
    span = range(-images, images + 1)
    shifts = torch.tensor([(i, j, k) for i in span for j in span for k in span], dtype=torch.float64,
                          device=pos.device) * box
    at, atom, disp = [], [], []
    step = max(1, 40_000_000 // (pos.shape[0] * len(shifts)))
    for lo in range(0, len(sites), step):
        s = sites[lo:lo + step]
        d = pos[None] - pos[s][:, None]
        if images == 0:
            d = d - box * torch.round(d / box)
        d = d[:, :, None] + shifts[None, None]
        close = (d * d).sum(-1) < reach_of * reach_of
        close[torch.arange(len(s), device=pos.device), s, len(shifts) // 2] = False
        i, j, k = torch.nonzero(close, as_tuple=True)
        at.append(i + lo)
        atom.append(j)
        disp.append(d[i, j, k])
    return torch.cat(at), torch.cat(atom), torch.cat(disp)


def _geometry(case, seed):
    """A structure as a run of molecular dynamics passes through it: the case
    fixes the cell, the species and who neighbours whom, the seed moves the
    atoms (none across another's cutoff, so that every seed gives the same
    number of pairs), turns the axes and shifts the origin.  Returns positions,
    box side, species, sites and the neighbours (site index, atom,
    displacement) ordered by site, atom and distance."""
    n_sp = len(_alpha(case))
    st = synthetic.random_structure(case["atoms"], density=DENSITY[n_sp], d_min=1.1 if n_sp == 1 else 0.9,
                                    fractions=FRACTIONS[n_sp], seed=case["atoms"])
    dev = _device()
    pos, box = torch.as_tensor(st.positions, device=dev), st.box
    species = torch.as_tensor(st.species.astype(np.int64), device=dev)
    sites = torch.arange(case["atoms"], device=dev) if n_sp == 1 else torch.nonzero(species == 1)[:, 0]
    rng = np.random.default_rng(seed)
    move = torch.as_tensor(rng.normal(scale=0.02, size=(case["atoms"], 3)).clip(-0.05, 0.05), device=dev)
    at, atom, disp = _near(pos, box, sites, RCUT + 0.2)
    inside = torch.linalg.vector_norm(disp, dim=1) < RCUT
    while True:
        moved = disp + move[atom] - move[sites[at]]
        crossed = (torch.linalg.vector_norm(moved, dim=1) < RCUT) != inside
        if not bool(crossed.any()):
            break
        move[atom[crossed]] = 0.0
        move[sites[at[crossed]]] = 0.0
    axes = torch.as_tensor(rng.permutation(3), device=dev)
    signs = torch.as_tensor(rng.choice([-1.0, 1.0], 3), device=dev)
    origin = torch.as_tensor(rng.random(3) * box, device=dev)
    pos = torch.remainder(((pos + move) * signs)[:, axes] + origin, box)
    at, atom, disp = at[inside], atom[inside], (moved[inside] * signs)[:, axes]
    key = torch.argsort(torch.linalg.vector_norm(disp, dim=1), stable=True)
    key = key[torch.argsort((at * case["atoms"] + atom)[key], stable=True)]
    return pos, box, species, sites, at[key], atom[key], disp[key]


def _list(case, seed):
    """The neighbour list in get_soap's layout (each row starts with the site itself)."""
    _, _, species, sites, at, atom, disp = _geometry(case, seed)
    n_sites, n_sp = len(sites), len(_alpha(case))
    counts = torch.bincount(at, minlength=n_sites) + 1
    start = torch.cumsum(counts, 0) - counts
    n_pairs = n_sites + len(at)
    where = torch.arange(len(at), device=at.device) + at + 1  # the rows before, and this one, have a self pair
    d = torch.zeros(n_pairs, 3, dtype=torch.float64, device=at.device)
    j = torch.empty(n_pairs, dtype=torch.int64, device=at.device)
    d[where], j[where], j[start] = disp, atom, sites
    r = torch.linalg.vector_norm(d, dim=1)
    theta = torch.atan2(torch.hypot(d[:, 0], d[:, 1]), d[:, 2])
    phi = torch.atan2(d[:, 1], d[:, 0])
    mask = torch.stack([species[j] == s for s in range(n_sp)]).to(torch.uint8)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    return synthetic.NeighbourList(
        n_sites=n_sites, n_neigh=host(counts.to(torch.int32)), rjs=host(r), thetas=host(theta), phis=host(phi),
        mask=host(mask), species=host((species[sites] + 1).to(torch.int32)).reshape(n_sites, 1),
        species_multiplicity=np.ones(n_sites, dtype=np.int32), site_atom=host(sites), neigh_atom=host(j),
        disp=host(d))


def _weights(seed, *shape):
    """The upstream gradient, or the Hessian's weight vectors: normal deviates."""
    gen = torch.Generator(device=_device()).manual_seed(seed * 7919 + 11)
    return torch.randn(*shape, dtype=torch.float64, device=_device(), generator=gen)


def prepare(case, seed):
    hp = _hyper(case)
    path = case["path"]
    state = {"path": path, "case": case}
    if path == "host":
        nl = _list(case, seed)
        if len(hp.alpha_max) > 1:
            n_soap, nz, p_i, p_j, p_el = drop_in.get_compress_indices("trivial", hp.alpha_max, hp.l_max)
        else:
            n_soap, nz, p_i, p_j, p_el = hp.n_max * (hp.n_max + 1) // 2 * (hp.l_max + 1), 0, None, None, None
        state["args"] = dict(
            n_sites=nl.n_sites, n_neigh=nl.n_neigh, n_species=hp.n_species, species=np.asfortranarray(nl.species.T),
            species_multiplicity=nl.species_multiplicity, n_atom_pairs=nl.n_pairs, mask=nl.mask.T, rjs=nl.rjs,
            thetas=nl.thetas, phis=nl.phis, alpha_max=hp.alpha_max, l_max=hp.l_max, basis=hp.basis,
            scaling_mode=hp.scaling_mode, radial_enhancement=hp.radial_enhancement, do_timing=False,
            do_derivatives=True, compress_soap=len(hp.alpha_max) > 1, compress_P_nonzero=nz, compress_P_i=p_i,
            compress_P_j=p_j, compress_P_el=p_el, soap_cart_der=None, contract=True,
            **{k: getattr(hp, k) for k in (
                "rcut_hard", "rcut_soft", "nf", "global_scaling", "atom_sigma_r", "atom_sigma_r_scaling",
                "atom_sigma_t", "atom_sigma_t_scaling", "amplitude_scaling", "central_weight")})
        state["soap"] = np.zeros((n_soap, nl.n_sites), order="F")
        state["pair"] = np.zeros((3, nl.n_pairs), order="F")
        state["G"] = np.asfortranarray(_weights(seed, n_soap, nl.n_sites).cpu().numpy().T)
        return state
    # the second radial derivatives exist for the unified filter seed only
    ctx = Context(hp, legacy_filter_seed=path != "hessian")
    state["ctx"] = ctx
    if path == "md":
        pos, box, species, sites = _geometry(case, seed)[:4]
        state.update(pos=pos, lattice=np.eye(3) * box, species=(species + 1).to(torch.int32),
                     sites=sites.to(torch.int32), G=_weights(seed, ctx.n_soap, len(sites)))
        return state
    nl = _list(case, seed)
    state["batch"] = ctx.batch(nl)
    if path == "hessian":
        state["vecs"] = _weights(seed, nl.n_sites, case["n_vec"], ctx.n_soap)
    elif path != "descriptor":
        state["G"] = _weights(seed, ctx.n_soap, nl.n_sites)  # the reference's G(n_sites, n_soap)
    return state


def run(state):
    path = state["path"]
    if path == "host":
        soap, pair = state["soap"], state["pair"]
        soap[...] = 0.0  # get_soap adds into a compressed soap
        drop_in.get_soap(soap=soap, **state["args"])
        drop_in.soap_contract(soap, state["G"], 1.0, pair)
        return {"soap": soap, "pair": pair}
    ctx = state["ctx"]
    if path == "md":
        b = ctx.build_neighbors(state["pos"], state["lattice"], state["species"], state["sites"])
        soap = ctx.descriptor(b)
        return {"soap": soap, "pair": ctx.contract(b, soap, state["G"])}
    b = state["batch"]
    if path == "step":
        soap = ctx.descriptor(b)
        return {"soap": soap, "pair": ctx.contract(b, soap, state["G"])}
    if path == "descriptor":
        return {"soap": ctx.descriptor(b, keep=False)}
    if path == "cart":
        soap, cart = ctx.descriptor_fp64(b, cart=True)
        return {"soap": soap, "cart": cart, "pair": ctx.contract_cart_der(b, cart, state["G"])}
    return {"hess": ctx.central_hessian(b, state["vecs"])}


# ------------------------------------------------------------------ what a pass needs
def _kept(case):
    """(n, n', l) of every component, in order."""
    al = _alpha(case)
    first = {sum(al[:s]) for s in range(len(al))}
    n_max = sum(al)
    return [(n, m, l) for n in range(n_max) for m in range(n, n_max) for l in range(case["l_max"] + 1)
            if len(al) == 1 or n in first or m in first]


def work(case):
    al, n_sp = _alpha(case), len(_alpha(case))
    path, n_max, n_soap = case["path"], sum(_alpha(case)), len(_kept(case))
    k_max = (case["l_max"] + 1) * (case["l_max"] + 2) // 2
    sites = case["atoms"] * (1.0 if n_sp == 1 else FRACTIONS[n_sp][1])
    pairs = sites * (1.0 + DENSITY[n_sp] * 4.0 / 3.0 * math.pi * RCUT ** 3)
    a = sum(al) / n_sp
    geometry = pairs * (24 + n_sp) + 12 * sites
    soap, grad, force = 8 * n_soap * sites, 8 * n_soap * sites, 24 * pairs
    forward = pairs * (4 * a * a + 4 * a * k_max) + sites * 4 * n_soap * (case["l_max"] + 1)
    vjp = pairs * 16 * a * k_max + sites * 4 * n_max * n_max * k_max
    if path == "descriptor":
        return {"bytes": geometry + soap, "flops": forward}
    if path in ("step", "host"):
        return {"bytes": geometry + soap + grad + force, "flops": forward + vjp}
    if path == "md":
        return {"bytes": 28 * case["atoms"] + soap + grad + force, "flops": forward + vjp}
    if path == "cart":  # each derivative component: three products of the pair's sums, and its contraction
        cart = 24 * n_soap * pairs
        return {"bytes": geometry + soap + grad + force + cart,
                "flops": forward + pairs * (32 * n_max * k_max + 45 * n_soap)}
    v = case["n_vec"]
    return {"bytes": geometry + v * (grad + 72 * pairs),
            "flops": forward + sites * v * 16 * n_max * n_max * k_max / n_sp
            + pairs * k_max * (24 * a + v * (6 * a * 2 + 18 * a + 120))}


# ------------------------------------------------------------------ the values in 64 bits
def _overlap(basis, a):
    """Overlaps of one species' primitive functions (cutoff 1)."""
    s = np.ones((a, a))
    top = a - 1 if basis == "poly3gauss" else a
    for i in range(1, top + 1):
        for j in range(i + 1, top + 1):
            s[i - 1, j - 1] = s[j - 1, i - 1] = math.sqrt(float((5 + 2 * i) * (5 + 2 * j))) / (5 + i + j)
    if basis == "poly3gauss":
        sig = SIGMA / RCUT
        s2, i0, n0, n1 = sig * sig, 0.0, 1.0, 1.0
        i1 = math.sqrt(math.pi / 2.0) * sig * math.erf(1.0 / math.sqrt(2.0) / sig)
        for n in range(-1, a):
            n2 = math.sqrt(1.0 / (2 * n + 5))
            i2 = s2 * (n + 1) * n0 / n2 * i0 + n1 / n2 * i1 - s2 / n2
            if n > 0:
                s[n - 1, a - 1] = s[a - 1, n - 1] = i2 * math.sqrt(2.0) / math.sqrt(sig) / math.pi ** 0.25
            n0, n1, i0, i1 = n1, n2, i1, i2
        s[a - 1, a - 1] = 1.0
    return s


def _orthonormal(s):
    """S^(-1/2), by Jacobi rotations in extended precision: S is too
    ill-conditioned for 64 bits."""
    a = np.array(s, dtype=np.longdouble)
    v = np.eye(len(a), dtype=np.longdouble)
    for _ in range(60):
        if (np.tril(a, -1) ** 2).sum() < 1e-70:
            break
        for p in range(len(a)):
            for q in range(p + 1, len(a)):
                if abs(a[p, q]) < 1e-300:
                    continue
                th = (a[q, q] - a[p, p]) / (2 * a[p, q])
                t = (1 if th >= 0 else -1) / (abs(th) + np.sqrt(th * th + 1))
                c = 1 / np.sqrt(t * t + 1)
                rot = np.array([[c, t * c], [-t * c, c]])
                a[:, [p, q]] = a[:, [p, q]] @ rot
                a[[p, q]] = rot.T @ a[[p, q]]
                v[:, [p, q]] = v[:, [p, q]] @ rot
    return ((v / np.sqrt(np.diag(a))) @ v.T).astype(np.float64)


def _recursion(r, basis, a, c, legacy, n_hi):
    """The primitive overlaps pol(1..n_hi) of poly3 and poly3gauss with the
    atom's Gaussian (filtered beyond the soft cutoff) and what their
    derivatives need, in units of the cutoff."""
    rj, rs, dr = r / RCUT, RSOFT / RCUT, 1.0 - RSOFT / RCUT
    nv = lambda n: 1.0 if n == -3 else math.sqrt(1.0 / (2 * n + 5))  # noqa: E731
    root, h = math.sqrt(math.pi / 2.0), math.sqrt(0.5)
    sig = SIGMA / RCUT + c * rj
    s2 = sig * sig
    c1 = s2 * torch.exp(-0.5 * (rs - rj) ** 2 / s2)
    c2 = s2 * torch.exp(-0.5 * rj * rj / s2)
    q = (dr / NF) ** 2
    sf = sig * (dr / NF) / torch.sqrt(s2 + q)
    rf = (s2 * rs + q * rj) / (s2 + q)
    sf2 = sf * sf
    pref = torch.where(rs - rj < 4.0 * sig, torch.exp(-0.5 * (rs - rj) ** 2 / (s2 + q)), torch.zeros_like(rj))
    c2f = sf2 * torch.exp(-0.5 * (rs - rf) ** 2 / sf2)
    t = [torch.zeros_like(rj), root * sig * (torch.erf((rs - rj) * h / sig) + torch.erf(rj * h / sig))]
    z = [torch.zeros_like(rj), root * sf * (torch.erf((1.0 - rf) * h / sf) - torch.erf((rs - rf) * h / sf))]
    for n in range(-1, n_hi + 1):
        if n >= 0:
            c1, c2f = c1 * dr, c2f * dr
        ra = 0.0 if n == -1 else (n + 1) * nv(n - 2) / nv(n)
        rb, rc = nv(n - 1) / nv(n), 1.0 / nv(n)
        t.append(s2 * ra * t[-2] - rb * (rj - 1.0) * t[-1] + (c1 - c2) * rc)
        z.append(sf2 * ra * z[-2] - rb * (rf - 1.0) * z[-1] - c2f * rc)
        if n == -1 and not legacy:
            z[-1] = z[-1] + sf2 * torch.exp(-0.5 * (1.0 - rf) ** 2 / sf2) * rc
    t, z = t[4:], z[4:]  # n = 1, 2, ...
    return rj, sig, t, z, pref, rf, sf, q


def _amplitude(rj, sig, c, ends=True):
    """The amplitude and its derivative; poly3 and poly3gauss end it where it is below 1e-10."""
    hh = 1.0 + 2.0 * rj ** 3 - 3.0 * rj * rj
    on = hh > (1.0e-10 if ends else -1.0)
    zero = torch.zeros_like(rj)
    return torch.where(on, hh / sig, zero), torch.where(on, (6.0 * rj * rj - 6.0 * rj) / sig - c * hh / sig ** 2, zero)


def _gauss_moments(rj, sig):
    """The overlap of the atom's Gaussian with the one at the origin, and its two next moments."""
    s0 = SIGMA / RCUT
    s2, s02 = sig * sig, s0 * s0
    tot = s02 + s2
    near = rj < 4.0 * (s0 + sig)
    norm = math.sqrt(2.0 / s0) / math.pi ** 0.25
    m0 = torch.exp(-0.5 * rj * rj / tot) * math.sqrt(math.pi / 2.0) * sig * s0 / torch.sqrt(tot) * norm * (
        1.0 + torch.erf(s0 / sig * rj * math.sqrt(0.5) / torch.sqrt(tot)))
    edge = norm * torch.exp(-0.5 * rj * rj / s2)
    zero = torch.zeros_like(rj)
    m0, edge = torch.where(near, m0, zero), torch.where(near, edge, zero)
    m1 = s02 * s2 / tot * edge - s2 * rj / tot * m0
    m2 = -s02 * s2 / tot * edge * rj - s2 * rj / tot * m1 + s02 * s2 / tot * m0
    return m0, m1, m2


def _operator_overlaps(rj, sig, a):
    """poly3operator's overlaps of the piecewise-cubic atom density, by
    Gauss-Legendre quadrature of its polynomial pieces (exact to rounding)."""
    rs, cw = RSOFT / RCUT, 2.0 * math.sqrt(2.0 * math.log(2.0))
    w = cw * sig
    x, g = np.polynomial.legendre.leggauss(16)
    x, g = (torch.as_tensor(v, device=rj.device) for v in (x, g))
    power = torch.arange(3, a + 3, device=rj.device)
    fac = torch.sqrt(2.0 * power.double() + 1.0)
    total = 0.0
    zero, one, soft = torch.zeros_like(rj), torch.ones_like(rj), torch.full_like(rj, rs)
    for buffer in (False, True):
        lo_z, hi_z = (soft, one) if buffer else (zero, soft)
        for right in (False, True):
            lo = torch.maximum(lo_z, rj if right else rj - w)
            hi = torch.minimum(hi_z, rj + w if right else rj)
            half = torch.clamp(hi - lo, min=0.0) / 2.0
            y = lo[:, None] + half[:, None] * (1.0 + x)
            u = (y - rj[:, None]) / w[:, None]
            f = 1.0 - 3.0 * u * u + (2.0 if right else -2.0) * u ** 3
            if buffer:
                v = (y - rs) / (cw * (1.0 - rs))
                f = f * (1.0 - 3.0 * v * v + 2.0 * v ** 3)
            total = total + ((f * g * half[:, None])[:, :, None] * (1.0 - y)[:, :, None] ** power).sum(1)
    return total * fac


def _radial(r, basis, a, c, w, legacy, differentiable):
    """R_n(r): (pairs, a).  With the legacy filter seed the derivative that the
    method defines is not that of the value; it is attached to it here."""
    w = torch.as_tensor(w, device=r.device)
    if basis == "poly3operator":
        rj = r / RCUT
        sig = SIGMA / RCUT + c * rj
        amp, _ = _amplitude(rj, sig, c, ends=False)
        return (amp[:, None] * _operator_overlaps(rj, sig, a)) @ w * math.sqrt(RCUT)
    n_poly = a - 1 if basis == "poly3gauss" else a
    r0 = r if differentiable else r.detach()
    rj, sig, t, z, pref, rf, sf, q = _recursion(r0, basis, a, c, legacy, n_poly + 2)
    amp, ampd = _amplitude(rj, sig, c)
    pol = [t[n] + pref * z[n] for n in range(n_poly + 2)]
    rows = pol[:n_poly]
    if basis == "poly3gauss":
        m0, m1, m2 = _gauss_moments(rj, sig)
        rows = rows + [m0]
    val = amp[:, None] * torch.stack(rows, 1) @ w * math.sqrt(RCUT)
    if differentiable:
        return val
    nv = lambda n: math.sqrt(1.0 / (2 * n + 5))  # noqa: E731
    rs, f = RSOFT / RCUT, rj - 1.0
    s2 = sig * sig
    g = c * f / sig
    fs = rs - rj
    dpref = pref * (fs / (s2 + q) + fs * fs / (s2 + q) ** 2 * sig * c)
    drf = (2.0 * sig * rs * c + q) / (s2 + q) - (s2 * rs + q * rj) * 2.0 * sig * c / (s2 + q) ** 2
    dsf = c * (1.0 - RSOFT / RCUT) / NF / torch.sqrt(s2 + q) * (1.0 - s2 / (s2 + q))
    ff = rf - 1.0
    gg = dsf * ff / sf
    der = []
    for n in range(1, n_poly + 1):
        r1, r2 = nv(n + 1) / nv(n), nv(n + 2) / nv(n)
        d = f / s2 * (g - 1.0) * t[n - 1] + r1 / s2 * (2.0 * g - 1.0) * t[n] + r2 * c / sig ** 3 * t[n + 1]
        d = d + pref * (ff / sf ** 2 * (gg - drf) * z[n - 1] + r1 / sf ** 2 * (2.0 * gg - drf) * z[n]
                        + r2 * dsf / sf ** 3 * z[n + 1]) + dpref * z[n - 1]
        der.append(amp * d + ampd * pol[n - 1])
    if basis == "poly3gauss":
        der.append(amp * (m1 / s2 + c * m2 / sig ** 3) + ampd * m0)
    der = torch.stack(der, 1) @ w / math.sqrt(RCUT)
    return val + der * (r - r0)[:, None]


def _angular(d, l_max, c):
    """amp i_l e^{-x^2} Y_lm factor of displacements d: (pairs, k) complex, from
    Q_l^m = d^m P_l / dt^m and ((x - iy)/r)^m, which have no pole."""
    r = torch.sqrt((d * d).sum(1))
    t = d[:, 2] / r
    w = torch.complex(d[:, 0] / r, -d[:, 1] / r)
    sig = SIGMA + c * r
    amp = RCUT ** 2 / sig ** 2
    z = (r / sig) ** 2
    e = torch.exp(-2.0 * z)
    il = [(1.0 - e) / (2.0 * z), (z - 1.0 + e * (z + 1.0)) / (2.0 * z * z)]
    for l in range(2, l_max + 1):
        il.append(il[l - 2] - (2 * l - 1) / z * il[l - 1])
    leg = {}
    for l in range(l_max + 1):
        for m in range(l + 1):
            if l == m:
                leg[l, m] = torch.full_like(t, float(np.prod(np.arange(1, 2 * l, 2)))) if l else torch.ones_like(t)
            elif l == m + 1:
                leg[l, m] = (2 * m + 1) * t * leg[m, m]
            else:
                leg[l, m] = ((2 * l - 1) * t * leg[l - 1, m] - (l + m - 1) * leg[l - 2, m]) / (l - m)
    out, powers = [], [torch.ones_like(w)]
    for m in range(l_max):
        powers.append(powers[-1] * w)
    for l in range(l_max + 1):
        for m in range(l + 1):
            y = math.sqrt((2 * l + 1) / (4.0 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            out.append((amp * il[l] * leg[l, m] * (-1) ** m * y) * powers[m])
    return torch.stack(out, 1)


class _Exact:
    """The descriptor of a chunk of sites as a function of the displacements."""

    def __init__(self, case, legacy):
        self.case, self.legacy, self.al = case, legacy, _alpha(case)
        self.l_max, self.c, self.basis = case["l_max"], case["sigma_scaling"], case["basis"]
        self.n_max, self.dev = sum(self.al), _device()
        over = [_overlap("poly3gauss" if self.basis == "poly3gauss" else "poly3", a) for a in self.al]
        self.w = [_orthonormal(s) for s in over]
        kept = np.array(_kept(case))
        self.n, self.m, self.l = (torch.as_tensor(kept[:, i], device=self.dev) for i in range(3))
        self.base = torch.tensor([1.0 if n == m else math.sqrt(2.0) for n, m, _ in kept.tolist()],
                                 dtype=torch.float64, device=self.dev)
        self.mult = [torch.tensor([1.0] + [2.0] * l, dtype=torch.float64, device=self.dev)
                     for l in range(self.l_max + 1)]
        # the site itself: the origin Gaussian's term, or its own expansion at r = 0
        self.central = []
        y00 = math.sqrt(0.25 / math.pi) * RCUT ** 2 / SIGMA ** 2
        for s, a in enumerate(self.al):
            if self.basis == "poly3gauss":
                f = math.sqrt(4.0 * math.pi) * math.pi ** 0.25 * math.sqrt(SIGMA / 2.0) * RCUT ** 3 / SIGMA ** 3
                row = f * (self.w[s] @ over[s][:, a - 1])
            else:
                zero = torch.zeros(1, dtype=torch.float64, device=self.dev)
                row = (4.0 * math.pi * y00 * self.radial_of(s, zero, False)[0]).cpu().numpy()
            self.central.append(torch.as_tensor(row, device=self.dev))

    def radial_of(self, s, r, differentiable):
        return _radial(r, self.basis, self.al[s], self.c, self.w[s], self.legacy, differentiable)

    def radial(self, d, spec, differentiable):
        r = torch.sqrt((d * d).sum(1))
        out = torch.zeros(len(d), self.n_max, dtype=torch.float64, device=self.dev)
        nb = 0
        for s, a in enumerate(self.al):
            own = torch.nonzero(spec == s)[:, 0]
            block = torch.zeros(len(own), self.n_max, dtype=torch.float64, device=self.dev)
            cols = torch.arange(nb, nb + a, device=self.dev)
            block = block.index_copy(1, cols, self.radial_of(s, r[own], differentiable))
            out = out.index_copy(0, own, block)
            nb += a
        return 4.0 * math.pi * out

    def coefficients(self, rad, ang, row, n_sites, site_spec):
        """c_nlm: (sites, n, k)."""
        counts = torch.bincount(row, minlength=n_sites)
        col = torch.arange(len(row), device=self.dev) - (torch.cumsum(counts, 0) - counts)[row]
        width = max(1, int(counts.max()))
        at = (row * width + col)
        dense = lambda v: torch.zeros(n_sites * width, v.shape[1], dtype=v.dtype, device=self.dev).index_copy(  # noqa: E731
            0, at, v).reshape(n_sites, width, -1)
        c = dense(rad).to(torch.complex128).transpose(1, 2) @ dense(ang)
        own = torch.zeros_like(c)
        nb = 0
        for s, a in enumerate(self.al):
            hit = torch.nonzero(site_spec == s)[:, 0]
            own[hit, nb:nb + a, 0] = self.central[s].to(torch.complex128)
            nb += a
        return c + own

    def power(self, c):
        """The unnormalised components: (sites, n_soap)."""
        full = []
        for l in range(self.l_max + 1):
            x = c[:, :, l * (l + 1) // 2:(l + 1) * (l + 2) // 2]
            full.append(((x * self.mult[l]) @ x.conj().transpose(1, 2)).real)
        return torch.stack(full, 1)[:, self.l, self.n, self.m] * self.base

    def soap(self, d, spec, row, n_sites, site_spec, differentiable=False):
        c = self.coefficients(self.radial(d, spec, differentiable), _angular(d, self.l_max, self.c), row, n_sites,
                              site_spec)
        p = self.power(c)
        return p / torch.linalg.vector_norm(p, dim=1, keepdim=True)

    def jacobian(self, d, spec, row, n_sites, site_spec):
        """d soap / d displacement of every pair: (pairs, n_soap, 3)."""
        rad = self.radial(d.clone().requires_grad_(), spec, False).detach()
        ang = _angular(d, self.l_max, self.c)
        c = self.coefficients(rad, ang, row, n_sites, site_spec)
        p = self.power(c)
        norm = torch.linalg.vector_norm(p, dim=1)
        out = torch.empty(len(d), len(self.l), 3, dtype=torch.float64, device=self.dev)
        for lo in range(0, len(d), 2048):
            sl = slice(lo, lo + 2048)
            for a in range(3):
                step = torch.zeros_like(d[sl])
                step[:, a] = 1.0
                dang = torch.func.jvp(lambda v: _angular(v, self.l_max, self.c), (d[sl],), (step,))[1]
                drad = torch.func.jvp(lambda v: self.radial(v, spec[sl], False), (d[sl],), (step,))[1] \
                    if self.basis == "poly3operator" else self._radial_slope(d[sl], spec[sl], a)
                da = (drad.to(torch.complex128)[:, :, None] * ang[sl][:, None]
                      + rad[sl].to(torch.complex128)[:, :, None] * dang[:, None])
                full = []
                for l in range(self.l_max + 1):
                    k = slice(l * (l + 1) // 2, (l + 1) * (l + 2) // 2)
                    x = ((da[:, :, k] * self.mult[l]) @ c[row[sl]][:, :, k].conj().transpose(1, 2)).real
                    full.append(x + x.transpose(1, 2))
                out[sl, :, a] = torch.stack(full, 1)[:, self.l, self.n, self.m] * self.base
            q = p[row[sl]] / norm[row[sl], None]
            v = out[sl]
            out[sl] = (v - q[:, :, None] * (q[:, None] @ v)) / norm[row[sl], None, None]
        return out, p / norm[:, None]

    def _radial_slope(self, d, spec, a):
        """d R_n / d d_a: R_n depends on its own pair alone, one backward pass per n."""
        x = d.clone().requires_grad_()
        rad = self.radial(x, spec, False)
        return torch.stack([torch.autograd.grad(rad[:, n].sum(), x, retain_graph=True)[0][:, a]
                            for n in range(self.n_max)], 1)


def _with_self(row, per_pair, n_sites):
    """Rows of neighbour values with each site's own entry, minus their sum, in front."""
    n = len(row)
    out = torch.zeros(n + n_sites, *per_pair.shape[1:], dtype=torch.float64, device=per_pair.device)
    where = torch.arange(n, device=row.device) + row + 1
    out[where] = per_pair
    counts = torch.bincount(row, minlength=n_sites) + 1
    out[torch.cumsum(counts, 0) - counts] = -torch.zeros(
        n_sites, *per_pair.shape[1:], dtype=torch.float64, device=per_pair.device).index_add(0, row, per_pair)
    return out


def exact(case, seed):
    path = case["path"]
    _, _, species, sites, at, atom, disp = _geometry(case, seed)
    ex = _Exact(case, legacy=path != "hessian")
    n_soap, n_sites = len(_kept(case)), len(sites)
    bounds = torch.cat([torch.zeros(1, dtype=torch.int64, device=at.device),
                        torch.cumsum(torch.bincount(at, minlength=n_sites), 0)]).tolist()
    weights = None
    if path == "hessian":
        weights = _weights(seed, n_sites, case["n_vec"], n_soap)
    elif path != "descriptor":
        weights = _weights(seed, n_soap, n_sites).T
    soaps, firsts, carts = [], [], []
    step = {"hessian": 96, "cart": 64}.get(path, 1024)
    for lo in range(0, n_sites, step):
        hi = min(n_sites, lo + step)
        sl = slice(bounds[lo], bounds[hi])
        row, d = at[sl] - lo, disp[sl].clone().requires_grad_(path in ("step", "md", "host", "hessian"))
        args = (species[atom[sl]], row, hi - lo, species[sites[lo:hi]])
        if path == "cart":
            cart, soap = ex.jacobian(d, *args)
            cart = _with_self(row, cart, hi - lo)
            rows = torch.repeat_interleave(torch.arange(hi - lo, device=row.device),
                                           torch.bincount(row, minlength=hi - lo) + 1)
            firsts.append((weights[lo:hi][rows][:, None] @ cart)[:, 0])
            carts.append(cart)
            soaps.append(soap)
            continue
        soap = ex.soap(d, *args, differentiable=path == "hessian")
        soaps.append(soap.detach())
        if path == "hessian":
            blocks = []
            for v in range(case["n_vec"]):
                (g,) = torch.autograd.grad((soap * weights[lo:hi, v]).sum(), d, create_graph=True)
                blocks.append(torch.stack([-torch.autograd.grad(g[:, a].sum(), d, retain_graph=True)[0]
                                           for a in range(3)], 2))
            firsts.append(_with_self(row, torch.stack(blocks, 1), hi - lo))
        elif weights is not None:
            (g,) = torch.autograd.grad((soap * weights[lo:hi]).sum(), d)
            firsts.append(_with_self(row, g, hi - lo))
    soap = torch.cat(soaps)
    if path == "descriptor":
        return {"soap": soap}
    first = torch.cat(firsts)
    if path == "hessian":
        return {"hess": first}
    if path == "host":
        return {"soap": soap.T.cpu().numpy(), "pair": first.T.cpu().numpy()}
    if path == "cart":
        return {"soap": soap, "cart": torch.cat(carts), "pair": first}
    return {"soap": soap, "pair": first}
