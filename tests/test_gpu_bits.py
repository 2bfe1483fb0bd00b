"""What the mixed path's arithmetic has to give bit for bit, whatever instantiation
or CTA size a call takes: equalities of IEEE arithmetic, so there is no tolerance
beyond the roundings that each test counts."""
from fractions import Fraction

import numpy as np
import pytest
import torch

from soap_turbo_b200 import synthetic as syn
from soap_turbo_b200.context import Context
from test_gpu_size_rules import edge_sites, repeated

pytestmark = pytest.mark.gpu


def components(alpha, l_max):
    """(n, n', l) of every component of the trivial compression (of every one, with one species)."""
    first = {sum(alpha[:s]) for s in range(len(alpha))}
    n_max = sum(alpha)
    return [(n, m, l) for n in range(n_max) for m in range(n, n_max) for l in range(l_max + 1)
            if len(alpha) == 1 or n in first or m in first]


@pytest.mark.parametrize("tables", [True, False])
@pytest.mark.parametrize("sigma_scaling", [0.0, 0.05])
@pytest.mark.parametrize("basis", ["poly3", "poly3gauss", "poly3operator"])
@pytest.mark.parametrize("alpha", [[8], [8, 8, 8]])
def test_the_pair_kernels_instantiations_expand_a_pair_alike(alpha, basis, sigma_scaling, tables):
    """l_max 8 and 9 take the two instantiations of the kernels.  Their radial
    expansions are one source, rounded to FP32, so the components of l <= 8 differ by
    the norm alone: two quotients of a product s / |p| each, three roundings."""
    base = edge_sites([40, 60, 80, 100] * 60, len(alpha), seed=11)
    soap = []
    for l_max in (8, 9):
        ctx = Context(syn.Hyper(alpha_max=alpha, l_max=l_max, basis=basis, atom_sigma_r_scaling=sigma_scaling,
                                atom_sigma_t_scaling=sigma_scaling,
                                compress_mode="trivial" if len(alpha) > 1 else "None"))
        ctx.set_radial_tables(tables)
        soap.append(ctx.descriptor(ctx.batch(base)).cpu().numpy())
    at = {c: i for i, c in enumerate(components(alpha, 9))}
    a, b = soap[0], soap[1][:, [at[c] for c in components(alpha, 8)]]
    np.testing.assert_array_equal(a == 0.0, b == 0.0)
    ratio = np.where(a == 0.0, np.nan, a / np.where(b == 0.0, 1.0, b))
    spread = np.nanmax(ratio, axis=1) / np.nanmin(ratio, axis=1) - 1.0
    assert spread.max() <= 2 * 3 * 2.0 ** -53 * 1.01


def slot_sum(terms, slots, fma=False):
    """The documented order: slot v adds its terms v, v + slots, .. to zero, the lanes
    of 32 slots are added by xor shuffles of 16, 8, .., 1 and the 32-slot sums by those
    of 16, .., 1 over lanes of which the rest hold zero.  terms: (n, ...) floats to add,
    or with fma (a, b) pairs of numbers whose products are added with one rounding."""
    n = len(terms)
    if fma:
        acc = [0.0] * slots
        for i, (a, b) in enumerate(terms):
            acc[i % slots] = float(Fraction(a) * Fraction(b) + Fraction(acc[i % slots]))
        acc = np.array(acc)
    else:
        terms = np.asarray(terms)
        acc = np.zeros((slots,) + terms.shape[1:])
        for lo in range(0, n, slots):
            acc[:min(slots, n - lo)] += terms[lo:lo + slots]

    def tree(v):
        for o in (16, 8, 4, 2, 1):
            v = v + v[np.arange(32) ^ o]
        return v[0]
    part = np.zeros((32,) + acc.shape[1:])
    for w in range(slots // 32):
        part[w] = tree(acc[32 * w:32 * w + 32])
    return tree(part)


def float32_row(row):
    """The FP32 components s whose products with one FP64 factor are the row: found from
    the largest one, whose significand is searched."""
    top = np.abs(row).argmax()
    m = np.arange(2 ** 23, 2 ** 24, dtype=np.float64)
    for o in np.argsort(-np.abs(row))[1:]:
        if len(m) <= 1 or row[o] == 0.0:
            break
        s = row[o] / row[top] * m
        m = m[np.abs(s - s.astype(np.float32)) <= 1e-14 * np.abs(s)]
    assert len(m) == 1
    return (row / row[top] * m[0]).astype(np.float32)


DEFS = {"3sp": syn.Hyper(alpha_max=[8, 8, 8], basis="poly3gauss", compress_mode="trivial"),  # 621 components
        "1sp": syn.Hyper(alpha_max=[8], basis="poly3"),                                      # 324
        "wide": syn.Hyper(alpha_max=[10], l_max=12, basis="poly3")}                          # 715


@pytest.mark.parametrize("threads", [0, 64, 256])
@pytest.mark.parametrize("name", list(DEFS))
def test_fp64_sums_in_their_documented_order(name, threads):
    """The norm, q . G and the central pair's force are sums over 128 slots (over the
    chosen threads per site): bit for bit what that order gives."""
    hp = DEFS[name]
    slots = threads or 128
    base = edge_sites([30, 40, 50, 60, 70, 128, 129, 260, 300], hp.n_species, seed=5)
    ctx = Context(hp)
    ctx.set_threads_per_site(threads)
    b = ctx.batch(base)
    soap_d = ctx.descriptor(b)
    soap = soap_d.cpu().numpy()
    for row in soap[:3]:
        s = float32_row(row).astype(np.float64)
        norm = np.sqrt(slot_sum(s * s, slots))  # (a square of an FP32 value is exact: its fused sum is this one)
        np.testing.assert_array_equal(row, s * (1.0 / norm))
    # with G = q the forces are those of q (1 - q . G): zero exactly where the rounded q . G is one
    force = ctx.contract(b, soap_d, soap_d.t().contiguous()).cpu().numpy()
    first = np.concatenate([[0], np.cumsum(base.n_neigh)])
    for i, q in enumerate(soap):
        qg = slot_sum([(x, x) for x in q.tolist()], slots, fma=True)
        row = force[first[i]:first[i + 1]]
        assert (np.abs(row).max() == 0.0) == (qg == 1.0)
    G = torch.as_tensor(np.random.default_rng(2).standard_normal((ctx.n_soap, base.n_sites))).cuda()
    force = ctx.contract(b, soap_d, G).cpu().numpy()
    for i in range(base.n_sites):
        row = force[first[i]:first[i + 1]].copy()
        self_force, row[0] = row[0].copy(), 0.0
        np.testing.assert_array_equal(self_force, slot_sum(-row, slots))


@pytest.mark.parametrize("name", list(DEFS))
def test_a_sites_bits_do_not_depend_on_the_batch(name):
    """The launchers give a site other CTA sizes, splits and orders by the number of
    sites; its descriptor and forces stay the same bits."""
    hp = DEFS[name]
    base = edge_sites([1, 2, 33, 64, 65, 100, 128, 129, 290], hp.n_species, seed=31)
    ctx = Context(hp)
    G = np.random.default_rng(4).standard_normal((ctx.n_soap, base.n_sites))
    want = None
    for n_sites in (base.n_sites, 300, 700, 1500, 2500, 5000):
        nl, site, pair = repeated(base, n_sites)
        b = ctx.batch(nl)
        soap = ctx.descriptor(b)
        force = ctx.contract(b, soap, torch.as_tensor(np.ascontiguousarray(G[:, site])).cuda())
        got = soap.cpu().numpy(), force.cpu().numpy()
        want = want or got
        np.testing.assert_array_equal(got[0], want[0][site])
        np.testing.assert_array_equal(got[1], want[1][pair])


LONG = {"8sp_a4": syn.Hyper(alpha_max=[4] * 8, l_max=8, basis="poly3gauss", compress_mode="trivial"),
        "5sp_a6": syn.Hyper(alpha_max=[6, 5, 6, 4, 6], l_max=6, basis="poly3", compress_mode="trivial"),
        "3sp_a8": syn.Hyper(alpha_max=[8, 8, 8], l_max=8, basis="poly3gauss", compress_mode="trivial")}


@pytest.mark.parametrize("threads", [0, 64, 256])
@pytest.mark.parametrize("name", list(LONG))
def test_groups_of_warps_give_the_same_sums(name, threads):
    """Batches whose rows are several chunks on average give every species its own
    warps, or some at a time, by the number of sites: each site's bits are those of a
    batch of short rows, which the sites' species take in turn."""
    hp = LONG[name]
    base = edge_sites([64, 129, 256, 257, 300, 600], hp.n_species, seed=41)
    ctx = Context(hp)
    ctx.set_threads_per_site(threads)
    short = edge_sites([1], hp.n_species, seed=1)
    mixed = syn.concatenate([base] + [short] * 400)  # under a chunk on average
    want = ctx.descriptor(ctx.batch(mixed)).cpu().numpy()[:base.n_sites]
    for n_sites in (base.n_sites, 148, 149, 444, 445):
        nl, site, _ = repeated(base, n_sites)
        np.testing.assert_array_equal(ctx.descriptor(ctx.batch(nl)).cpu().numpy(), want[site])


@pytest.mark.parametrize("name", ["3sp", "wide"])
def test_the_autotuner_changes_no_bits(name):
    """It times the contract's CTA sizes, which share their sums' slots, and leaves the
    descriptor's chunks as they are; a batch of another size takes the rule again."""
    hp = DEFS[name]
    base = edge_sites([64, 129, 256, 257, 300], hp.n_species, seed=43)
    ctx = Context(hp)
    ctx.set_tensor_cores(False)
    G = np.random.default_rng(6).standard_normal((ctx.n_soap, base.n_sites))

    def both(n_sites):
        nl, site, _ = repeated(base, n_sites)
        b = ctx.batch(nl)
        soap = ctx.descriptor(b)
        force = ctx.contract(b, soap, torch.as_tensor(np.ascontiguousarray(G[:, site])).cuda())
        return b, soap, force
    before = {n: both(n)[1:] for n in (5, 700)}
    for tuned in (5, 700, 200, 5):
        ctx.autotune(both(tuned)[0])
        for n, (soap, force) in before.items():
            _, s, f = both(n)
            assert torch.equal(s, soap) and torch.equal(f, force)
