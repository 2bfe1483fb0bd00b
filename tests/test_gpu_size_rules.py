"""Both sides of every rule that picks a kernel, a CTA size or a split by the sizes
of a call, against the oracle: sites of each edge length (a warp's pairs, a chunk,
several chunks), repeated to site counts on either side of each line.

Tolerances: the gates of conftest.  The rules change which thread adds what, not
the precision of any term, so every form is held to the gates of its path."""
import numpy as np
import pytest
import torch

import oracle as O
from conftest import FP64_TOL, SOAP_TOL, VJP_TOL, max_rel_err, site_rel_err
from soap_turbo_b200 import synthetic as syn
from soap_turbo_b200.context import Context
from test_gpu_edge import make_nl
from test_gpu_neighbors import built, compare

pytestmark = pytest.mark.gpu


def edge_sites(n_pairs, n_species, seed):
    """Sites of the given numbers of pairs (the self pair included), a fifth of
    the neighbours carrying two species."""
    rng = np.random.default_rng(seed)
    sites = []
    for n in n_pairs:
        neigh = []
        for _ in range(n - 1):
            bits = 1 << int(rng.integers(0, n_species))
            if rng.random() < 0.2:
                bits |= 1 << int(rng.integers(0, n_species))
            neigh.append((float(rng.uniform(0.9, 5.3)), float(np.arccos(rng.uniform(-1, 1))),
                          float(rng.uniform(-np.pi, np.pi)), bits))
        sites.append((int(rng.integers(0, n_species)), neigh))
    return make_nl(sites, n_species)


def repeated(nl, n_sites):
    """nl's sites over and over, n_sites of them; and the site and pair of nl that
    each is a copy of."""
    site = np.arange(n_sites) % nl.n_sites
    first = np.concatenate([[0], np.cumsum(nl.n_neigh)])
    pair = np.concatenate([np.arange(first[i], first[i + 1]) for i in site])
    return syn.NeighbourList(
        n_sites=n_sites, n_neigh=nl.n_neigh[site], rjs=nl.rjs[pair], thetas=nl.thetas[pair], phis=nl.phis[pair],
        mask=np.ascontiguousarray(nl.mask[:, pair]), species=nl.species[site],
        species_multiplicity=nl.species_multiplicity[site], site_atom=np.arange(n_sites),
        neigh_atom=nl.neigh_atom[pair], disp=nl.disp[pair]), site, pair


MIXED = {
    "3sp_l8": syn.Hyper(alpha_max=[8, 8, 8], basis="poly3gauss", compress_mode="trivial"),
    "2sp_l4": syn.Hyper(alpha_max=[5, 4], l_max=4, basis="poly3"),  # every k in one warp
}


@pytest.mark.parametrize("n_sites", [1, 296, 297, 592, 593, 1185, 2048, 2049, 4095, 4096])
@pytest.mark.parametrize("name", list(MIXED))
def test_mixed_path_at_the_lines_of_its_rules(name, n_sites):
    hp = MIXED[name]
    base = edge_sites([1, 32, 33, 64, 65, 128, 129, 256, 290], hp.n_species, seed=17)
    ctx = Context(hp)
    W, S = ctx.basis()
    ref = O.get_soap(hp, base, W, S, do_derivatives=True)
    G = np.random.default_rng(7).standard_normal((ctx.n_soap, base.n_sites))
    pref = ref.contract(G, 1.0)
    nl, site, pair = repeated(base, n_sites)
    b = ctx.batch(nl)
    # the descriptor alone: with the rows' parts for the derivatives left out
    alone = ctx.descriptor(b, keep=False).cpu().numpy()
    soap = ctx.descriptor(b)
    force = ctx.contract(b, soap, torch.as_tensor(np.ascontiguousarray(G[:, site])).cuda()).cpu().numpy()
    ctx.check_inputs()
    ok = np.abs(ref.soap).max(axis=1)[site] > 0
    for s in (alone, soap.cpu().numpy()):
        if ok.any():
            assert site_rel_err(s[ok], ref.soap[site][ok]) <= SOAP_TOL
        assert np.abs(s[~ok]).max(initial=0.0) == 0.0
    if np.abs(pref[pair]).max() > 0:
        assert max_rel_err(force, pref[pair]) <= VJP_TOL
    else:
        assert np.abs(force).max() == 0.0


@pytest.mark.parametrize("l_max", [0, 2, 4, 5, 7, 8, 9, 12])
@pytest.mark.parametrize("basis", ["poly3", "poly3operator"])
def test_pair_rows_of_every_length(l_max, basis):
    """The last piece of a row's parts is full, or has one to three values over;
    the last warp of pairs is full or has one."""
    hp = syn.Hyper(alpha_max=[4, 3], l_max=l_max, basis=basis)
    ctx = Context(hp)
    W, S = ctx.basis()
    for n_pairs in ([32, 96], [64, 65]):
        nl = edge_sites(n_pairs, 2, seed=l_max)
        ref = O.get_soap(hp, nl, W, S, do_derivatives=True)
        G = np.random.default_rng(l_max).standard_normal((ctx.n_soap, nl.n_sites))
        b = ctx.batch(nl)
        assert site_rel_err(ctx.descriptor(b, keep=False).cpu().numpy(), ref.soap) <= SOAP_TOL
        soap = ctx.descriptor(b)
        assert site_rel_err(soap.cpu().numpy(), ref.soap) <= SOAP_TOL
        force = ctx.contract(b, soap, torch.as_tensor(G).cuda()).cpu().numpy()
        assert max_rel_err(force, ref.contract(G, 1.0)) <= VJP_TOL


FP64 = {
    "one_item": syn.Hyper(alpha_max=[4, 3], l_max=4, basis="poly3"),  # uncompressed: an identity map
    "two_items": syn.Hyper(alpha_max=[8, 8], l_max=8, basis="poly3", compress_mode="trivial"),
    "spread_map": syn.Hyper(alpha_max=[4, 4, 4], l_max=4, basis="poly3gauss", compress_mode="1_1"),
    "wide": syn.Hyper(alpha_max=[8, 8, 8], l_max=8, basis="poly3gauss"),
}


@pytest.mark.parametrize("name,n_sites", [
    ("one_item", 3), ("one_item", 98), ("one_item", 148), ("one_item", 296), ("one_item", 297), ("one_item", 592),
    ("two_items", 98), ("two_items", 148), ("two_items", 296), ("spread_map", 98), ("wide", 7)])
def test_fp64_path_at_the_lines_of_its_rules(name, n_sites):
    hp = FP64[name]
    base = edge_sites([1, 2, 31, 32, 33, 65, 130], hp.n_species, seed=23)
    ctx = Context(hp)
    W, S = ctx.basis()
    ref = O.get_soap(hp, base, W, S, do_derivatives=True, cart_der=True)
    G = np.random.default_rng(9).standard_normal((ctx.n_soap, base.n_sites))
    pref = ref.contract(G, 1.0)
    nl, site, pair = repeated(base, n_sites)
    b = ctx.batch(nl)
    soap, cart = ctx.descriptor_fp64(b, cart=True)
    force = ctx.contract_cart_der(b, cart, torch.as_tensor(np.ascontiguousarray(G[:, site])).cuda())
    ctx.check_inputs()
    ok = np.abs(ref.soap).max(axis=1)[site] > 0
    assert site_rel_err(soap.cpu().numpy()[ok], ref.soap[site][ok]) <= FP64_TOL
    want = torch.as_tensor(ref.soap_cart_der).cuda()
    scale = want.abs().max().item()
    assert (cart - want[torch.as_tensor(pair).cuda()]).abs().max().item() <= FP64_TOL * scale
    assert max_rel_err(force.cpu().numpy(), pref[pair]) <= FP64_TOL


@pytest.mark.parametrize("n_sites,n_vec", [(4, 1), (296, 3), (297, 3), (5, 16), (5, 17)])
def test_hessian_at_the_lines_of_its_rules(n_sites, n_vec):
    hp = syn.Hyper(alpha_max=[4, 4], l_max=4, basis="poly3gauss", atom_sigma_t_scaling=0.05,
                   atom_sigma_r_scaling=0.05)
    base = edge_sites([2, 33, 257, 290], 2, seed=29)
    ctx = Context(hp, legacy_filter_seed=False)
    W, S = ctx.basis()
    ref = O.get_soap(hp, base, W, S, do_derivatives=True, legacy_filter_seed=False, hessian=True)
    vecs = np.random.default_rng(3).standard_normal((base.n_sites, n_vec, ctx.n_soap))
    want, err = ref.central_hessian(vecs)
    assert err < 1e-10
    nl, site, pair = repeated(base, n_sites)
    got = ctx.central_hessian(ctx.batch(nl), torch.as_tensor(np.ascontiguousarray(vecs[site])).cuda())
    ctx.check_inputs()
    assert max_rel_err(got.cpu().numpy(), want[pair]) <= FP64_TOL


def lattice_atoms(n_atoms, side, spacing, n_sites, seed):
    """n_atoms of a jittered cubic lattice of side^3 points; the first n_sites of
    them are of species 0, the others of species 1."""
    rng = np.random.default_rng(seed)
    at = rng.permutation(side ** 3)[:n_atoms]
    pos = np.stack([at // side ** 2, at // side % side, at % side], -1) * spacing
    pos = pos + rng.uniform(0.0, 0.3 * spacing, pos.shape)
    return syn.Structure(pos, side * spacing, (np.arange(n_atoms) >= n_sites).astype(np.int32))


def test_neighbour_list_at_the_lines_of_its_rules():
    """One context for every size: buffers that hold the call before, and buffers
    that have to grow.  About 65 atoms lie within 5 A at a spacing of 2 A."""
    ctx = Context(syn.Hyper(alpha_max=[4, 4], l_max=4, basis="poly3"))
    for n_atoms, side, spacing, n_sites in [(343, 7, 2.0, 343), (8192, 21, 2.0, 4096), (8193, 21, 2.0, 4097),
                                            (8192, 21, 2.0, 8192), (600, 23, 5.0, 600), (343, 7, 2.0, 5),
                                            (2744, 14, 1.9, 1), (4096, 16, 2.0, 1036), (4096, 16, 2.0, 1037),
                                            (4096, 16, 2.0, 2072), (4096, 16, 2.0, 2073), (4096, 16, 2.0, 2664),
                                            (4096, 16, 2.0, 2665)]:
        st = lattice_atoms(n_atoms, side, spacing, n_sites, seed=n_atoms + n_sites)
        nl = syn.neighbour_list(st, 5.0, 2, central_species=0)
        _, a = built(ctx, st.positions, np.eye(3) * st.box, st.species + 1, nl.site_atom)
        compare(a, nl)
