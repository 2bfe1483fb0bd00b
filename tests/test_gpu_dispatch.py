"""Forms of the kernels that a definition's sizes pick, against the oracle: the items
per thread of the FP64 site kernel, the wide instantiation of the site kernels with
rows of several chunks, and the workspaces that only some forms use.

Tolerances: the gates of conftest."""
import numpy as np
import pytest
import torch

import oracle as O
from conftest import FP64_TOL, SOAP_TOL, VJP_TOL, max_rel_err, site_rel_err
from soap_turbo_b200 import _lib
from soap_turbo_b200 import synthetic as syn
from soap_turbo_b200.context import Context
from test_gpu_size_rules import edge_sites, repeated

pytestmark = pytest.mark.gpu

# species, alpha, l_max: (species, four radial indices, k) items of 256 threads
ITEMS = {1: ([8, 8], 8), 2: ([8, 8, 8], 8), 3: ([5] * 6, 8), 4: ([10, 10, 10], 12), 5: ([8] * 8, 10)}


@pytest.mark.parametrize("items", list(ITEMS))
def test_fp64_site_kernel_at_each_number_of_items(items):
    alpha, l_max = ITEMS[items]
    per_thread = -(-sum((a + 3) // 4 for a in alpha) * (l_max + 1) * (l_max + 2) // 2 // 256)
    assert per_thread == items
    hp = syn.Hyper(alpha_max=alpha, l_max=l_max, basis="poly3", compress_mode="trivial")
    base = edge_sites([1, 2, 33, 70], hp.n_species, seed=3)
    ctx = Context(hp)
    W, S = ctx.basis()
    ref = O.get_soap(hp, base, W, S).soap
    nl, site, _ = repeated(base, 9)
    soap = ctx.descriptor_fp64(ctx.batch(nl))[0].cpu().numpy()
    ctx.check_inputs()
    ok = np.abs(ref).max(axis=1)[site] > 0
    assert site_rel_err(soap[ok], ref[site][ok]) <= FP64_TOL


def test_soap_cart_der_takes_no_workspace_of_another_form():
    """An uncompressed definition of 2700 components is beyond the form that shares a
    site among CTAs: its call does not take that form's (n_sites, split, 3 n_soap) sums."""
    hp = syn.Hyper(alpha_max=[8, 8, 8], basis="poly3")
    nl, _, _ = repeated(edge_sites([2], 3, seed=1), 445)  # a count that the form splits
    ctx = Context(hp)
    b = ctx.batch(nl)
    soap = torch.empty(b.n_sites, ctx.n_soap, dtype=torch.float64, device="cuda")
    cart = torch.empty(b.n_pairs, ctx.n_soap, 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _lib.check(ctx._lib.soapb_descriptor_fp64(ctx._h, b.c, soap.data_ptr(), cart.data_ptr()))
    torch.cuda.synchronize()
    k_max, pairs, sites = 45, b.n_pairs + 1, b.n_sites + 1
    need = (2 * 8 * 24 + 4 * 16 * k_max) * pairs + (16 * 24 * k_max + 8 * ctx.n_soap) * sites
    # each of some twenty buffers is rounded up to the allocator's 2 MB
    assert free - torch.cuda.mem_get_info()[0] <= need + 20 * 2 ** 21


def test_hessian_forms_the_pairs_once_per_call():
    """17 weight vectors are two launches of the Hessian kernel, and one more launch
    than one vector: the pairs' second derivatives and records serve both."""
    hp = syn.Hyper(alpha_max=[4, 4], l_max=4, basis="poly3gauss")
    base = edge_sites([2, 33, 60], 2, seed=29)
    ctx = Context(hp, legacy_filter_seed=False)
    b = ctx.batch(base)
    count = []
    for n_vec in (1, 17):
        before = ctx.launch_count
        ctx.central_hessian(b, torch.ones(base.n_sites, n_vec, ctx.n_soap, dtype=torch.float64, device="cuda"))
        count.append(ctx.launch_count - before)
    assert count[1] == count[0] + 1


@pytest.mark.parametrize("alpha,l_max", [([4, 4], 4), ([10], 12)])
def test_hessian_bits_do_not_depend_on_the_batch(alpha, l_max):
    """The site count picks 256 or 512 threads per site (l_max 12: always 512); every
    sum keeps its order.  (Against the oracle: test_gpu_hessian and test_gpu_size_rules;
    alpha 10 is beyond their gate, W's conditioning amplifies the radial expansion's
    last bits to 4.5e-7.)"""
    hp = syn.Hyper(alpha_max=alpha, l_max=l_max, basis="poly3gauss" if l_max == 4 else "poly3")
    base = edge_sites([2, 33, 60], hp.n_species, seed=37)
    ctx = Context(hp, legacy_filter_seed=False)
    vecs = np.random.default_rng(5).standard_normal((base.n_sites, 2, ctx.n_soap))
    first = None
    for n_sites in (3, 148, 149, 296, 297, 444, 445):
        nl, site, pair = repeated(base, n_sites)
        v = torch.as_tensor(np.ascontiguousarray(vecs[site])).cuda()
        got = ctx.central_hessian(ctx.batch(nl), v).cpu().numpy()
        first = got if first is None else first
        np.testing.assert_array_equal(got, first[pair])
    assert np.isfinite(first).all() and np.abs(first).max() > 0


@pytest.mark.parametrize("threads", [0, 64, 256])
@pytest.mark.parametrize("n_sites", [1, 6, 297, 1185])
def test_wide_instantiation_over_rows_of_several_chunks(n_sites, threads):
    """alpha above 8 and l_max above 8: two groups of radial indices, of which the second
    species' last is partly past its alpha, three warps of k, H read from shared memory.
    The first site's row is several chunks long, so that a batch of one has one too."""
    hp = syn.Hyper(alpha_max=[10, 7], l_max=10, basis="poly3gauss", compress_mode="trivial")
    base = edge_sites([290, 64, 129, 256, 33, 1], 2, seed=47)
    ctx = Context(hp)
    ctx.set_threads_per_site(threads)
    W, S = ctx.basis()
    ref = O.get_soap(hp, base, W, S, do_derivatives=True)
    G = np.random.default_rng(8).standard_normal((ctx.n_soap, base.n_sites))
    pref = ref.contract(G, 1.0)
    nl, site, pair = repeated(base, n_sites)
    b = ctx.batch(nl)
    soap = ctx.descriptor(b)
    force = ctx.contract(b, soap, torch.as_tensor(np.ascontiguousarray(G[:, site])).cuda()).cpu().numpy()
    ctx.check_inputs()
    ok = np.abs(ref.soap).max(axis=1)[site] > 0
    assert ok.any()
    assert site_rel_err(soap.cpu().numpy()[ok], ref.soap[site][ok]) <= SOAP_TOL
    assert max_rel_err(force, pref[pair]) <= VJP_TOL
