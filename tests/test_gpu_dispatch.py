"""Forms of the kernels that a definition's sizes pick, against the oracle: the items
per thread of the FP64 site kernel, the wide instantiation of the site kernels with
rows of several chunks, and the workspaces that only some forms use.

Tolerances: the gates of conftest."""
import numpy as np
import pytest
import torch

import oracle as O
from conftest import FP64_TOL, SOAP_TOL, VJP_TOL, max_rel_err, site_rel_err
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
