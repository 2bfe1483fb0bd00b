"""What the mixed path's arithmetic has to give bit for bit, whatever instantiation
or CTA size a call takes: equalities of IEEE arithmetic, so there is no tolerance
beyond the roundings that each test counts."""
import numpy as np
import pytest

from soap_turbo_b200 import synthetic as syn
from soap_turbo_b200.context import Context
from test_gpu_size_rules import edge_sites

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
