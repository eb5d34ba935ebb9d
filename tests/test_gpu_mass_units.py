"""Mass assembly where its column units can go wrong: every number of nodes per
element, elements that hold a node twice, nodes of as many elements as a warp
orders and of one more, nodes of none.  Against the oracle, which sums
duplicates in the same order: FP64 sums of at most a few hundred terms."""
import numpy as np
import pytest
import torch

import oracle
from feelmri_b200 import ops

pytestmark = pytest.mark.gpu


def _check(elems, n_nodes, nb, dtype, seed=0):
    rng = np.random.default_rng(seed)
    nodes = rng.uniform(-1.0, 1.0, (n_nodes, 3)).astype(dtype)
    qw = rng.uniform(0.1, 1.0, 3).astype(dtype)
    tab = rng.uniform(0.1, 1.0, (3, 4, nb)).astype(dtype)
    indptr, indices, data = oracle.mass_csc(elems, nodes, qw, tab)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = (up(elems), up(nodes), up(qw), up(tab))
    p, i, d = (t.cpu().numpy() for t in ops.mass_assemble(*args))
    np.testing.assert_array_equal(p, indptr)
    np.testing.assert_array_equal(i, indices)
    if nb >= 3:  # else the Jacobian's rank is below 3 and its determinant is rounding alone
        eps = 1e-12 if dtype == np.float64 else 1e-5
        np.testing.assert_allclose(d, data, rtol=0, atol=eps * np.abs(data).max())
    lump = np.array([np.add.reduce([], dtype=dtype) for _ in range(n_nodes)])
    for c in range(n_nodes):
        for k in range(p[c], p[c + 1]):
            lump[c] = lump[c] + d[k]
    np.testing.assert_array_equal(ops.mass_lumped(*args).cpu().numpy(), lump)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nb", range(1, 11))
def test_element_sizes(cuda, nb, dtype):
    rng = np.random.default_rng(nb)
    elems = rng.integers(0, 60, (90, nb)).astype(np.int32)  # nodes repeat within elements
    elems[elems == 7] = 8                                   # a node of no element
    _check(elems, 64, nb, dtype)


@pytest.mark.parametrize("nb,most", [(4, 64), (8, 64), (10, 51)])
@pytest.mark.parametrize("more", [0, 1, 300])
def test_many_elements_around_a_node(cuda, nb, most, more):
    rng = np.random.default_rng(3)
    elems = np.stack([rng.permutation(np.arange(1, 500))[:nb] for _ in range(most + more)]).astype(np.int32)
    elems[:, 1] = 0
    _check(elems, 501, nb, np.float64)
