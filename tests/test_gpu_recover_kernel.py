"""The recovery's element kernel on element counts around its lanes and blocks, on strongly distorted elements
and on mirrored ones (negative Jacobian), for each choice of outputs, against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 16, 17, 33])
@pytest.mark.parametrize("mirrored", [False, True])
def test_element_kernel(n, mirrored):
    from feab200.device import DeviceMesh
    nodes, el = O.box_mesh(0.1 * n, 0.13, 0.11, n, 1, 1)
    X = nodes + 0.02 * (np.random.default_rng(n).random(nodes.shape) - 0.5)
    if mirrored:
        X = X * np.array([1.0, 1.0, -1.0])
    D = O.D_solid3d(3.0, 0.31)
    u = np.random.default_rng(n + 50).standard_normal(3 * len(X))
    dm = DeviceMesh(X, el)
    s_nodes, s_elem = O.recover(X, el, u, D)
    e_nodes, e_elem = O.recover(X, el, u)
    # sums of some 30 terms each with conditioning of the distorted Jacobian (below 10)
    tol = 2e-14
    both = dm.recover(u, D, nodal=True, elements=True, von_mises=True)
    for key, want in (("nodal", s_nodes), ("elements", s_elem), ("nodal_vm", O.von_mises(s_nodes)),
                      ("elements_vm", O.von_mises(s_elem))):
        assert _rel(both[key].cpu().numpy(), want) < tol, key
    assert _rel(dm.recover(u, D, nodal=False, elements=True)["elements"].cpu().numpy(), s_elem) < tol
    assert _rel(dm.recover(u, nodal=False, elements=True)["elements"].cpu().numpy(), e_elem) < tol
    assert _rel(dm.recover(u)["nodal"].cpu().numpy(), e_nodes) < tol
