"""The layer ordering of the direct solve, on CPU tensors built from the oracle's K_ff: a bijection that
keeps each node's rows together, with a band of one layer of nodes where the ordering by coordinates
has two, on meshes whose nodes are not in their planes, and never wider than that on others."""
import numpy as np
import pytest
import torch

import oracle as O


def _operator(X, el, fixed):
    from feab200.device import Pattern
    n_dof = 3 * len(X)
    free = O.free_dofs(n_dof, fixed)
    K = O.reduce_free(O.structural_csr(O.hex8_element_stiffness(X[el], O.D_solid3d(1.0, 0.3)), el, n_dof), free).tocsr()
    node = free // 3
    starts = np.flatnonzero(np.r_[True, node[1:] != node[:-1]])
    fm = -np.ones(n_dof, np.int32)
    fm[free] = np.arange(len(free), dtype=np.int32)

    class Op:
        pattern = Pattern(K.shape[0], K.nnz, len(starts), torch.as_tensor(K.indptr.astype(np.int32)),
                          torch.as_tensor(K.indices.astype(np.int32)),
                          torch.as_tensor(np.r_[starts, len(free)].astype(np.int32)), torch.as_tensor(fm))
        vals64 = torch.as_tensor(K.data)
        n = K.shape[0]

    return Op(), K, starts


def _band(K, iperm):
    C = K.tocoo()
    return int(np.abs(iperm[C.row].astype(np.int64) - iperm[C.col]).max())


@pytest.mark.parametrize("shape,size", [((16, 3, 2), (2.0, 0.4, 0.4)), ((5, 12, 4), (0.5, 3.0, 0.6)),
                                        ((4, 4, 9), (0.4, 0.4, 0.9)), ((7, 1, 1), (1.0, 0.1, 0.1)),
                                        ((1, 1, 1), (1.0, 1.0, 1.0)), ((3, 3, 3), (1.0, 1.0, 1.0))])
@pytest.mark.parametrize("moved", [False, True])
def test_layer_order(shape, size, moved):
    from feab200.direct import coordinate_order, dof_permutation, layer_order
    X, el = O.box_mesh(*size, *shape)
    rng = np.random.default_rng(5)
    if moved:
        X = X + 0.1 * np.asarray(size) / shape * (rng.random(X.shape) - 0.5)
        new = rng.permutation(len(X))                    # node numbers in no order
        Y = np.empty_like(X)
        Y[new] = X
        X, el = Y, new[el]
    fixed = rng.choice(3 * len(X), 3 * len(X) // 9, replace=False)     # nodes of 0 to 3 free DOFs
    op, K, starts = _operator(X, el, np.sort(fixed))
    order, layers = layer_order(op, X)
    assert sorted(order.tolist()) == list(range(len(starts)))
    iperm = dof_permutation(op, order).numpy()
    assert sorted(iperm.tolist()) == list(range(op.n))
    sizes = np.diff(np.r_[starts, op.n])
    for s, z in zip(starts, sizes):
        assert np.array_equal(iperm[s:s + z], iperm[s] + np.arange(z))
    axis = int(np.argmax(size))
    assert layers == shape[axis] + 1
    cross = np.prod([shape[a] + 1 for a in range(3) if a != axis])
    line = max(shape[a] + 1 for a in range(3) if a != axis)
    assert _band(K, iperm) <= 3 * (cross + line + 2) + 2            # the next layer's far neighbour
    by_coordinates = dof_permutation(op, coordinate_order(op, X)).numpy()
    assert _band(K, iperm) <= _band(K, by_coordinates) + 3 * line


def test_layer_order_on_graded_spacing_is_a_bijection():
    from feab200.direct import dof_permutation, layer_order
    X, el = O.box_mesh(1.0, 0.3, 0.3, 12, 3, 3)
    X[:, 0] = X[:, 0] ** 3 + 0.01 * X[:, 0]
    op, K, starts = _operator(X, el, O.fixed_dofs_on_plane(X, 0, 0.0))
    order, layers = layer_order(op, X)
    assert sorted(order.tolist()) == list(range(len(starts))) and layers >= 1
    assert sorted(dof_permutation(op, order).tolist()) == list(range(op.n))


@pytest.mark.parametrize("G", [1, 2, 2047, 2048, 2049, 2 ** 24 + 2, 20000004, 33554435, 79000001])
def test_sampled_nodes_are_nodes(G):
    from feab200.direct import _spread
    s = _spread(G, min(G, 2048), "cpu")
    assert len(s) == min(G, 2048) and int(s[0]) == 0 and int(s[-1]) == G - 1
    assert bool((s[1:] > s[:-1]).all())


def _chosen(X, el, fixed):
    """The band that the direct solve chooses, by its ordering, and the bands of the orderings that it had
    before the one in layers."""
    from feab200.direct import coordinate_order, dof_permutation, narrowest_order, node_order
    op, K, starts = _operator(X, el, fixed)
    iperm, bw, _ = narrowest_order(op, X, lambda ip: _band(K, ip.numpy()))
    assert bw == _band(K, iperm.numpy()) and sorted(iperm.tolist()) == list(range(op.n))
    return bw, [_band(K, dof_permutation(op, o).numpy()) for o in (coordinate_order(op, X), node_order(op))]


@pytest.mark.parametrize("shape,size", [((4, 48, 48), (2.0, 0.4, 0.4)), ((4, 60, 10), (2.0, 1.0, 0.4)),
                                        ((6, 24, 24), (2.0, 0.4, 0.4)), ((10, 30, 30), (2.0, 0.4, 0.4)),
                                        ((2, 2, 40), (2.0, 1.0, 0.4)), ((33, 9, 8), (2.0, 0.4, 0.4)),
                                        ((25, 25, 2), (2.0, 0.4, 0.4)), ((7, 1, 1), (1.0, 0.1, 0.1)),
                                        ((12, 12, 12), (1.0, 1.0, 1.0))])
def test_the_chosen_band_is_the_narrowest(shape, size):
    """Flat and stretched boxes among them: the longest axis is not always that of most layers."""
    X, el = O.box_mesh(*size, *shape)
    bw, others = _chosen(X, el, O.fixed_dofs_on_plane(X, 0, 0.0))
    assert bw <= min(others)


@pytest.mark.parametrize("kind", ["bent", "slit"])
def test_the_chosen_band_is_the_narrowest_on_other_meshes(kind):
    """Two legs side by side, and a plate that slits of one element's width make one long strip: the layers
    of the bounding box cross the strip many times, an order along it once."""
    nx, ny = (24, 20) if kind == "bent" else (40, 40)
    X, el = O.box_mesh(float(nx), float(ny), 1.0, nx, ny, 1)
    c = X[el].mean(axis=1)
    if kind == "bent":
        keep = (c[:, 0] > nx - 3) | (c[:, 1] < 3) | (c[:, 1] > ny - 3)
    else:
        leg = np.floor(c[:, 1]).astype(int)
        turn = np.where((leg // 8) % 2 == 0, c[:, 0] > nx - 7, c[:, 0] < 7)
        keep = (leg % 8 != 7) | turn
    el = el[keep]
    used = np.unique(el)
    new = np.full(len(X), -1)
    new[used] = np.arange(len(used))
    X, el = X[used], new[el]
    bw, others = _chosen(X, el, O.fixed_dofs_on_plane(X, 0, 0.0)[:30])
    assert bw <= min(others)
