"""Node numberings other than a grid's row by row, for the tests of the sweeps."""
import numpy as np


def renumber(coords, conn, order):
    """The mesh with node order[k] renumbered to k."""
    inv = np.empty(len(order), np.int64)
    inv[np.asarray(order)] = np.arange(len(order))
    return np.ascontiguousarray(coords[order]), np.ascontiguousarray(inv[conn].astype(np.int32))


def boundary_first(coords, conn):
    from delfem_gb300 import meshgen as mg
    on = np.zeros(coords.shape[0], bool)
    on[mg.boundary_nodes(conn)] = True
    return np.concatenate([np.nonzero(on)[0], np.nonzero(~on)[0]])


def radial(coords, conn):
    return np.argsort(((coords - coords.mean(axis=0)) ** 2).sum(axis=1), kind="stable")


def rcm(coords, conn):
    """Reverse Cuthill-McKee: breadth first from a node of least degree, neighbours by degree."""
    n = coords.shape[0]
    k = conn.shape[1]
    pairs = np.unique(np.concatenate([conn[:, [i, j]] for i in range(k) for j in range(k) if i != j]), axis=0)
    ptr = np.searchsorted(pairs[:, 0], np.arange(n + 1))
    deg = np.diff(ptr)
    seen, order = np.zeros(n, bool), []
    for root in np.argsort(deg, kind="stable"):
        if seen[root]:
            continue
        seen[root] = True
        queue = [root]
        for q in queue:
            order.append(q)
            nb = pairs[ptr[q]:ptr[q + 1], 1]
            nb = nb[~seen[nb]]
            seen[nb] = True
            queue.extend(nb[np.argsort(deg[nb], kind="stable")])
    return np.array(order[::-1])
