"""Breadth-first levels of emg_dof_build_device at the widths and counts where
the way they are run changes: levels at and beside the widest that the
one-launch kernel takes, a narrow level after a wide one and the other way
round, and more levels than one launch runs.  Whole numbers, compared bit for
bit with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_numbering import device_map

pytestmark = pytest.mark.gpu


def fans(k):
    """Ring of k nodes with an axis edge on either side: from the first axis
    (nodes 0, 1) the levels hold 1, k + 1 and 2 nodes; a chain to a second ring
    of k nodes follows."""
    a = np.arange(k)
    b = (a + 1) % k
    ring = 2
    axis = ring + k
    ring2 = axis + 4
    one = np.stack([0 * a, 0 * a + 1, ring + a, ring + b], axis=1)
    two = np.stack([0 * a + axis, 0 * a + axis + 1, ring + a, ring + b], axis=1)
    link = np.array([[axis, axis + 1, axis + 2, axis + 3]])
    three = np.stack([0 * a + axis + 2, 0 * a + axis + 3, ring2 + a, ring2 + b], axis=1)
    return np.vstack([one, two, link, three]).astype(np.int32), ring2 + k


def compare(tets, n_nodes, seed):
    le = np.array([(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)])
    pairs = tets[:, le].reshape(-1, 2)
    some = pairs[np.random.default_rng(seed).permutation(len(pairs))[::5]].astype(np.int32)
    for d in (np.zeros((0, 2), np.int32), some):
        rc, l2g, ne, nf, nd = device_map(tets, n_nodes, d, O.GAUGE_REF)
        assert rc == 0
        o = O.dof_build(tets, d, gauge=O.GAUGE_REF)
        np.testing.assert_array_equal(l2g, o["l2g"])
        assert (ne, nf, nd) == (o["n_edges"], o["n_free"], o["n_dofs"])


@pytest.mark.parametrize("k", [3, 255, 2047, 8190, 8191, 8192, 20000])
def test_level_widths(k):
    compare(*fans(k), seed=k)


@pytest.mark.parametrize("n", [12287, 12300, 27000])
def test_level_counts(n):
    i = np.arange(n - 3)
    compare(np.stack([i, i + 1, i + 2, i + 3], axis=1).astype(np.int32), n, seed=n)
