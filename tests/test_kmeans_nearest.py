"""The assignment of points to centroids inside the ranking product.  On small
whole numbers every rank is exact (the low halves of the split are zero and all
sums fit 24 bits), so the assignment equals the first minimum of the integer
distances: ties go to the smaller index within a block of 32 columns, across
blocks, across the two halves of a 256-column tile and across tiles; row and
column remainders and rows of one warp or of a block are covered by the sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k", [(1, 8, 1), (129, 3, 7), (1000, 64, 33), (777, 13, 255), (640, 256, 256),
                                     (2000, 5, 300), (2001, 260, 1025), (1500, 16, 1024)])
def test_ties_go_to_the_first(n, dim, k):
    from erq_b200.clustering import kmeans_step

    rng = np.random.default_rng(n + dim + k)
    x = rng.integers(-2, 3, (n, dim)).astype(np.float32)
    c = rng.integers(-2, 3, (k, dim)).astype(np.float32)
    c[rng.integers(0, k, k // 2)] = c[rng.integers(0, k, k // 2)]  # equal centroids
    _, assign, counts = kmeans_step(x, c, seed=1)
    d = (c * c).sum(1)[None] - 2 * x @ c.T  # small whole numbers: exact
    want = d.argmin(1)
    assert (assign == want).all()
    assert (counts == np.bincount(want, minlength=k)).all()
