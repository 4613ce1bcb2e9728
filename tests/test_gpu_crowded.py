"""Searches in crowded blocks: below, about and far above the counts at which their kernels change
over, against the oracle."""
import numpy as np
import pytest

import normals_oracle
import synthetic as syn

pytestmark = pytest.mark.gpu


def normalised(p):
    """The float coordinates that the search and the fit see: the bounding box enlarged 1.25 times around
    its middle, mapped to the unit cube.  Their rounding alone turns a normal of a crowd this small by up
    to 0.06 (0.998 in the cosine)."""
    f = np.float32
    hi, lo = p.max(0), p.min(0)
    edge = f((hi - lo).max() * f(1.25))
    return ((p - ((hi + lo) / f(2) - edge / f(2))) / edge).astype(f)


# points in a ball narrower than a level-7 cell beside a sparse shell: the 27 finest cells around them
# hold that many, on both sides of the coarser levels' cap of 1024
@pytest.mark.parametrize("crowd", [900, 1024, 1100, 6000])
def test_normals_of_a_crowd(crowd):
    import psr
    p, _, _, _ = syn.workload("sphere20k", n=2000)
    q, _, _, _ = syn.workload("sphere20k", cloud=1, n=crowd)
    p = np.concatenate([p, (q * np.float32(0.004) + p[0]).astype(np.float32)])
    with psr.PoissonReconstruction(max_depth=7, max_points=20000) as r:
        g = r.CalculatePointCloudNormal(p)
    o, cond = normals_oracle.estimate_normals(normalised(p))
    m = (cond["gap"] > 0.05) & ~cond["tie"]
    assert m.sum() > 1000 and np.all(np.isfinite(g))
    dots = np.abs((g[m].astype(np.float64) * o[m]).sum(axis=1))
    assert dots.min() > 1.0 - 1e-4
