"""The solvers on systems off the ordinary: rows whose neighbour table does not name them, and every
way of dealing a system's rows to the GPU."""
import numpy as np
import pytest

import synthetic as syn
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu


def sheet_cloud(seed):
    """A sphere and a tilted sheet that reaches into the low corner of the box, so that the first nodes of
    some depths get a parent that is not theirs (mesh/BuildOctree.cu:392-488)."""
    rng = np.random.default_rng(seed)
    p, nr, _, _ = syn.workload("sphere20k", cloud=seed, n=6000)
    k, ax = 3000, seed % 3
    s = rng.uniform(-1, 1, (k, 3))
    tilt = rng.uniform(-1, 1)
    s[:, ax] = -0.6 + 0.5 * (s[:, (ax + 1) % 3] + s[:, (ax + 2) % 3]) * tilt + 0.003 * rng.standard_normal(k)
    return (np.concatenate([p, s.astype(np.float32)]),
            np.concatenate([nr, np.tile(np.eye(3, dtype=np.float32)[ax], (k, 1))]))


@pytest.mark.parametrize("seed,depth", [(75, 6), (89, 6)])
@pytest.mark.parametrize("graphs", [True, False])
def test_rows_outside_their_own_table_against_oracle(oracle_mod, seed, depth, graphs):
    """The first eight rows of `depth` carry a right-hand side and are not in their own neighbour rows:
    after a few iterations (such a system need not converge) their solution is the oracle's, as every
    other row's.  The mesh of such a cloud is undefined."""
    import psr
    p, nr = sheet_cloud(seed)
    o = oracle_mod.Oracle()
    assert o.run(p, nr, None, depth=8, cg_iters=8, stop_after=3) == 0
    b = int(o.get("base")[depth])
    M = o.scalars()["M"]
    assert o.get("neighs").reshape(M, 27)[b, 13] != b and np.abs(o.get("div")[b:b + 8]).max() > 0
    with psr.PoissonReconstruction(max_depth=8, max_points=300000, disable_graphs=not graphs) as r:
        with pytest.raises(psr.PsrError) as e:
            r.SolvePoissionReconstructionMesh(p, nr, depth=8, cg_iterations=8)
        assert e.value.status == psr.PSR_INVALID_INPUT
        x = r.debug("x", np.float32)
    ref = o.get("x")
    assert parity.rel_l2(x, ref) <= parity.REL_L2
    assert parity.rel_l2(x[b:b + 8], ref[b:b + 8]) <= parity.REL_L2
