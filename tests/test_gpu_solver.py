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


def solution(r):
    st = r.stats()
    return (r.debug("x", np.float32), st.iso_value, list(st.cg_iterations), list(st.cg_residual),
            list(st.cg_true_residual), list(st.cg_restarts))


def equal(a, b):
    np.testing.assert_array_equal(a[0], b[0])
    assert a[1:] == b[1:]


# systems that give a row, a group and several groups to a thread, and systems that outgrow the shared
# memory of the smaller clusters
@pytest.mark.parametrize("name,cloud,n,depth", [("sphere20k", 0, 4000, 5), ("mix", 1, 40000, 6), ("mix", 2, 60000, 7),
                                               ("torus_ellipsoid200k", 0, 150000, 7), ("serve", 3, 300000, 7)])
def test_solution_does_not_depend_on_the_cluster_size(name, cloud, n, depth):
    """Every sum of the CG is the same however its rows are dealt to CTAs and threads: iterations,
    residuals (as doubles) and solutions are equal bit for bit for every cluster size, from the global-memory
    path, in one chain, and in a batch."""
    import psr
    p, nr, _, _ = syn.workload(name, cloud=cloud, n=n, colour=False)
    caps = dict(max_depth=7, max_points=300000)
    with psr.PoissonReconstruction(**caps) as r:
        r.SolvePoissionReconstructionMesh(p, nr, depth=depth)
        want = solution(r)
    for options in (dict(cg_cluster_ctas=1, cg_cluster_ctas_fine=1), dict(cg_cluster_ctas=2, cg_cluster_ctas_fine=4),
                    dict(cg_cluster_ctas=5, cg_cluster_ctas_fine=3), dict(cg_cluster_ctas=8, cg_cluster_ctas_fine=16),
                    dict(concurrent_stages=False), dict(concurrent_stages=False, cg_cluster_ctas=3),
                    dict(disable_graphs=True)):
        with psr.PoissonReconstruction(**caps, **options) as r:
            r.SolvePoissionReconstructionMesh(p, nr, depth=depth)
            equal(want, solution(r))
    count = 5   # enough that the launch takes its smaller clusters
    with psr.PoissonReconstruction(batch_clouds=count, max_mesh_vertices=200000, max_triangles=400000, **caps) as r:
        r.reconstruct_batch([(p, nr, None)] * count, depth=depth)
        for k in (0, count - 1):
            status, st = r.batch_result(k)
            assert status == psr.PSR_OK
            assert want[1:] == (st.iso_value, list(st.cg_iterations), list(st.cg_residual), list(st.cg_true_residual),
                                list(st.cg_restarts))


def test_systems_that_fill_their_box_against_oracle(oracle_mod):
    """Samples throughout a box: depths 5 to 7 hold 20,000 to several 100,000 rows, which leave the pairs
    alone in shared memory (depth 5 on the one CTA of the chain, 6 on small clusters) or nothing (7)."""
    import psr
    rng = np.random.default_rng(7)
    p = rng.uniform(-1, 1, (120000, 3)).astype(np.float32)
    nr = (p / np.linalg.norm(p, axis=1, keepdims=True)).astype(np.float32)
    o = oracle_mod.Oracle()
    assert o.run(p, nr, None, depth=7, stop_after=3) == 0
    ref, base = o.get("x"), o.get("base")
    want = None
    for options in (dict(), dict(concurrent_stages=False), dict(cg_cluster_ctas=8, cg_cluster_ctas_fine=6),
                    dict(cg_cluster_ctas=16, cg_cluster_ctas_fine=1)):
        with psr.PoissonReconstruction(max_depth=7, max_points=120000, max_nodes=2000000, **options) as r:
            try:
                r.SolvePoissionReconstructionMesh(p, nr, depth=7)
            except psr.PsrError as e:   # whether the reference's algorithm can mesh it is not the question
                assert e.status == psr.PSR_INVALID_INPUT
            got = solution(r)
            counts = list(r.stats().level_count)
        assert counts[5] // 8 > 1791 and counts[6] // 8 > 6 * 1791 and counts[7] > 200000
        if want is None:
            want = got
            for d in (5, 6, 7):
                s = slice(int(base[d]), int(base[d]) + counts[d])
                assert parity.rel_l2(got[0][s], ref[s]) <= parity.REL_L2
        equal(want, got)
