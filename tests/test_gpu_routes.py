"""The same cloud by every route, with a mesh at the end of each; the whole-GPU solver at the lines of
its own dispatch."""
import numpy as np
import pytest

import synthetic as syn
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu


def same(a, b):
    for x, y in ((a.vertices, b.vertices), (a.triangles, b.triangles), (a.colors, b.colors), (a.normals, b.normals)):
        np.testing.assert_array_equal(x, y)


ROUTES = (dict(), dict(concurrent_stages=False), dict(disable_graphs=True),
          dict(concurrent_stages=False, disable_graphs=True), dict(concurrent_stages=False, cg_cluster_ctas=4))


# clouds dense enough for their depth: every route returns the mesh
@pytest.mark.parametrize("name,n,depth", [("sphere20k", 600, 2), ("sphere20k", 2000, 3), ("sphere20k", 6000, 4),
                                         ("torus_ellipsoid200k", 30000, 5), ("torus_ellipsoid200k", 80000, 6),
                                         ("torus_ellipsoid200k", 200000, 7), ("mix", 150000, 8)])
def test_routes_return_the_same_mesh(name, n, depth):
    import psr
    p, nr, rgb, _ = syn.workload(name, n=n, colour=True)
    caps = dict(max_depth=8, max_points=200000, compute_colors=True, compute_normals=True, max_mesh_vertices=1000000,
                max_triangles=2000000, max_subdivision_nodes=4000000)
    want = None
    for options in ROUTES:
        with psr.PoissonReconstruction(**caps, **options) as r:
            m = r.SolvePoissionReconstructionMesh(p, nr, rgb, depth=depth)
        assert len(m.triangles) > 0
        want = want or m
        same(want, m)


def test_routes_refuse_the_same_cloud():
    """A cloud too sparse for its depth is refused by every route, with the same status."""
    import psr
    p, nr, rgb, _ = syn.workload("torus_ellipsoid200k", n=300)
    statuses = set()
    for options in ROUTES:
        with psr.PoissonReconstruction(max_depth=8, max_points=20000, **options) as r:
            with pytest.raises(psr.PsrError) as e:
                r.SolvePoissionReconstructionMesh(p, nr, depth=8)
            statuses.add(e.value.status)
    assert len(statuses) == 1 and statuses <= {psr.PSR_INVALID_INPUT, psr.PSR_OUT_OF_CAPACITY}


@pytest.mark.parametrize("name,cloud,n", [("mix", 0, 150000), ("sphere20k", 0, 100000)])
def test_depth8_mesh_against_oracle(oracle_mod, name, cloud, n):
    """Depth 8 to the mesh.  (Roots of a second coarse depth make the oracle note the reference's stale
    offsets, for which it takes the intended ones as the GPU does.)"""
    import psr
    p, nr, _, _ = syn.workload(name, cloud=cloud, n=n, colour=False)
    o = oracle_mod.Oracle()
    assert o.run(p, nr, None, depth=8, vert_cap=2000000, tri_cap=4000000) == 0
    with psr.PoissonReconstruction(max_depth=8, max_points=150000, max_mesh_vertices=2000000, max_triangles=4000000) as r:
        mesh = r.SolvePoissionReconstructionMesh(p, nr, depth=8)
        assert len(mesh.triangles) > 100000
        x, iso = parity.check_field_and_solve(r, o)
        parity.check_mesh_mirror(r, o, mesh, x, iso)


def test_whole_gpu_solver_of_a_large_batch_equals_alone():
    """Depth 9, two clouds: units of more than 32 virtual blocks (their totals go round by one record) and
    more than 6 passes of virtual blocks a block (A p of the others in global memory)."""
    import psr
    clouds = [syn.workload("superquadric2m", cloud=k, n=n, colour=False)[:2] for k, n in ((0, 1500000), (1, 1300000))]
    caps = dict(max_depth=9, max_points=1500000, laplacian_epsilon=0.0, max_mesh_vertices=4000000,
                max_triangles=8000000, max_subdivision_nodes=12000000)
    ref = []
    with psr.PoissonReconstruction(**caps) as r:
        for p, nr in clouds:
            m = r.SolvePoissionReconstructionMesh(p, nr, depth=9)
            ref.append((m, r.stats()))
    counts = [list(st.level_count) for _, st in ref]
    assert min(c[d] for c in counts for d in (8, 9)) // 2048 > 32
    assert sum(sum(c[5:]) for c in counts) // 2048 > 147 * 2 * 6
    with psr.PoissonReconstruction(batch_clouds=2, **caps) as r:
        got = r.reconstruct_batch([(p, nr, None) for p, nr in clouds], depth=9)
        for k, (m, st) in enumerate(ref):
            status, b = r.batch_result(k)
            assert status == psr.PSR_OK
            assert list(b.cg_iterations) == list(st.cg_iterations) and list(b.cg_residual) == list(st.cg_residual)
            np.testing.assert_array_equal(got[k].vertices, m.vertices)
            np.testing.assert_array_equal(got[k].triangles, m.triangles)
