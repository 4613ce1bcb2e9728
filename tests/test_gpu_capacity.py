"""Octrees that outgrow max_nodes, at whichever level: refused, and the handle goes on."""
import numpy as np
import pytest

import synthetic as syn

pytestmark = pytest.mark.gpu


def same(a, b):
    for x, y in ((a.vertices, b.vertices), (a.triangles, b.triangles), (a.colors, b.colors)):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("depth,chain", [(5, False), (7, True), (8, False)])
def test_node_capacity_runs_out_at_every_level(depth, chain):
    import psr
    big = syn.workload("torus_ellipsoid200k", n=60000)[:3]
    small = syn.workload("sphere20k", n=900, colour=True)[:3]
    caps = dict(max_depth=depth, max_points=60000, compute_colors=True, concurrent_stages=not chain,
                max_subdivision_nodes=2000000)
    with psr.PoissonReconstruction(max_nodes=1000000, **caps) as r:
        r.SolvePoissionReconstructionMesh(*big, depth=depth)
        counts = list(r.stats().level_count)[:depth + 1]
        want = r.SolvePoissionReconstructionMesh(*small, depth=3)
        fits = r.stats().nodes
    # the leaves do not fit; they do, and the first, second, .. level above them does not
    limits = [8, 72, counts[depth] // 2, counts[depth] - 8]
    limits += [sum(counts[d + 1:]) + counts[d] // 2 for d in range(depth - 1, 1, -1)] + [sum(counts) - 1]
    for nodes in limits:
        with psr.PoissonReconstruction(max_nodes=nodes, **caps) as r:
            for _ in range(2):
                with pytest.raises(psr.PsrError) as e:
                    r.SolvePoissionReconstructionMesh(*big, depth=depth)
                assert e.value.status == psr.PSR_OUT_OF_CAPACITY, nodes
                assert r.stats().points == 60000
            if nodes >= 2 * fits:
                same(want, r.SolvePoissionReconstructionMesh(*small, depth=3))
