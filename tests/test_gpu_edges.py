"""The kernels at the edges of their tiles and at the lines of their dispatch: sizes just below,
at and above a tile, every depth's solver, crowded and sparse clouds in the colour and normal
searches, inputs read in place and staged, and capacities that run out.  Everything is compared
bit for bit with the oracle's records and float mirror (test_gpu_parity, whose bound on the solved
values is used where values are compared) or with the same cloud by another route."""
import numpy as np
import pytest

import normals_oracle
import synthetic as syn
import test_gpu_parity as parity

pytestmark = pytest.mark.gpu

CAPS = dict(compute_colors=True, compute_normals=True)


# a sparse cloud's octree needs more nodes than the default of ten a sample
ROOM = dict(max_points=300000)


def same(a, b):
    for x, y in ((a.vertices, b.vertices), (a.triangles, b.triangles), (a.colors, b.colors), (a.normals, b.normals)):
        np.testing.assert_array_equal(x, y)


# 1, a block of 256, a sort tile of 2048 samples, each with its neighbours; the first solver modes
# (rows, one group a thread, several) come with the depths
@pytest.mark.parametrize("n,depth", [(255, 4), (256, 4), (257, 4), (2047, 5), (2048, 5), (2049, 5), (4097, 6)])
def test_tile_edges_against_oracle(oracle_mod, n, depth):
    import psr
    p, nr, rgb, _ = syn.workload("sphere20k", n=n, colour=True)
    with psr.PoissonReconstruction(max_depth=6, **ROOM, **CAPS) as r:
        parity.full_check_arrays(r, oracle_mod, p, nr, rgb, depth)


@pytest.mark.parametrize("name,cloud,n", [("superquadric2m", 0, 120000), ("mix", 0, 150000)])
def test_depth8_against_oracle(oracle_mod, name, cloud, n):
    """Depth 8: the whole-GPU solver, value rows, chunks of coarse divergence from depth 5 down.  The mesh
    is compared where the algorithm is defined (the oracle read no unset record)."""
    import psr
    p, nr, _, _ = syn.workload(name, cloud=cloud, n=n, colour=False)
    o = oracle_mod.Oracle()
    assert o.run(p, nr, None, depth=8, vert_cap=2000000, tri_cap=4000000) == 0
    with psr.PoissonReconstruction(max_depth=8, compute_normals=True, max_mesh_vertices=2000000,
                                   max_triangles=4000000, **ROOM) as r:
        mesh = r.SolvePoissionReconstructionMesh(p, nr, depth=8)
        parity.check_octree(r, o)
        x, iso = parity.check_field_and_solve(r, o)
        parity.check_geometry(r, o)
        defined = o.scalars()["ub_events"] == 0
        assert o.run_mesh32(x, iso) == 0
        np.testing.assert_array_equal(r.debug("vvalue", np.float32), o.get("vvalue32"))
        if defined:
            parity.check_mesh_mirror(r, o, mesh, x, iso)


# samples per colour cell: about 1 (coarser levels, the wide search), 20 and 300 a block (both sides of
# the line from which a block is searched from the inside), thousands
@pytest.mark.parametrize("n,depth", [(300, 5), (2000, 5), (20000, 5), (200000, 4)])
def test_colour_search_against_oracle(oracle_mod, n, depth):
    import psr
    p, nr, rgb, _ = syn.workload("torus_ellipsoid200k", n=n)
    with psr.PoissonReconstruction(max_depth=5, max_points=200000, **CAPS) as r:
        parity.full_check_arrays(r, oracle_mod, p, nr, rgb, depth)


@pytest.mark.parametrize("depth", [2, 3, 4, 5, 6, 7, 8])
def test_one_chain_equals_forked_stages(depth):
    """concurrent_stages off takes one launch for all depths of the solve (up to depth 7) and no
    forked streams; disable_graphs issues the same kernels directly."""
    import psr
    n = 60000 if depth > 6 else 4000
    p, nr, rgb, _ = syn.workload("torus_ellipsoid200k", n=n)
    out = []
    for options in (dict(), dict(concurrent_stages=False), dict(disable_graphs=True),
                    dict(concurrent_stages=False, cg_cluster_ctas=4)):
        with psr.PoissonReconstruction(max_depth=8, **ROOM, **CAPS, **options) as r:
            try:
                out.append(r.SolvePoissionReconstructionMesh(p, nr, rgb, depth=depth))
            except psr.PsrError as e:   # a cloud too sparse for its depth: refused by every route
                out.append(e.status)
    for m in out[1:]:
        if isinstance(out[0], int):
            assert out[0] == psr.PSR_INVALID_INPUT and m == out[0]
        else:
            assert len(m.triangles) > 0
            same(out[0], m)


@pytest.mark.parametrize("offset", [0, 1, 3])
def test_device_inputs_in_place_equal_staged(offset):
    """Device arrays are read where they are, whatever their alignment; host arrays are staged."""
    import torch
    import psr
    p, nr, rgb, _ = syn.workload("torus_ellipsoid200k", n=3001)
    dev = torch.device("cuda", 0)

    def shifted(a):
        flat = torch.from_numpy(np.concatenate([np.zeros(offset, a.dtype), a.ravel()])).to(dev)
        return flat[offset:]

    with psr.PoissonReconstruction(max_depth=6, max_points=4000, **CAPS) as r:
        a = r.SolvePoissionReconstructionMesh(p, nr, rgb, depth=6)
        x, q, c = shifted(p), shifted(nr), shifted(rgb)
        v = torch.empty((300000, 3), device=dev)
        t = torch.empty((1000000, 3), dtype=torch.int32, device=dev)
        cc, nn = torch.empty_like(v), torch.empty_like(v)
        m = psr.PsrMesh(v.data_ptr(), t.data_ptr(), cc.data_ptr(), nn.data_ptr(), 300000, 1000000, psr.PSR_DEVICE, 0, 0)
        r.reconstruct_device(x.data_ptr(), q.data_ptr(), c.data_ptr(), p.shape[0], depth=6, out=m)
        nv, nt = m.vertex_count, m.triangle_count
    np.testing.assert_array_equal(v[:nv].cpu().numpy(), a.vertices)
    np.testing.assert_array_equal(t[:nt].cpu().numpy(), a.triangles)
    np.testing.assert_array_equal(cc[:nv].cpu().numpy(), a.colors)
    np.testing.assert_array_equal(nn[:nv].cpu().numpy(), a.normals)


# spacings from far above to far below a cell of the finest level, and a crowd beside a sparse shell
@pytest.mark.parametrize("n,crowd", [(11, 0), (700, 0), (5000, 0), (3000, 3000)])
def test_normal_search_levels_against_oracle(n, crowd):
    import psr
    p, _, _, _ = syn.workload("sphere20k", n=n)
    if crowd:
        q, _, _, _ = syn.workload("sphere20k", cloud=1, n=crowd)
        p = np.concatenate([p, (q * np.float32(0.02) + p[0]).astype(np.float32)])
    with psr.PoissonReconstruction(max_depth=7, max_points=20000) as r:
        g = r.CalculatePointCloudNormal(p)
    o, cond = normals_oracle.estimate_normals(p)
    m = (cond["gap"] > 0.05) & ~cond["tie"] & (cond["cos"] > 1e-3)
    assert np.all(np.isfinite(g))
    dots = (g[m].astype(np.float64) * o[m]).sum(axis=1)
    assert dots.min() > 1.0 - 1e-4


@pytest.mark.parametrize("depth,cap", [(7, 1000), (7, 20000), (8, 60000)])
def test_subdivision_capacity_runs_out_and_recovers(depth, cap):
    """More subdivision candidates than the workspace holds is refused, wherever the levels stop, and
    the handle reconstructs the next cloud as a fresh one does."""
    import psr
    big = syn.workload("torus_ellipsoid200k", n=60000)
    small = syn.workload("sphere20k", n=3000, colour=True)
    caps = dict(max_depth=depth, **ROOM, **CAPS)
    with psr.PoissonReconstruction(**caps) as r:
        want = r.SolvePoissionReconstructionMesh(*small[:3], depth=4)
        fits = r.stats().subdivision_nodes <= cap
        r.SolvePoissionReconstructionMesh(*big[:3], depth=depth)
        assert r.stats().subdivision_nodes > cap
    with psr.PoissonReconstruction(max_subdivision_nodes=cap, **caps) as r:
        with pytest.raises(psr.PsrError) as e:
            r.SolvePoissionReconstructionMesh(*big[:3], depth=depth)
        assert e.value.status == psr.PSR_OUT_OF_CAPACITY
        if fits:
            same(want, r.SolvePoissionReconstructionMesh(*small[:3], depth=4))
        else:
            with pytest.raises(psr.PsrError) as e:
                r.SolvePoissionReconstructionMesh(*small[:3], depth=4)
            assert e.value.status == psr.PSR_OUT_OF_CAPACITY
