"""Device inputs by every route of psr_submit: read in place, or staged where the kernels could not
read them as they are."""
import numpy as np
import pytest

import synthetic as syn

pytestmark = pytest.mark.gpu

VCAP, TCAP = 300000, 1000000


def outputs():
    import torch
    import psr
    v = torch.zeros((VCAP, 3), device="cuda")
    t = torch.zeros((TCAP, 3), dtype=torch.int32, device="cuda")
    return v, t, psr.PsrMesh(v.data_ptr(), t.data_ptr(), None, None, VCAP, TCAP, psr.PSR_DEVICE, 0, 0)


# byte offsets of the two float arrays: each alone off the boundary of a float, both, by 1 to 3 bytes
@pytest.mark.parametrize("ox,on", [(1, 0), (0, 2), (3, 1), (2, 2), (4, 8)])
def test_byte_shifted_device_inputs_equal_staged(ox, on):
    """A packed record uploaded as bytes: the floats need not sit on a 4-byte boundary."""
    import torch
    import psr
    p, nr, _, _ = syn.workload("torus_ellipsoid200k", n=3001)

    def shifted(a, by):
        raw = np.concatenate([np.zeros(by, np.uint8), np.ascontiguousarray(a).view(np.uint8).ravel()])
        flat = torch.from_numpy(raw).cuda()
        return flat, flat.data_ptr() + by

    with psr.PoissonReconstruction(max_depth=6, max_points=4000) as r:
        a = r.SolvePoissionReconstructionMesh(p, nr, depth=6)
        keep_x, x = shifted(p, ox)
        keep_n, n = shifted(nr, on)
        v, t, m = outputs()
        r.reconstruct_device(x, n, None, p.shape[0], depth=6, out=m)
        del keep_x, keep_n
        np.testing.assert_array_equal(v[:m.vertex_count].cpu().numpy(), a.vertices)
        np.testing.assert_array_equal(t[:m.triangle_count].cpu().numpy(), a.triangles)



def test_captured_submission_replays_its_own_inputs():
    """A caller's own capture of psr_submit (kernels issued one by one): a replay reconstructs the cloud
    that was captured, also after other clouds went through the handle."""
    import torch
    import psr
    clouds = []
    for n, seed in ((3001, 0), (2500, 1)):
        p, nr, _, _ = syn.workload("torus_ellipsoid200k", cloud=seed, n=n)
        clouds.append((torch.from_numpy(p).cuda(), torch.from_numpy(nr).cuda(), n))
    with psr.PoissonReconstruction(max_depth=6, max_points=4000, disable_graphs=True) as r:
        want = [r.SolvePoissionReconstructionMesh(x.cpu().numpy(), q.cpu().numpy(), depth=6) for x, q, _ in clouds]
        x, q, n = clouds[0]
        v, t, m = outputs()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            r.submit_device(x.data_ptr(), q.data_ptr(), None, n, m, depth=6, stream=stream.cuda_stream)
        with pytest.raises(psr.PsrError):   # its completion is the caller's to wait for
            r.wait()
        x, q, n = clouds[1]
        v1, t1, m1 = outputs()
        r.reconstruct_device(x.data_ptr(), q.data_ptr(), None, n, depth=6, out=m1)
        np.testing.assert_array_equal(v1[:m1.vertex_count].cpu().numpy(), want[1].vertices)
        graph.replay()
        torch.cuda.synchronize()
    nv, nt = len(want[0].vertices), len(want[0].triangles)
    np.testing.assert_array_equal(v[:nv].cpu().numpy(), want[0].vertices)
    np.testing.assert_array_equal(t[:nt].cpu().numpy(), want[0].triangles)
    assert not v[nv:].any() and not t[nt:].any()
