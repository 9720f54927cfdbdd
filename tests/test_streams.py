"""Calls on one scene handle from several streams: each gives the results of the
same call alone, and a device call of 8,192 rays or more has finished when it
returns."""
import numpy as np
import pytest

from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu

N = (6000, 16384, 64)


@pytest.fixture(scope="module")
def tetra(built):
    import torch
    sc = api.Scene(scenes.scene_tetra_spheres(), config=C.default_config(coarse_grid_n=17, newton_tol=1e-12))
    work = []
    for k, n in enumerate(N):
        o, d = (np.ascontiguousarray(a[:n]) for a in scenes.cone_rays(n, 40 + k, 5.0, 3.0, 10.0))
        to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
        out = _outputs(n)
        sc.trace_device(to.data_ptr(), td.data_ptr(), n, 200, {k: t.data_ptr() for k, t in out.items()})
        torch.cuda.synchronize()
        work.append((o, d, to, td, {k: t.cpu().numpy() for k, t in out.items()}))
    return sc, work


def _outputs(n):
    import torch
    return {"status": torch.full((n,), -9, dtype=torch.int32, device="cuda"),
            "bounce_count": torch.full((n,), -9, dtype=torch.int32, device="cuda"),
            "end_point": torch.full((n, 3), -9.0, dtype=torch.float64, device="cuda")}


# pairs of (size of the first call, size of the second): both in flight, one
# waited for, and a host-array call on the scene's own stream after a device call
@pytest.mark.parametrize("first,second", [(0, 0), (0, 1), (1, 0), (1, 1), (0, 2), (1, 2)])
def test_back_to_back_calls_on_two_streams(tetra, first, second):
    import torch
    sc, work = tetra
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(10):
        outs = [_outputs(N[first]), _outputs(N[second])]
        torch.cuda.synchronize()
        for which, st, out in zip((first, second), streams, outs):
            o, d, to, td, _ = work[which]
            if which == 2:
                host = sc.trace(o, d, 200, outputs=tuple(out))
            else:
                sc.trace_device(to.data_ptr(), td.data_ptr(), N[which], 200, {k: t.data_ptr() for k, t in out.items()},
                                stream=st.cuda_stream)
        torch.cuda.synchronize()
        for which, out in zip((first, second), outs):
            for k, ref in work[which][4].items():
                got = host[k] if which == 2 else out[k].cpu().numpy()
                assert np.array_equal(got, ref), (which, k)


@pytest.mark.parametrize("n", [8192, 16384])
def test_device_call_of_wavefront_size_has_finished_when_it_returns(tetra, n):
    import torch
    sc, work = tetra
    _, _, to, td, ref = work[1]
    out, st = _outputs(n), torch.cuda.Stream()
    torch.cuda.synchronize()
    sc.trace_device(to.data_ptr(), td.data_ptr(), n, 200, {k: t.data_ptr() for k, t in out.items()}, stream=st.cuda_stream)
    assert st.query()
    for k in out:
        assert np.array_equal(out[k].cpu().numpy(), ref[k][:n]), k


def test_captured_call_replays_beside_other_calls(tetra):
    """A small device call captured on a stream: the capture neither waits for
    the call in flight before it nor leaves anything behind that a call outside
    could wait for.  A call that waits for its trace is refused in a capture."""
    import torch
    sc, work = tetra
    _, _, to, td, ref = work[0]
    pre, cap, post = _outputs(N[0]), _outputs(N[0]), _outputs(N[0])
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def call(out, stream):
        sc.trace_device(to.data_ptr(), td.data_ptr(), N[0], 200, {k: t.data_ptr() for k, t in out.items()}, stream=stream)

    torch.cuda.synchronize()
    call(pre, st.cuda_stream)
    with torch.cuda.graph(g, stream=st):
        with pytest.raises(RuntimeError, match="capture"):
            sc.trace_device(work[1][2].data_ptr(), work[1][3].data_ptr(), N[1], 200, {},
                            stream=torch.cuda.current_stream().cuda_stream)
        call(cap, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    call(post, st.cuda_stream)
    torch.cuda.synchronize()
    for out in (pre, cap, post):
        for k in out:
            assert np.array_equal(out[k].cpu().numpy(), ref[k]), k
