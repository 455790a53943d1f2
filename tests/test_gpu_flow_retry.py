"""2-D flow arrays after a call that ran out of device memory: update_flow fails
again while the memory is short, and once there is room it builds the flows and
steps as a handle that never failed.  The shortage is a torch tensor that takes
all but two or three of the four arrays; a handle beforehand loads the kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(nt, npp, nr):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    g = H.HipftGPU(t, p, nr, advance_flow=True, flow_num_method=4)
    br = np.random.default_rng(5).standard_normal((1, nt, npp + 1))
    br[..., -1] = br[..., 0]
    g.load_initial_map(br)
    half = 0.5 * (t[:-1] + t[1:])
    # vt on theta half points x phi, vp on theta x phi half points, m/s
    vt = 10.0 * np.sin(2.0 * np.concatenate([[0.0], half, [np.pi]]))[:, None] * np.cos(p)[None, :]
    vp = 20.0 * np.sin(t)[:, None] * np.sin(np.concatenate([p, [p[1] + 2.0 * np.pi]]))[None, :]
    g.set_flow()
    g.set_flow_from_files(vt, vp)
    return g


def test_update_flow_repeated_after_running_out_of_memory():
    import torch
    from hipft_b200 import gpu
    shape = (512, 1024, 32)  # 134 MB an array: none of them shares an allocation
    with _handle(*shape) as g:
        g.update_flow()
        dt = 0.5 * g.flow_dtmax()
        g.advection_step(dt)
        want = g.get_field()
        dev = g.field_tensor()
        array = dev.numel() * 8
        del dev
    with _handle(*shape) as g:
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - int(2.6 * array), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            assert g.L.hipft_gpu_update_flow(g.h, None) == gpu.HIPFT_ENOMEM
        del hog
        torch.cuda.empty_cache()
        assert g.update_flow()
        g.advection_step(dt)
        assert np.array_equal(g.get_field(), want)
