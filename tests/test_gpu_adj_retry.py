"""The reverse pass's work arrays after a call that ran out of device memory: the
same call fails again while the memory is short, and once there is room the
handle computes the gradient of one that never failed.  The shortage is a torch
tensor that takes all but two or three work fields of the free memory; a small
gradient beforehand loads the kernels."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Run:
    def __init__(self, nt, npp, nr):
        import torch
        import hipft_b200 as H
        self.torch = torch
        self.g = H.HipftGPU(np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1), nr,
                            advance_diffusion=True, diffusion_subcycles=1, diffusion_coef_constants=300.0)
        br = np.random.default_rng(2).standard_normal((1, nt, npp + 1))
        br[..., -1] = br[..., 0]
        self.g.load_initial_map(br)
        # a field's cotangent is its own copy: seam columns carry nothing
        self.fbar = self.g.field_tensor().clone()
        self.fbar[:, 0] = self.fbar[:, -1] = 0.0
        self.dacc = torch.zeros(nr, dtype=torch.float64, device="cuda")
        self.gflow = torch.zeros(1, dtype=torch.float64, device="cuda")  # no flow: not touched
        self.dt = 2.0 * self.g.info().dtime_diffusion_euler

    def record(self):
        return self.g.L.hipft_adj_record(self.g.h, ctypes.c_double(self.dt))

    def reverse(self):
        p = lambda v: ctypes.c_void_p(v.data_ptr())
        self.torch.cuda.synchronize()
        rc = self.g.L.hipft_adj_reverse(self.g.h, p(self.fbar), p(self.dacc), p(self.gflow))
        self.g.synchronize()
        return rc, self.fbar.cpu().numpy(), self.dacc.cpu().numpy()


def test_call_repeated_after_running_out_of_memory():
    import torch
    from hipft_b200 import gpu
    small = _Run(512, 1024, 1)
    assert small.record() == 0 and small.reverse()[0] == 0
    small.g.close()
    shape = (512, 1024, 32)  # 134 MB a field: one field per allocation
    good = _Run(*shape)
    assert good.record() == 0
    rc, f0, d0 = good.reverse()
    assert rc == 0
    good.g.close()
    run = _Run(*shape)
    field = run.fbar.numel() * 8
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - int(2.6 * field), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        assert run.record() == gpu.HIPFT_ENOMEM
    del hog
    torch.cuda.empty_cache()
    assert run.record() == 0
    rc, f1, d1 = run.reverse()
    assert rc == 0 and np.array_equal(f0, f1) and np.array_equal(d0, d1)
