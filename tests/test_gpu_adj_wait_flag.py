"""A bounded wait that gave up reaches the caller of the adjoint call it
belongs to: hipft_adj_step, hipft_adj_record and hipft_adj_reverse (steps left
on the stack or not) return HIPFT_ETIMEOUT, and the handle computes the same
gradient afterwards as one that never saw the error.  The flag is set by a wait
that nothing completes (hipft_gpu_expire_wait).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT, NPP, NR, DT = 24, 48, 2, 3.0


class _Adjoint:
    def __init__(self):
        import torch
        import hipft_b200 as H
        self.torch = torch
        self.g = H.HipftGPU(np.linspace(0.0, np.pi, NT), np.linspace(0.0, 2.0 * np.pi, NPP + 1), NR,
                            advance_diffusion=True, diffusion_coef_constants=[300.0, 700.0])
        rng = np.random.default_rng(5)
        self.g.load_initial_map(rng.standard_normal((NR, NT, NPP + 1)))
        self.x = self.g.field_tensor().clone()
        cot = torch.zeros_like(self.x)
        cot[:, 1:-1, :NT] = torch.as_tensor(rng.standard_normal((NR, NPP, NT)))
        self.cot = cot
        self.fresh()

    def fresh(self):
        t = self.torch
        self.fbar, self.dacc = self.cot.clone(), t.zeros(NR, dtype=t.float64, device="cuda")
        self.gflow = t.zeros((5,) + tuple(self.x.shape), dtype=t.float64, device="cuda")
        t.cuda.synchronize()

    def call(self, name, expire=False):
        p = lambda v: ctypes.c_void_p(v.data_ptr())
        out = (p(self.fbar), p(self.dacc), p(self.gflow))
        L, h = self.g.L, self.g.h
        if expire:
            assert L.hipft_gpu_expire_wait(h, 64) == 0
        if name == "step":
            return L.hipft_adj_step(h, ctypes.c_double(DT), p(self.x), *out)
        if name == "record":
            return L.hipft_adj_record(h, ctypes.c_double(DT))
        return L.hipft_adj_reverse(h, *out)

    def recorded(self):
        n = ctypes.c_int64(0)
        assert self.g.L.hipft_adj_recorded(self.g.h, ctypes.byref(n), None) == 0
        return n.value

    def two_steps(self):
        self.fresh()
        assert self.g.L.hipft_gpu_set_field_device(self.g.h, ctypes.c_void_p(self.x.data_ptr())) == 0
        for name in ("record", "record", "reverse", "reverse"):
            assert self.call(name) == 0
        return self.fbar.cpu().numpy(), self.dacc.cpu().numpy()


@pytest.mark.parametrize("name", ["step", "record", "reverse_one_left", "reverse_last"])
def test_expired_wait_is_reported_by_the_adjoint_call(name):
    from hipft_b200 import gpu
    ref = _Adjoint().two_steps()
    a = _Adjoint()
    if name.startswith("reverse"):
        for _ in range(2 if name == "reverse_one_left" else 1):
            assert a.call("record") == 0
    before = a.recorded()
    assert a.call(name.split("_")[0], expire=True) == gpu.HIPFT_ETIMEOUT
    assert a.recorded() == before - (1 if name.startswith("reverse") else 0)
    assert a.g.L.hipft_adj_clear(a.g.h) == 0
    got = a.two_steps()
    assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])
