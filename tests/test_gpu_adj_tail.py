"""A pass of two reverse RKG2 stages whose last chunk owns one to three phi
columns: its loop takes whole turns of four columns, so some slots of the ring
in shared memory are read that the chunk never fetched.  Nothing of them may
reach the D gradient: the gradient has the same bits whether those slots hold
whatever was there or NaN, left by a diffusion step of a NaN field that fills
the shared memory of every SM between the recorded step and its reverse.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stages", [3, 7])
@pytest.mark.parametrize("npp", [181, 182, 183, 184])
def test_unfetched_columns_stay_out_of_the_gradient(npp, stages):
    import torch
    import hipft_b200 as H

    nt, nr = 30, 2
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())
    kw = dict(advance_diffusion=True, diffusion_num_method=3, diffusion_subcycles=1)
    rng = np.random.default_rng(npp + stages)
    x = rng.standard_normal((nr, npp + 2, nt))
    x[:, :, 0], x[:, :, -1] = x[:, :1, 0], x[:, :1, -1]
    x[:, 0], x[:, -1] = x[:, -2], x[:, 1]
    theta, phi = lambda n: np.linspace(0.0, np.pi, n), lambda n: np.linspace(0.0, 2.0 * np.pi, n + 1)
    with H.HipftGPU(theta(nt), phi(npp), nr, diffusion_coef_constants=[300.0, 700.0], **kw) as g, \
            H.HipftGPU(theta(512), phi(1024), 8, diffusion_coef_constants=300.0, **kw) as nan:
        # s = ceil((sqrt(25 + 24 r) - 3) / 2) for r = dt / dt_euler, half a stage below the wanted (odd) count
        dt = ((2.0 * (stages - 0.5) + 3.0) ** 2 - 25.0) / 24.0 * g.info().dtime_diffusion_euler
        nan.set_field(np.full((8, 1026, 512), np.nan))
        g.set_field(x)
        ldt = g.info().ldt
        cot = torch.zeros((nr, npp + 2, ldt), dtype=torch.float64, device="cuda")
        cot[:, 1:-1, :nt] = torch.as_tensor(rng.standard_normal((nr, npp, nt)))

        def gradient(poison):
            g.set_field(x)
            fbar, dacc = cot.clone(), torch.zeros(nr, dtype=torch.float64, device="cuda")
            gflow = torch.zeros((5,) + tuple(cot.shape), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            g._ck(g.L.hipft_adj_record(g.h, dt), "hipft_adj_record")
            g.synchronize()
            assert g.info().sts_s == stages
            if poison:
                nan.diffusion_step(nan.info().dtime_diffusion_euler)
                nan.synchronize()
            g._ck(g.L.hipft_adj_reverse(g.h, ptr(fbar), ptr(dacc), ptr(gflow)), "hipft_adj_reverse")
            g.synchronize()
            return fbar[:, :, :nt].cpu().numpy(), dacc.cpu().numpy()

        f0, d0 = gradient(False)
        for _ in range(3):
            f1, d1 = gradient(True)
            assert np.isfinite(f1).all() and np.array_equal(f0, f1)
            assert np.isfinite(d1).all() and np.array_equal(d0, d1), (d0, d1)
