"""Reverse RKG2 stages in passes of four and two (k_adj_march, k_adj_poles) at
the sizes where their division of the field can go wrong: the smallest grid they
take (12 rows), the edges of their strips (64 rows held, 52 owned), few
columns, several blocks per pole, the wide blocks; all stages on the tape and
stage checkpoints of 6, which leave a pass of two.

Diffusion alone is linear in the field, so <g, F(x)> = <F^T g, x>: both sides are
sums of about a thousand rounded operations per term on nt npp terms, far below
1e-11 of sum |g||F(x)|.  The gradient with respect to D against a central
difference of relative step 1e-4, whose error is of the order 1e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOW0 = {k: np.zeros(2) for k in ("p0", "p2", "p4", "p1", "p3", "p5")}
GRIDS = [(12, 20), (13, 6), (64, 60), (65, 61), (67, 30), (117, 70), (120, 64), (24, 250), (20, 1000), (14, 2300)]


def _handle(nt, npp, D):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    g = H.HipftGPU(t, p, 2, advance_flow=True, flow_num_method=4, strang_splitting=True, advance_diffusion=True,
                   diffusion_num_method=3, diffusion_subcycles=1, diffusion_coef_constants=D)
    g.set_flow(dr_model=1, mf_model=1)
    return g


@pytest.mark.parametrize("spacing", [0, 6])
@pytest.mark.parametrize("stages", [9, 15])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_transpose_and_diffusivity(nt, npp, stages, spacing):
    from hipft_b200.adjoint import MisfitAdjoint, fold_cotangent
    D = np.array([300.0, 700.0])
    with _handle(nt, npp, D) as g:
        dte = g.info().dtime_diffusion_euler
    # s = ceil((sqrt(25 + 24 r) - 3) / 2) for r = dt / dt_euler, half a stage below the wanted (odd) count
    r = ((2.0 * (stages - 0.5) + 3.0) ** 2 - 25.0) / 24.0
    dt = r * dte
    rng = np.random.default_rng(nt * npp + stages)
    x = rng.standard_normal((2, npp + 2, nt))
    x[:, :, 0], x[:, :, -1] = x[:, :1, 0], x[:, :1, -1]  # one value at a pole
    x[:, 0], x[:, -1] = x[:, -2], x[:, 1]
    gb = rng.standard_normal(x.shape)

    def forward(Dd):
        with _handle(nt, npp, Dd) as h:
            return MisfitAdjoint(h, Dd, FLOW0).forward(x, [dt, dt])

    with _handle(nt, npp, D) as g:
        if spacing:
            g._ck(g.L.hipft_adj_set_tape_limit(g.h, 0, spacing), "hipft_adj_set_tape_limit")
        A = MisfitAdjoint(g, D, FLOW0)
        F = A.forward(x, [dt, dt])
        assert g.info().sts_s == stages
        gr = A.backward(fold_cotangent(gb))
    lhs, rhs = (gb * F).sum(axis=(1, 2)), (gr["f0"] * x).sum(axis=(1, 2))
    assert np.all(np.abs(lhs - rhs) <= 1e-11 * np.abs(gb * F).sum(axis=(1, 2))), (lhs, rhs)
    # the schedule follows the largest D, which is left alone
    e = 1e-4 * D[0]
    up, dn = forward(D + [e, 0.0]), forward(D - [e, 0.0])
    fd = (gb[0] * (up[0] - dn[0])).sum() / (2.0 * e)
    scale = np.sqrt(((gb[0] ** 2).sum()) * (((up[0] - dn[0]) / (2.0 * e)) ** 2).sum())
    assert abs(gr["D"][0] - fd) <= 1e-6 * scale, (gr["D"][0], fd, scale)
