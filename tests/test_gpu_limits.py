"""The step limits whose reductions go block by block (32 x 32 cells): the
practical time step limit of the diffusion subcycles (k_ax, k_ptl), with the
largest |A f| placed at the edges of a block, of the last, ragged block and of
the seam, and the CFL limit (k_flow_dtmax).  A subcycle of another length gives
another field, far above the bar."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
GRIDS = [(31, 30), (33, 33), (34, 66), (65, 36), (66, 129)]
DIFF = [9000.0, 20000.0]


def _spiked(nt, npp, seed):
    rng = np.random.default_rng(seed)
    m = 3.0 * rng.standard_normal((nt, npp))
    rows = [r for r in (2, 31, 32, 33, nt - 3) if 1 < r < nt - 2]
    cols = [c for c in (1, 31, 32, 33, 34, npp - 2) if c < npp - 1]
    m[rows[seed % len(rows)], cols[(seed + 1) % len(cols)]] += 900.0
    m[:, -1] = m[:, 0]
    m[0], m[-1] = m[0, 0], m[-1, 0]
    return m


@pytest.mark.parametrize("grid_d", [False, True])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_subcycles_from_a_spike(nt, npp, grid_d):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp)
    for seed in range(5):
        m = np.stack([_spiked(nt, npp, seed), _spiked(nt, npp, seed + 3)])
        raw = dict(n_realizations=2, advance_diffusion=True, time_end=12.0, dt_max=12.0, diffusion_coef_constants=DIFF,
                   diffusion_coef_grid=grid_d)
        ref = [O.run(O.process_parameters(raw), map_pt=m, s1=p, s2=t)["f"]]
        if not grid_d:  # each realization alone
            ref.append(np.concatenate([O.run(O.process_parameters(dict(raw, n_realizations=1, diffusion_coef_constants=[d])),
                                             map_pt=m[i:i + 1], s1=p, s2=t)["f"] for i, d in enumerate(DIFF)]))
        for ragged, want in enumerate(ref):
            with H.HipftGPU(t, p, 2, advance_diffusion=True, diffusion_coef_constants=DIFF,
                            diffusion_coef_grid=grid_d) as g:
                g.load_initial_map(m)
                if ragged:
                    g.set_ragged(True)
                g.flux_transport_step(12.0)
                f = g.get_field()
            err = np.abs(f - want).max() / np.abs(want).max()
            assert err <= 1e-12, (seed, ragged, err)


@pytest.mark.parametrize("nt,npp", GRIDS)
def test_cfl_limit(nt, npp):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp)
    fl = dict(flow_dr_coef_p0_values=[10.0], flow_dr_coef_p2_values=[-337.43], flow_dr_coef_p4_values=[-253.07],
              flow_mf_coef_p1_values=[300.0], flow_mf_coef_p3_values=[-200.0], flow_mf_coef_p5_values=[30.0])
    raw = dict(n_realizations=1, advance_flow=True, flow_num_method=4, strang_splitting=True, flow_dr_model=1,
               flow_mf_model=1, time_end=1e4, dt_max=1e4, **fl)
    r = O.run(O.process_parameters(raw), map_pt=np.ones((1, nt, npp)), s1=p, s2=t, max_steps=1)
    with H.HipftGPU(t, p, 1, advance_flow=True, flow_num_method=4, strang_splitting=True) as g:
        g.load_initial_map(np.ones((1, nt, npp)))
        g.set_flow(dr_model=1, mf_model=1, dr_p0=10.0, dr_p2=-337.43, dr_p4=-253.07, mf_p1=300.0, mf_p3=-200.0,
                   mf_p5=30.0)
        g.update_flow()
        lim = g.flow_dtmax()
    assert abs(lim - r["num"][-1, 0, 2]) <= 4e-15 * lim
