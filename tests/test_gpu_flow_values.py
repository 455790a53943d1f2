"""A second set_flow with other attenuation values: the flows are those of a
handle that had these values from the start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_attenuation_values_set_again():
    import hipft_b200 as H
    nt, npp = 40, 82
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    br = 300.0 * np.random.default_rng(6).standard_normal((1, nt, npp + 1))
    br[..., -1] = br[..., 0]
    flow = dict(dr_model=1, mf_model=1, dr_p0=46.0, dr_p2=-262.0, dr_p4=-379.0, mf_p1=22.0, mf_p3=11.0, mf_p5=-28.0,
                attenuate=True)

    def step(values):
        with H.HipftGPU(t, p, 2, advance_flow=True, flow_num_method=4) as g:
            g.load_initial_map(br)
            for v in values:
                g.set_flow(attenuate_values=v, **flow)
                g.update_flow()
            g.advection_step(0.05)
            return g.get_field()

    a, b = np.array([500.0, 200.0]), np.array([50.0, 1000.0])
    once = step([b])
    assert not np.array_equal(once, step([a]))
    assert np.array_equal(once, step([a, b]))
