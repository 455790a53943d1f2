"""Advection stages whose pole rows' blocks, or whose blocks per SM, follow from the
number of realizations: the realizations of a batch bit for bit as one alone.
WENO3: a block per pole row (fewer than 8 realizations) or one for both, and two
per row beyond 1024 columns; upwind: grids of up to 16 blocks per SM and larger."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WENO = [(20, 40, 8), (12, 130, 9), (33, 257, 8), (16, 1000, 8), (12, 1030, 8), (12, 1030, 17), (70, 66, 30)]
UPWIND = [(300, 500, 9), (64, 514, 40), (200, 1030, 5)]


@pytest.mark.parametrize("nt,npp,nr,method", [g + (4,) for g in WENO] + [g + (2,) for g in UPWIND])
def test_batch_equals_one_alone(nt, npp, nr, method):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    br = np.random.default_rng(8).standard_normal((1, nt, npp + 1))
    br[..., -1] = br[..., 0]
    out = []
    for n in (1, nr):
        with H.HipftGPU(t, p, n, advance_flow=True, flow_num_method=method) as g:
            g.load_initial_map(br)
            g.set_flow(dr_model=1, mf_model=1, dr_p0=46.0, dr_p2=-262.0, dr_p4=-379.0, mf_p1=22.0, mf_p3=11.0,
                       mf_p5=-28.0)
            g.update_flow()
            g.advection_step(0.5 * g.flow_dtmax())
            out.append(g.get_field())
    assert np.isfinite(out[0]).all() and all(np.array_equal(out[0][0], f) for f in out[1])
