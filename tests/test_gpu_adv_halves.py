"""WENO3 stage with two chunks per warp (32 rows each), which batches take where
that is less work than one chunk of 64 rows: strips with one row over and one
short, an odd number of chunks (the last warp's second one is past the end) and
short last chunks, 1-D flows and attenuated ones, which are 2-D, and fields whose
faces take the IEEE division (smoothness above 2^100).  The realizations of a
batch bit for bit as one alone (a chunk per warp)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows: 12 and 29 (28 owned by one strip), 30 (two strips: one chunk per warp),
# 62 and 85 (three strips of 28 for two of 60), 86, 122
GRIDS = [(12, 201, 200), (5, 65, 700), (29, 61, 400), (29, 130, 250), (30, 61, 400), (62, 131, 120), (64, 128, 100),
         (85, 97, 150), (86, 97, 150), (122, 75, 120), (29, 260, 90), (20, 40, 100), (12, 200, 60), (64, 33, 8)]


@pytest.mark.parametrize("attenuate,scale", [(False, 100.0), (True, 100.0), (False, 1e22)])
@pytest.mark.parametrize("method", [3, 4])
@pytest.mark.parametrize("nt,npp,nr", GRIDS)
def test_batch_equals_one_alone(nt, npp, nr, method, attenuate, scale):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    br = scale * np.random.default_rng(8).standard_normal((1, nt, npp + 1))
    br[..., -1] = br[..., 0]
    out = []
    for n in (1, nr):
        with H.HipftGPU(t, p, n, advance_flow=True, flow_num_method=method) as g:
            g.load_initial_map(br)
            g.set_flow(dr_model=1, mf_model=1, dr_p0=46.0, dr_p2=-262.0, dr_p4=-379.0, mf_p1=22.0, mf_p3=11.0,
                       mf_p5=-28.0, attenuate=attenuate)
            g.update_flow()
            g.advection_step(0.5 * g.flow_dtmax())
            out.append(g.get_field())
    assert np.isfinite(out[0]).all() and all(np.array_equal(out[0][0], f) for f in out[1])
