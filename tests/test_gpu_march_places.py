"""Chunks of the RKG2 march that take the places of narrow pole strips into
account (at most 20 columns) and those that do not, on both sides of that line:
the realizations of a batch bit for bit as those of a larger one, plain, ragged
and graph-run (whose chunks the schedule kernel works out)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows, columns, realizations: 512x1024 x 3 has chunks of 20 columns, x 4 of 28 or 24,
# 256x512 x 12 of 28 or 20
GRIDS = [(512, 1024, 3), (512, 1024, 4), (256, 512, 12), (180, 360, 32), (359, 722, 9), (90, 880, 12)]


@pytest.mark.parametrize("mode", ["plain", "ragged", "graph"])
@pytest.mark.parametrize("nt,npp,nr", GRIDS)
def test_batch_equals_a_larger_one(nt, npp, nr, mode):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    br = np.random.default_rng(4).standard_normal((1, nt, npp + 1))
    br[..., -1] = br[..., 0]
    dt, out = None, []
    for n, m in ((64, "plain"), (nr, mode)):
        with H.HipftGPU(t, p, n, advance_diffusion=True, diffusion_subcycles=1, diffusion_coef_constants=300.0) as g:
            g.load_initial_map(br)
            if dt is None:
                dt = 60.0 * g.info().dtime_diffusion_euler  # three or four passes
            if m == "ragged":
                g.set_ragged(True)
            g.set_graph(m == "graph")
            (g.flux_transport_step if m == "graph" else g.diffusion_step)(dt)
            out.append(g.get_field())
    assert all(np.array_equal(out[0][0], f) for f in out[1])
