"""hipft_gpu_describe names what a handle's diffusion step runs: per form the
grid that takes it, with the launches per pass counted on the handle (two steps
of different stage counts).  The forms without passes by name alone."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows, columns, graph-run steps, in the text, launches per pass
PASSES = [(65, 640, False, "in one launch", 1), (65, 639, False, "(k_sts_poles)", 2),
          (300, 65, False, "ws-quad (four stages per pass): k_sts_march, pole strips beside it", 2),
          (65, 640, True, "(k_sts_poles)", None), (12, 4400, False, "(k_sts_poles_any)", 5),
          (7, 100, False, "(k_sts_whole)", 1), (7, 600, False, "(k_sts_whole)", 4)]


def _handle(nt, npp, **kw):
    import hipft_b200 as H
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    g = H.HipftGPU(t, p, 1, advance_diffusion=True, diffusion_subcycles=1, diffusion_coef_constants=300.0, **kw)
    br = np.cos(t)[:, None] * np.ones(npp + 1)
    g.load_initial_map(br[None])
    return g


@pytest.mark.parametrize("nt,npp,graph,text,launches", PASSES)
def test_pass_forms(nt, npp, graph, text, launches):
    with _handle(nt, npp) as g:
        g.set_graph(graph)
        assert text in g.describe()
        if launches is None:
            return
        dte, n = g.info().dtime_diffusion_euler, []
        for r in (20.0, 400.0):
            before = g.info().kernel_launches
            s = g.diffusion_step(r * dte).sts_s
            n.append((math.ceil(s / 4), g.info().kernel_launches - before))
        (p0, l0), (p1, l1) = n
        assert p1 > p0 and l1 - l0 == launches * (p1 - p0)


def test_other_forms():
    with _handle(20, 30, diffusion_num_method=1) as g:
        assert "explicit Euler" in g.describe() and "ws-quad" not in g.describe()
    with _handle(20, 30, diffusion_coef_grid=True) as g:
        assert "k_diffusion_stage" in g.describe() and "ws-quad" not in g.describe()
        assert "schedule=shared" in g.describe()
