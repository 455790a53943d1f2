"""The stages whose pole rows are a block of the same launch (k_diffusion_stage
with a grid-dependent D or explicit Euler steps, k_adv_upwind), against the
oracle: fewer phi columns than the pole block's 256 threads, around them, and
more; odd and even rows around a tile's 32."""
import numpy as np
import pytest

import test_gpu_features as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GRIDS = [(4, 6), (9, 40), (31, 62), (33, 256), (34, 257), (20, 520)]


def _check(tmp_path, **kw):
    import hipft_b200 as H
    d = dict(F.BASE, validation_run=1, n_realizations=2)
    d.update(kw)
    text = F._namelist(d)
    (tmp_path / "hipft.in").write_text(text)
    r = O.run(O.process_parameters(O.parse_namelist(text)))
    f = H.run_field(str(tmp_path / "hipft.in"), str(tmp_path), tuple(r["f"].shape))
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= 1e-12, f"field rel max-norm {err:.3e}"


@pytest.mark.parametrize("method", [1, 2, 3])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_grid_dependent_diffusion(nt, npp, method, tmp_path):
    dt = 0.2 if method == 1 and npp > 100 else 1.5
    _check(tmp_path, res_nt=nt, res_np=npp, advance_diffusion=True, diffusion_num_method=method, diffusion_subcycles=1,
           diffusion_coef_grid=True, diffusion_coef_constants=[400.0, 2000.0], time_end=2 * dt, dt_max=dt)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_upwind_advection(nt, npp, method, tmp_path):
    _check(tmp_path, res_nt=nt, res_np=npp, advance_flow=True, flow_num_method=method, flow_dr_model=1, flow_mf_model=1,
           time_end=6.0, dt_max=3.0)
