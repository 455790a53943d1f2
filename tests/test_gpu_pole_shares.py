"""Stages whose pole rows several blocks share, on wide grids, at the edges of
that division: one block and one column more (512 columns for the grid-dependent
diffusion and the upwind stages, 1024 for the WENO3 stage), a last share of few
columns, the most blocks a pole has and shares larger than one turn beyond them;
grids of one and of several blocks in theta, and more realizations than shares.
Against the oracle, relative max-norm 1e-12.
"""
import pytest

from test_gpu_pole_blocks import _check

pytestmark = pytest.mark.gpu
GRIDS = [(6, 512), (6, 513), (70, 514), (10, 1024), (10, 1025), (40, 2051), (9, 8192), (9, 8210), (6, 17000)]


@pytest.mark.parametrize("method", [2, 3])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_grid_dependent_diffusion(nt, npp, method, tmp_path):
    dt = 15.0 / npp
    _check(tmp_path, res_nt=nt, res_np=npp, advance_diffusion=True, diffusion_num_method=method, diffusion_subcycles=1,
           diffusion_coef_grid=True, diffusion_coef_constants=[400.0, 2000.0], time_end=2 * dt, dt_max=dt)


@pytest.mark.parametrize("method", [1, 2, 3, 4])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_advection(nt, npp, method, tmp_path):
    dt = 20.0 / npp
    _check(tmp_path, res_nt=nt, res_np=npp, advance_flow=True, flow_num_method=method, flow_dr_model=1, flow_mf_model=1,
           time_end=2 * dt, dt_max=dt)


@pytest.mark.parametrize("nr", [5, 17])
def test_advection_of_a_batch(nr, tmp_path):
    _check(tmp_path, res_nt=12, res_np=4100, n_realizations=nr, advance_flow=True, flow_num_method=4, flow_dr_model=1,
           flow_mf_model=1, time_end=0.01, dt_max=0.005)
