"""RKG2/RKL2 passes whose pole strips run stage by stage (k_sts_poles_any: more
phi columns than a thread each in a cluster) and those of grids with fewer than
8 theta rows (k_sts_whole), at the edges of their division: one block of 64
columns and its edges, the largest cluster (8 blocks, all stages in one launch)
and one column more, a last block of one column, more blocks than a block has
threads.  Against the oracle within 1e-12; ragged batches and graph-run steps
give the bits of the plain step; the reverse pass, which keeps the stages' fields
and recomputes blocks of them, passes the transpose test of test_gpu_adj_march.
"""
import numpy as np
import pytest

import test_gpu_adj_march as A
import test_gpu_march as M

pytestmark = pytest.mark.gpu

# rows, columns and the hours of a step: 3 to 83 stages
GRIDS = [(4, 63, 100.0), (6, 64, 60.0), (7, 65, 40.0), (5, 128, 40.0), (6, 512, 6.0), (5, 513, 6.0),
         (6, 1030, 1.5), (8, 4352, 0.0138), (12, 4353, 0.0138), (70, 5000, 0.012), (4, 33000, 0.0018), (9, 33000, 0.0018)]


@pytest.mark.parametrize("coef", [1000.0, 20000.0])
@pytest.mark.parametrize("nt,npp,hours", GRIDS)
def test_pass_against_oracle(nt, npp, hours, coef, tmp_path):
    f, r = M._run(tmp_path, res_nt=nt, res_np=npp, n_realizations=2, diffusion_subcycles=1,
                  diffusion_coef_constants=[coef, 150.0], time_end=2.0 * hours, dt_max=hours)
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= M.FIELD_TOL, f"{int(r['num'][-1, 0, 6])} stages: rel max-norm {err:.3e}"


@pytest.mark.parametrize("nt,npp", [(5, 60), (5, 130), (9, 4400)])
def test_ragged_pass_equals_plain(nt, npp):
    M.test_ragged_pass_equals_plain(nt, npp)


@pytest.mark.parametrize("spacing", [0, 6])
@pytest.mark.parametrize("nt,npp", [(6, 50), (7, 200), (13, 4400)])
def test_transpose_and_diffusivity(nt, npp, spacing):
    A.test_transpose_and_diffusivity(nt, npp, 9, spacing)
