"""Four RKG2/RKL2 stages per pass (k_sts_march, k_sts_poles, k_sts_poles_any,
k_sts_whole) against the oracle, at the grid sizes where their division of the
field can go wrong:

* theta: fewer rows than the strip kernels take (4..7: k_sts_whole), the
  smallest they take (8, 9: the two pole strips meet), one strip and its edges
  (64 rows held, 56 owned, 4 + 4 at the poles), odd and even last rows;
* phi: fewer columns than the halo of a chunk (5, 6), around a multiple of the
  columns of a turn, around the columns of one block of the pole strips' cluster
  (248), on its largest cluster, and beyond a column per thread;
* stage counts: one pass (s = 3) and several, both paddings of the first pass.

The bar is the one every field has against the oracle, 1e-12 in relative
max-norm; the runs are a few short steps with few stages.
"""
import numpy as np
import pytest

import test_gpu_features as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-12
GRIDS = [(4, 5), (5, 40), (7, 9), (8, 5), (8, 70), (9, 6), (15, 33), (16, 64), (63, 47), (64, 48), (65, 49), (66, 31),
         (120, 62), (121, 63), (122, 64), (177, 90), (31, 248), (32, 249), (33, 497), (20, 1985), (10, 2050), (9, 4300)]


def _run(tmp_path, **kw):
    import hipft_b200 as H
    d = dict(F.BASE, validation_run=1, advance_diffusion=True, time_end=3.0, dt_max=1.5)
    d.update(kw)
    text = F._namelist(d)
    (tmp_path / "hipft.in").write_text(text)
    r = O.run(O.process_parameters(O.parse_namelist(text)))
    f = H.run_field(str(tmp_path / "hipft.in"), str(tmp_path), tuple(r["f"].shape))
    return f, r


@pytest.mark.parametrize("nt,npp", GRIDS)
def test_pass_against_oracle(nt, npp, tmp_path):
    f, r = _run(tmp_path, res_nt=nt, res_np=npp, n_realizations=2, diffusion_subcycles=1,
                diffusion_coef_constants=[20000.0, 400.0])
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= FIELD_TOL, f"field rel max-norm {err:.3e}"


@pytest.mark.parametrize("method", [2, 3])
@pytest.mark.parametrize("coef", [150.0, 1000.0, 4000.0, 9000.0, 30000.0])
def test_stage_counts_against_oracle(method, coef, tmp_path):
    f, r = _run(tmp_path, res_nt=70, res_np=141, n_realizations=1, diffusion_num_method=method, diffusion_subcycles=1,
                diffusion_coef_constants=[coef])
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert err <= FIELD_TOL, f"{int(r['num'][-1, 0, 6])} stages: field rel max-norm {err:.3e}"


@pytest.mark.parametrize("nt,npp", [(5, 20), (70, 67)])
def test_ragged_pass_equals_plain(nt, npp):
    """Equal realizations: a ragged batch and the shared schedule give the same
    bits, also when a step runs as a graph."""
    import hipft_b200 as H
    import test_gpu_refined as R
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp)
    out = []
    for ragged, graph in ((False, False), (True, False), (False, True), (True, True)):
        with H.HipftGPU(t, p, 3, advance_diffusion=True, diffusion_coef_constants=[500.0] * 3) as g:
            g.load_initial_map(R.smooth_map(t, p, 3)[None])
            g.set_ragged(ragged)
            g.set_graph(graph)
            for _ in range(2):
                g.flux_transport_step(4.0)
            out.append(g.get_field())
    for f in out[1:]:
        assert np.array_equal(out[0], f)
