"""The marching WENO3 stage with 2-D flows against the oracle bit for bit: flows
from files (with and without the analytic ones), which both sides form by the
same operations, at the edges of the stage's strips and chunks, both SSPRK
schemes and a set weno_eps.  One step from a map; bits away from the poles (ten
rows: what four stages of a two-row stencil reach, and the pole rows' ring sums,
which the oracle adds in another order), 1e-12 in relative max-norm everywhere.
"""
import numpy as np
import pytest

import test_gpu_features as F
from oracle import oracle as O
from test_gpu_flow_files import _flows

pytestmark = pytest.mark.gpu
GRIDS = [(31, 62), (59, 33), (60, 34), (61, 35), (62, 36), (63, 66), (121, 66), (122, 130), (181, 257)]


@pytest.mark.parametrize("models,eps", [(0, 0.0), (1, 0.0), (1, 0.01)])
@pytest.mark.parametrize("method", [3, 4])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_stage_against_oracle(nt, npp, method, models, eps, tmp_path):
    import hipft_b200 as H
    d = dict(F.BASE, validation_run=1, advance_flow=True, flow_num_method=method, use_flow_from_files=True,
             flow_list_filename="flows/list.txt", flow_root_dir="flows", flow_dr_model=models, flow_mf_model=models,
             weno_eps=eps, res_nt=nt, res_np=npp, n_realizations=2, time_end=0.4, dt_max=0.4)
    flows = _flows(tmp_path, nt, npp, 2)
    text = F._namelist(d)
    (tmp_path / "hipft.in").write_text(text)
    r = O.run(O.process_parameters(O.parse_namelist(text)), flows=flows)
    assert r["nsteps"] == 1
    f = H.run_field(str(tmp_path / "hipft.in"), str(tmp_path), tuple(r["f"].shape))
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= F.FIELD_TOL, f"field rel max-norm {err:.3e}"
    assert np.array_equal(f[..., 10:-10].view(np.uint64), r["f"][..., 10:-10].view(np.uint64))
