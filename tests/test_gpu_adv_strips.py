"""The marching WENO3 advection stage against the oracle at the sizes where its
division of the field can go wrong: theta rows around the 60 a strip owns and
the fewest there are, phi columns fewer than the window and around the blocks'
chunks, 1-D and 2-D (attenuated) flows, both SSPRK schemes.

One step from a map with 1-D flows: away from the poles (eight rows a step's
four stages reach with their two-row stencil, and the pole rows' ring sums,
which the oracle adds in another order) the fields are the oracle's bit for
bit, which holds the faces' quotients to the IEEE division's.  Everywhere, and
with 2-D flows (whose attenuation evaluates tanh on the device), the bar is
1e-12 in relative max-norm.
"""
import numpy as np
import pytest

import test_gpu_features as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-12
GRIDS = [(4, 5), (5, 6), (7, 12), (31, 5), (59, 33), (60, 34), (61, 35), (62, 36), (63, 40), (119, 65), (121, 66),
         (122, 130), (181, 257), (240, 500)]


@pytest.mark.parametrize("attenuate", [False, True])
@pytest.mark.parametrize("method", [3, 4])
@pytest.mark.parametrize("nt,npp", GRIDS)
def test_stage_against_oracle(nt, npp, method, attenuate, tmp_path):
    import hipft_b200 as H
    d = dict(F.BASE, validation_run=1, advance_flow=True, flow_num_method=method, flow_dr_model=1, flow_mf_model=1,
             res_nt=nt, res_np=npp, n_realizations=2, time_end=0.5, dt_max=0.5)
    if attenuate:
        d.update(flow_attenuate=True, flow_attenuate_values=[0.7, 2.0])
    text = F._namelist(d)
    (tmp_path / "hipft.in").write_text(text)
    r = O.run(O.process_parameters(O.parse_namelist(text)))
    assert r["nsteps"] == 1
    f = H.run_field(str(tmp_path / "hipft.in"), str(tmp_path), tuple(r["f"].shape))
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= FIELD_TOL, f"field rel max-norm {err:.3e}"
    if not attenuate and nt > 24:
        assert np.array_equal(f[..., 10:-10], r["f"][..., 10:-10])
