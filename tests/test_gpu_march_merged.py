"""RKG2 passes as one launch (k_sts_march with the pole strips in its first
clusters) at the edges of the grids that take it, 640 to 1216 phi columns with
few realizations, and just beyond them: against the oracle at the bar of every
field, 1e-12, and a pair of realizations bit for bit as each of them in a batch
too large for one launch."""
import numpy as np
import pytest

import test_gpu_features as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GRIDS = [(8, 641), (65, 640), (64, 639), (121, 961), (9, 1000), (40, 1216), (41, 1217)]


@pytest.mark.parametrize("nt,npp", GRIDS)
def test_merged_pass_against_oracle(nt, npp, tmp_path):
    import hipft_b200 as H
    d = dict(F.BASE, validation_run=1, advance_diffusion=True, time_end=0.2, dt_max=0.1, res_nt=nt, res_np=npp,
             n_realizations=2, diffusion_subcycles=1, diffusion_coef_constants=[2000.0, 400.0])
    text = F._namelist(d)
    (tmp_path / "hipft.in").write_text(text)
    r = O.run(O.process_parameters(O.parse_namelist(text)))
    f = H.run_field(str(tmp_path / "hipft.in"), str(tmp_path), tuple(r["f"].shape))
    err = np.abs(f - r["f"]).max() / np.abs(r["f"]).max()
    assert np.isfinite(f).all() and err <= 1e-12, f"field rel max-norm {err:.3e}"


def test_merged_pass_equals_two_launches():
    import hipft_b200 as H
    nt, npp = 122, 720
    t, p = np.linspace(0.0, np.pi, nt), np.linspace(0.0, 2.0 * np.pi, npp + 1)
    br = np.random.default_rng(4).standard_normal((nt, npp + 1))
    br[:, -1] = br[:, 0]
    out = []
    for nr in (1, 40):
        with H.HipftGPU(t, p, nr, advance_diffusion=True, diffusion_subcycles=1, diffusion_coef_constants=300.0) as g:
            g.load_initial_map(br[None])
            g.diffusion_step(2.0)
            out.append(g.get_field())
    assert all(np.array_equal(out[0][0], f) for f in out[1])
