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


def test_handles_of_different_widths_side_by_side():
    """A kernel's shared-memory limit serves every handle: a narrower grid made
    later leaves a wider one's passes and reverse passes as they were."""
    import hipft_b200 as H
    from hipft_b200.adjoint import MisfitAdjoint
    nt, zero = 70, {k: np.zeros(1) for k in ("p0", "p2", "p4", "p1", "p3", "p5")}
    kw = dict(advance_flow=True, flow_num_method=4, strang_splitting=True, advance_diffusion=True,
              diffusion_num_method=3, diffusion_subcycles=1, diffusion_coef_constants=np.array([300.0]))
    t = np.linspace(0.0, np.pi, nt)
    x = np.random.default_rng(0).standard_normal((1, 1202, nt))
    x[:, 0], x[:, -1] = x[:, -2], x[:, 1]

    def gradient(g):
        A = MisfitAdjoint(g, np.array([300.0]), zero)
        F = A.forward(x, [0.02])
        return F, A.backward(x)["f0"]

    with H.HipftGPU(t, np.linspace(0.0, 2.0 * np.pi, 1201), 1, **kw) as wide:
        wide.set_flow(dr_model=1, mf_model=1)
        F0, g0 = gradient(wide)
        with H.HipftGPU(t, np.linspace(0.0, 2.0 * np.pi, 641), 1, **kw) as g:
            g.set_flow(dr_model=1, mf_model=1)
            MisfitAdjoint(g, np.array([300.0]), zero).forward(x[:, :642], [0.02])
            F1, g1 = gradient(wide)
        assert np.array_equal(F0, F1) and np.array_equal(g0, g1)
