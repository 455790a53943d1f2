"""Weights of the mu^power blend, rounded from more bits than a double has: a
blend of the map 1 into the field 0 is the weight itself, compared with 50
digit arithmetic.  The error of the sum before rounding is below 2^-64 of it,
2^-11 of a unit in the last place."""
import math
from decimal import Decimal, localcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi,powers", [
    (0.01, 1.0, (4.0, 2.0, 0.5, 3.7, 1.0)),           # the range in use
    (0.9999999, 1.0000001, (4.0, -3.3, 1e5, 60.0, 0.0)),  # log close to 0
    (1e-30, 1e30, (4.0, -2.5, 0.1, -7.3, 1e-3)),      # large and small results
])
def test_gpu_da_weights_are_rounded_powers(lo, hi, powers):
    import hipft_b200 as H
    ntm, npm1, nr = 24, 41, len(powers)
    rng = np.random.default_rng(3)
    mu = np.exp(rng.uniform(math.log(lo), math.log(hi), size=(ntm, npm1)))
    mu[1, 1:4] = (1.0, -1.0, lo)
    with H.HipftGPU(np.linspace(0.0, np.pi, ntm), np.linspace(0.0, 2.0 * np.pi, npm1), nr) as g:
        g.set_field(np.zeros((nr, npm1 + 1, ntm)))
        g.assimilate(np.stack([np.ones_like(mu), np.full_like(mu, 7.0), mu]), custom_from_mu=True, mu_power=powers,
                     mu_limit=lo)
        w = g.get_field()[:, :npm1, :].transpose(0, 2, 1)  # column k holds map column k, 1 the seam
    with localcontext() as ctx:
        ctx.prec = 50
        for i, p in enumerate(powers):
            for j in range(ntm):
                for k in range(1, npm1):
                    x, got = mu[j, k], float(w[i, j, k])
                    if not x > lo:
                        assert got == 0.0
                        continue
                    err = abs(Decimal(got) - Decimal(x) ** Decimal(p)) / Decimal(math.ulp(got))
                    assert err <= Decimal(0.5 + 2.0 ** -11), (x, p, got, err)
