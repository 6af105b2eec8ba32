"""All RyRs' mouth values at once equal those read site by site, in batches whose values are copied
whole and in batches whose species is gathered on the device (on both sides of 48 KiB)."""
import numpy as np
import pytest

import casim_b200 as cb
from casim_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 61, 62, 200])
def test_all_mouth_equals_single_sites(cuda_device, n):
    p, s = configs.config1(n_sites=n)
    sim = cb.ReleaseSiteBatch(p, s, precision="fp32")
    sim.start(s["first_channel"])
    sim.step(30)
    for k in range(sim.n_species):
        a = sim.all_mouth(k)
        for site in sorted({0, n // 2, n - 1}):
            off = int(sim.n_ch[:site].sum())
            assert np.array_equal(a[off:off + int(sim.n_ch[site])], sim.mouth(site, k))
    sim.close()
