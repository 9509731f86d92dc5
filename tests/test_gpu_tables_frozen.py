"""Sets on the recorded steps of another set: one launch (each follower beside
a repetition of its leader) for up to three sets per SM, two launches above.

Both against the host producer, which follows its own record of the same
leader.  Bars as in test_gpu_tables.py: 1e-10 of each array's largest magnitude
for the background tables, 1e-5 for what the RECFAST integration at rtol 1e-3
yields, where a rounding difference may move a step decision of the leader.
"""
import numpy as np
import pytest
import torch

from discoeb_gb300 import tables_gpu
from discoeb_gb300.workloads import fiducial_mnu_param, lcdm_massless_param

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_thermo, where", [(256, "two"), (256, "last of one"), (256, "first of two"), (64, "two")])
def test_followers_match_the_host_producer(num_thermo, where):
    line = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    n = {"two": 2, "last of one": line, "first of two": line + 1}[where]
    lead = [fiducial_mnu_param(), lcdm_massless_param()][:1 if n == 2 else 2]
    sets = lead + [dict(lead[i % len(lead)], Omegam=lead[i % len(lead)]["Omegam"] * (1.0 + 1e-3 * (i + 1) / n))
                   for i in range(n - len(lead))]
    leader = [-1] * len(lead) + [i % len(lead) for i in range(n - len(lead))]
    host, st_h = tables_gpu.evolve_background_tables_host(sets, 5, num_thermo=num_thermo, leader=leader)
    dev, _, st = tables_gpu.evolve_background_tables(sets, 5, num_thermo=num_thermo, leader=leader)
    dev = dev.cpu().numpy()
    np.testing.assert_array_equal(st.cpu().numpy(), st_h)
    p = 32
    for s, m in enumerate(host[0, 20:27].astype(int)):
        bar = 1e-5 if s in (0, 1, 6) else 1e-10
        for part in range(2):
            h, d = host[:, p + part * m:p + (part + 1) * m], dev[:, p + part * m:p + (part + 1) * m]
            assert np.abs(d - h).max() <= bar * max(np.abs(h).max(), 1e-300), (s, part)
        p += 3 * m
