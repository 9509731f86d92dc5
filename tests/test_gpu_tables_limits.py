"""Table production at the sizes where a block's shared memory meets a limit:
around 48 KB (num_thermo 331 .. 342), beyond which a launch needs the kernel's
attribute raised, and up to what an SM gives a block (1604 .. 1614).

Each path in a process of its own, smallest size first, so that no earlier call
has raised the attribute.  Against the host producer, bars as in
test_gpu_tables_frozen.py.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np
import torch
from discoeb_gb300 import tables_gpu
from discoeb_gb300.workloads import fiducial_mnu_param, lcdm_massless_param

frozen, sizes = sys.argv[1] == "frozen", [int(v) for v in sys.argv[2:]]
lead = [fiducial_mnu_param(), lcdm_massless_param()]
n = 3 * torch.cuda.get_device_properties(0).multi_processor_count + 1 if frozen else 2
sets = lead + [dict(lead[i % 2], Omegam=lead[i % 2]["Omegam"] * (1.0 + 1e-3 * (i + 1) / n)) for i in range(n - 2)]
leader = [-1, -1] + [i % 2 for i in range(n - 2)] if frozen else None
for num_thermo in sizes:
    host, st_h = tables_gpu.evolve_background_tables_host(sets, 3, num_thermo=num_thermo, leader=leader)
    dev, _, st = tables_gpu.evolve_background_tables(sets, 3, num_thermo=num_thermo, leader=leader)
    dev = dev.cpu().numpy()
    np.testing.assert_array_equal(st.cpu().numpy(), st_h)
    p = 32
    for s, m in enumerate(host[0, 20:27].astype(int)):
        bar = 1e-5 if s in (0, 1, 6) else 1e-10
        for part in range(2):
            h, d = host[:, p + part * m:p + (part + 1) * m], dev[:, p + part * m:p + (part + 1) * m]
            assert np.abs(d - h).max() <= bar * max(np.abs(h).max(), 1e-300), (num_thermo, s, part)
        p += 3 * m
"""


@pytest.mark.parametrize("path, sizes", [("adaptive", (32, 331, 332, 341, 342, 1604, 1605, 1614)),
                                         ("frozen", (332, 341, 342))])
def test_tables_at_the_shared_memory_limits(path, sizes):
    r = subprocess.run([sys.executable, "-c", CHILD, path] + [str(v) for v in sizes], cwd=ROOT, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
