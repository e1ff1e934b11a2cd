"""launch_batch_pso_cost without sources or particles returns before any
arithmetic on the counts (a host call: no GPU, no pointer is read)."""
import subprocess
import sys

import pytest

from lightcurve_fitting_gb300 import build


@pytest.mark.parametrize("sources,particles", [(0, 30), (5, 0), (0, 0), (-1, -1), (-3, -40), (5, -1)])
@pytest.mark.parametrize("model", [1, 7])
def test_no_rows(sources, particles, model):
    build.build()
    code = ("from lightcurve_fitting_gb300.lib import load\n"
            f"load().launch_batch_pso_cost(*[None] * 8, {sources}, {particles}, 5, {model}, 1, 256)\n"
            "print('returned')\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "returned", r.stderr
