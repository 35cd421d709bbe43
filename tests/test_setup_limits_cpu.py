"""The set-up of the largest chemistries, under glibc's heap checks where they are installed."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from mocassin_xray_gb300 import configs

SCRIPT = """
import sys
sys.path.insert(0, sys.argv[3])
from mocassin_xray_gb300 import Setup
for _ in range(3):
    s = Setup(sys.argv[1], sys.argv[2])
    assert s.info.n_elem_used == 30 and s.info.nstages == int(sys.argv[4])
    s.close()
"""


@pytest.mark.parametrize("stages", [3, 27, 31])
def test_every_element(data_dir, tmp_path, stages):
    """All 30 elements: with 31 stages they have 465 ionisation edges."""
    p = configs.xray_gas(tmp_path, n=3, packets=10)
    p.write_text(p.read_text().replace("nstages 27", f"nstages {stages}"))
    (p.parent / "abun_xray.in").write_text("1.\n" + "1.e-4\n" * 29)
    env = dict(os.environ, MALLOC_CHECK_="3")
    if any(Path(d, "libc_malloc_debug.so.0").exists() for d in
           ("/lib/x86_64-linux-gnu", "/lib/aarch64-linux-gnu", "/lib64", "/usr/lib64")):
        env["LD_PRELOAD"] = "libc_malloc_debug.so.0"
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(p), str(data_dir), str(Path(__file__).parents[1]), str(stages)],
                       env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-500:]
