"""The repository's smoke entry point, in a process of its own as its callers run it (the launch counter starts at zero)."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_smoke_entry_point_passes(built_lib):
    res = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.smoke()"], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert res.returncode == 0 and "smoke ok" in res.stdout, res.stdout + res.stderr
