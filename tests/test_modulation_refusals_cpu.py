"""A modulation that is refused is refused before its tables are allocated: the
calls below ask for tables of 128 GiB in a process that may have 16."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]

pytest.importorskip("henon_map_cpp_b200._capi")

CODE = """
import resource, sys
resource.setrlimit(resource.RLIMIT_AS, (16 << 30, 16 << 30))
sys.path.insert(0, {repo!r})
from henon_map_cpp_b200 import _capi as C
N = 0xffffffff
nan = float("nan")
calls = {{
    "tracker": lambda: C.Tracker(N, 0.168, 0.201, {kind!r}, nan, 1.0, 0),
    "batch": lambda: C.Batch([dict(omega_x=0.1, omega_y=0.2, epsilon=1.0, mu=0.0, n_turns=N,
                                   n_particles=1, modulation_kind={kind!r})]),
}}
try:
    calls[{what!r}]()
except C.HMError as e:
    print(e.status, e)
"""


@pytest.mark.parametrize("what", ["tracker", "batch"])
@pytest.mark.parametrize("kind,message", [("bogus", "Unknown modulation kind"),
                                          ("basic", "basic modulation needs a finite omega_0")])
def test_refused_before_allocating(kind, message, what):
    r = subprocess.run([sys.executable, "-c", CODE.format(repo=str(REPO), kind=kind, what=what)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    assert message in r.stdout
