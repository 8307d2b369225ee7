"""The oracle's library can be built by several processes that find it missing at once,
as the worker processes of the reference arm do in a fresh checkout."""

import subprocess
import sys

from conftest import ROOT

WORKER = """
import sys
from pathlib import Path
sys.path.insert(0, sys.argv[1])
import ssm_oracle
ssm_oracle.LIB = Path(sys.argv[2])
while not Path(sys.argv[3]).exists():
    pass
ssm_oracle.lib()
"""


def test_processes_that_find_no_library_build_it_side_by_side(tmp_path):
    lib, go = tmp_path / "lib" / "liboracle.so", tmp_path / "go"
    ps = [subprocess.Popen([sys.executable, "-c", WORKER, str(ROOT / "oracle"), str(lib), str(go)],
                           stderr=subprocess.PIPE, text=True) for _ in range(8)]
    go.touch()
    errors = [p.communicate(timeout=120)[1] for p in ps]
    assert [p.returncode for p in ps] == [0] * 8, errors
    assert [f.name for f in lib.parent.iterdir()] == [lib.name]
