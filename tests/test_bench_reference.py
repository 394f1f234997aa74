"""bench.py --impl reference times the reference's own module or says that it is not there: the C
restatement of the tests never stands in for it."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT
from oracle import oracle as O


def test_unavailable_without_the_module():
    if O.ref_libcpp() is not None:
        pytest.skip("the reference's module is built here")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference",
                        "--steps", "1", "--warmup", "1"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
