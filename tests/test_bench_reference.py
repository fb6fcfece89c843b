"""The reference arm of bench.py never times this repository's own code: without the compiled reference it says so."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


def test_reference_arm_without_the_reference():
    from oracle import oracle as orc
    if orc.Reference.available(fast=True):
        pytest.skip("the reference is built here")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "1"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
