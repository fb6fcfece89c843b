"""2049 to 16,384 tokens per call: the grouping's larger cluster and, above 4096 tokens, its mark and place kernels, the combine's whole waves, streamed chunks and
host flows of that size.  Grouping against the oracle; the others against the same rows in parts of 2048, which the other tests pin, bit for bit."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
NAMES = (["grouping of %d tokens, %s" % (n, k) for n in (2049, 3000, 4096, 4097, 8191, 16384) for k in ("even", "skew", "same")] +
         ["stack of %d tokens" % n for n in (2049, 4096, 4097, 10000, 16384)] +
         ["stack of 4096 tokens, exact-order router", "stack of 16384 tokens, skewed", "layer call of 5000 tokens", "streamed chunks of 4096 tokens",
          "streamed chunks of 8192 tokens", "plug-in call of 4096 tokens", "plug-in call of 4999 tokens", "attention sides of 4097 tokens",
          "attention sides of 16384 tokens"])


@pytest.fixture(scope="module")
def said():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "large_worker.py")], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("name", NAMES)
def test_large_calls(name, said):
    assert said[name] == "ok"
