"""The library's compiled-in knobs, which a program that links it without the Python package runs with, are
the chosen values of tuning.json."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import json
from dpcrypto_b200 import kem
kem.apply_tuning = lambda *a: {}
print(json.dumps({k: kem.tuning_value(k) for k in kem.RUNTIME_KNOBS}))
"""


def test_compiled_defaults_are_the_chosen_knobs():
    from dpcrypto_b200 import build, kem

    build.build()
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    with open(os.path.join(ROOT, "dpcrypto_b200", "tuning.json")) as f:
        chosen = json.load(f)["chosen"]
    assert json.loads(r.stdout) == {k: chosen[k] for k in kem.RUNTIME_KNOBS}
