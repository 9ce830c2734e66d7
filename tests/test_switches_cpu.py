"""What an environment switch of the library decides, asked of the library in child processes (it reads each switch once)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def ask(expression, **env):
    code = ("import sys\nsys.path.insert(0, sys.argv[1])\nfrom kch_b200 import _lib\nlib = _lib.load()\n"
            f"print({expression})\n")
    r = subprocess.run([sys.executable, "-c", code, os.path.join(ROOT, "kda-csa-hca-fusion_b200")], capture_output=True, text=True,
                       check=True, env={**os.environ, **env}, timeout=300)
    return r.stdout.strip()


@pytest.mark.parametrize("value,want", [("", "1"), ("o", "0")])
def test_the_general_one_token_kernel_also_replaces_the_step_that_projects_its_gate(value, want):
    """KCH_KDA_DECODE=o asks for the general recurrent kernel: the step with the gate's projection inside has to stand back, or a
    comparison of the two would run the same kernel twice."""
    assert ask("lib.kch_kda_step_gate_supported(3, 2, 128, 128, _lib.KCH_BF16)", KCH_KDA_DECODE=value) == want
