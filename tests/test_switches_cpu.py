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


@pytest.mark.parametrize("heads,chunks,segments", [
    # a chain was the faster one, by 5 to 14 % where segments were taken until now
    (16, 20, False), (32, 80, False), (32, 200, False), (36, 300, False), (28, 512, False), (49, 63, False), (41, 60, False), (64, 63, False),
    (1, 19, False), (16, 23, False), (24, 30, False), (40, 43, False), (28, 129, False), (32, 64, False),
    (1, 20, True), (8, 20, True), (16, 24, True), (16, 512, True), (24, 31, True), (24, 512, True), (28, 128, True), (32, 63, True),
    (32, 37, True), (40, 44, True)])
def test_where_segments_of_a_sequence_are_scanned_side_by_side(heads, chunks, segments):
    """The workspace of the bf16 path tells which form a KDA call takes: records of 148480 bytes a chunk and head, and either one
    carried state a head or the segments' own buffers.  (The function behind the exported size, which also has the fp32 path's.)"""
    import ctypes
    from kch_b200 import _lib
    size = _lib.load()._Z27kch_kda_mma_workspace_bytesiii
    size.restype, size.argtypes = ctypes.c_int64, [ctypes.c_int] * 3
    chain = heads * chunks * 148480 + heads * 65536
    assert (size(1, 64 * chunks - 5, heads) > chain) == segments


@pytest.mark.parametrize("value,more", [("0", "False"), ("1", "True")])
def test_either_form_of_the_scan_can_be_asked_for(value, more):
    """KCH_KDA_SPLIT=0 and =1: one chain where segments pay, segments where they do not."""
    heads, chunks = (8, 64) if value == "0" else (32, 200)
    chain = heads * chunks * 148480 + heads * 65536
    size = f"[setattr(f, 'restype', __import__('ctypes').c_int64) or f(1, {64 * chunks}, {heads}) for f in [lib._Z27kch_kda_mma_workspace_bytesiii]][0]"
    assert ask(f"{size} > {chain}", KCH_KDA_SPLIT=value) == more
