"""Ordering of the fused dispatch's arrival signals: an announcement releases what its own thread has fenced.
The copy warp's source is compiled for the host and run lane by lane; each announcement has to be
covered by a fence of the announcing lane taken after the rows' plain stores (zeroed padding, weights)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "moonep_b200", "csrc")


@pytest.fixture(scope="module")
def copy_warp(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("copy_warp")
    (d / "device").mkdir()
    for name in ("sync.cuh", "tma.cuh"):
        (d / "device" / name).write_text("#pragma once\n")
    exe = str(d / "copy_warp")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{d}", f"-I{CSRC}", os.path.join(HERE, "copy_warp_host.cc"), "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


# tokens, experts, top-k, CTAs: padding of more than 32 groups at once, fewer entries than CTAs, several batches
@pytest.mark.parametrize("S,E,K,ctas", [(40, 8, 4, 3), (300, 70, 2, 1), (5, 3, 2, 4), (512, 8, 8, 6), (1, 1, 1, 2)])
def test_every_announcement_is_behind_its_own_fence(copy_warp, S, E, K, ctas):
    out = subprocess.run([copy_warp, *map(str, (S, E, K, ctas))], check=True, capture_output=True, text=True, timeout=60)
    uncovered, announced, complete, blocks = map(int, out.stdout.split())
    assert announced > 0 and complete == blocks, "every block's rows are announced exactly once"
    assert uncovered == 0
