"""A bounded wait that gives up lets the whole block drain: the head's epilogue, compiled from the kernel's own source, as CPU threads."""
import os
import re
import shutil
import subprocess

import pytest

from common import ROOT


@pytest.fixture(scope="module")
def head(tmp_path_factory):
    d = tmp_path_factory.mktemp("head")
    csrc = d / "package" / "csrc"
    csrc.mkdir(parents=True)
    (d / "include").mkdir()
    shutil.copy(os.path.join(ROOT, "include", "egg_b200.h"), d / "include")
    for f in ("egg_common.cuh", "egg_gemm.cuh"):
        with open(os.path.join(ROOT, "egg.c_b200", "csrc", f)) as src:
            (csrc / f).write_text(re.sub(r"\basm( volatile)?\(.*?\);", ";", src.read(), flags=re.S))
    (csrc / "egg_ptx.cuh").write_text("")
    exe = str(d / "head")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", "/usr/local/cuda/include", "-I", str(csrc), "-o", exe,
                    os.path.join(ROOT, "tests", "head_on_cpu.cpp"), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("warp,tile", [(-1, 0), (2, 0), (7, 1), (12, 2), (17, 4)])      # warps of each column and lane quarter; first and last tile
def test_a_warp_of_the_head_that_gives_up_leaves_nobody_at_a_barrier(head, warp, tile):
    r = subprocess.run([head, str(warp), str(tile)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    err, *loss = map(int, r.stdout.split())
    assert err == (0 if warp < 0 else 3)          # DEV_TIMEOUT_TMEM_FULL
    assert warp >= 0 or all(x > 0 for x in loss)
