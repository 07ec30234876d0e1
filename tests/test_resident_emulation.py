"""The resident kernel's source on host threads (tests/emulation), with halo copies as
late as its own synchronisation allows, or lost: what a GPU would only show by chance, or
as a fault."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "tomography_gb300", "csrc")


@pytest.fixture(scope="module")
def emulated(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("emulation")
    # the stand-ins lie beside the kernel's own headers, in the place of the originals
    for f in ("solve_desc.h", "fdtd_advance.cuh", "fdtd_resident.cuh"):
        shutil.copy(os.path.join(CSRC, f), d)
    for f in os.listdir(os.path.join(HERE, "emulation")):
        shutil.copy(os.path.join(HERE, "emulation", f), d)
    exes = {}
    for share in (2, 4):
        exes[share] = str(d / f"resident{share}")
        subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-ffp-contract=off", f"-DSHARE={share}", "-I", str(d),
                        str(d / "resident.cpp"), "-o", exes[share], "-pthread"], check=True)
    return exes


def _run(exe, *args):
    p = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.mark.parametrize("share", [2, 4])
@pytest.mark.parametrize("blocks,steps", [(2, 2), (2, 3), (3, 4)])
def test_late_rows(emulated, share, blocks, steps):
    """No block overwrites its rows, or ends, before its neighbour has its last one."""
    _run(emulated[share], 64, 8 * blocks + 1, 4, blocks, steps, 5, "late")


@pytest.mark.parametrize("what", ["lost", "slow"])
@pytest.mark.parametrize("blocks,steps", [(2, 5), (3, 6), (4, 3)])
def test_rows_that_do_not_come(emulated, what, blocks, steps):
    """The whole cluster gives up, reports it, and no row arrives after its end."""
    _run(emulated[2], 64, 8 * blocks + 1, 4, blocks, steps, 5, what)


@pytest.mark.parametrize("share,rows", [(4, 4), (4, 6), (2, 4)])
def test_every_receiver_is_sampled(emulated, share, rows):
    """64 receivers on blocks of one warp, and of two."""
    _run(emulated[share], 90, 3 * rows + 1, 0, 3, 3, 64, "ends")
