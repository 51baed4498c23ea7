"""Freed device memory goes back to CUDA: all of it when a program's only
handles are gone, or when it asks (virs_trim_memory); a slab's fields at once
(a neighbour's pull may still read them, which cudaFree waits for).  Each in a
process of its own, where no other handle or library allocates; 64 MiB of
slack for modules loaded late."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import numpy as np, torch
from virs_b200 import capi, slabs
def room(shape, slab=False):
    s = capi.Simulation(capi.default_params())
    flags = np.zeros(shape[::-1], np.uint8)
    flags[:, :, 0] = 1
    if slab:
        slabs.setup_slab(s, shape, 0.05, flags.reshape(-1), np.zeros(flags.size, np.uint8), 0, 2, 1)
    else:
        s.set_grid(shape, 0.05, flags.reshape(-1))
    s.classify()
    s.set_receivers([shape[0] * (shape[1] + 1) + 5])
    s.start(8)
    if not slab:
        s.run(4)
        s.synchronize()
    return s
free = lambda: torch.cuda.mem_get_info()[0]
small = room((64, 32, 16))      # context and kernels
"""


def _child(code):
    p = subprocess.run([sys.executable, "-c", HEAD + code], cwd=Path(__file__).resolve().parent.parent,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


def test_the_only_room_gives_its_memory_back():
    """80 M voxels: about 1.7 GB."""
    _child("""
before = free()
a = room((512, 512, 306))
held = before - free()
assert held > 1000 << 20, held
a.close()
small.close()
left = before - free()
assert left <= 64 << 20, left
""")


def test_rooms_after_rooms_give_it_back_when_asked():
    _child("""
small.close()
before = free()
for _ in range(3):
    room((512, 512, 100)).close()
other = room((64, 32, 16))
capi.trim_memory()
left = before - free()
assert left <= 64 << 20, left
other.run(4)
assert np.isfinite(other.ir()).all()
""")


def test_a_slabs_fields_are_not_kept():
    """Both fields of a slab of 32 M voxels at the least, while another handle lives."""
    _child("""
s = room((512, 512, 246), slab=True)
before = free()
s.close()
got = free() - before
assert got >= 2 * 4 * 512 * 512 * 122, got
""")
