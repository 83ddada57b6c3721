"""Item sizes and shared-memory room of spin-resolved products, checked on the host: tests/cpp/hop_room_check.cu is
compiled as host code by nvcc and counts the up hops of every item of every split of every sector of up to 20 sites."""
import os
import subprocess

import pytest

from test_ffloat_cpu import HERE, _nvcc


def test_every_item_of_a_product_has_room_for_its_hops(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "hop_room_check")
    src = os.path.join(HERE, "cpp", "hop_room_check.cu")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
