"""The bench line's figures for half sweeps (CPU: arithmetic and files): the
bytes of the rows that are swept, and captures that belong to the kernel and
the window width that ran."""
import importlib.util
import json
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
_spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
bench = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(bench)


@pytest.mark.parametrize("n,d,w,sweeps", [(65536, 16, 8192, 2), (24580, 8, 8192, 3), (20002, 4, 8192, 1)])
def test_half_sweep_bytes(n, d, w, sweeps):
    row, windows = w // 8, -(-n // w)
    want = 0
    for i in range(windows):
        for s in range(sweeps):
            writes = i == 0 or s + 1 < sweeps
            for v0 in range(i * w, n, w):               # a block of rows that is swept
                rows = min(w, n - v0)
                want += rows * (4 * d + (d + 1 + writes) * row)
            if writes:
                want += i * w * 2 * row                 # the rows above, by transposes
    assert bench.half_sweep_bytes(n, d, windows * sweeps, w) == want
    assert want < bench.sweep_bytes(n, d, windows * sweeps, w)


def test_captures_belong_to_the_width_that_ran():
    prof = json.loads((ROOT / "profiles" / "apsp_n65536d16_traffic.json").read_text())
    for kernel, width, other in [("apsp_sym_kernel", 8192, 4096), ("sym_ball_kernel", 8192, 4096),
                                 ("apsp_persistent_kernel", 4096, 1024), ("ball_kernel", 4096, 8192)]:
        assert bench.captured(prof, kernel, width)["dram_bytes_per_launch"] > 0
        assert bench.captured(prof, kernel, other) == {}
    assert bench.captured({}, "apsp_sym_kernel", 8192) == {}
