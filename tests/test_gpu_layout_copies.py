"""The copies between the caller's flat node order and the padded layout.

A fixed row of the operator is the identity, so on a board whose nodes are all
fixed but one an action returns its input bit for bit: whatever differs was
lost or moved by the copies on the way in or out.  Sizes: rows shorter than a
group of lanes, around a group's width, around a segment, and of several
segments.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import pcb_analysis_b200.thermal as thermal
from pcb_analysis_b200 import workloads
from pcb_analysis_b200._native import DeviceSystem

pytestmark = pytest.mark.gpu


def _nearly_fixed(slabs, rows, cols):
    nodes = (slabs + 1) * (rows + 1) * (cols + 1)
    free = np.zeros(nodes, dtype=np.uint8)
    free[nodes // 2] = 1
    return DeviceSystem(slab_thickness_m=np.full(slabs, 0.2e-3), pitch_x_m=np.full(cols, 0.25e-3),
                        pitch_y_m=np.full(rows, 0.25e-3), k_in=np.ones((slabs, rows, cols)),
                        k_z=np.ones((slabs, rows, cols)), robin_total=np.zeros(nodes), free_nodes=free), free == 0


@pytest.mark.parametrize(
    "slabs, rows, cols",
    [(1, 1, 1), (1, 40, 1), (2, 9, 2), (1, 130, 3), (2, 5, 4), (1, 17, 7), (3, 11, 8), (1, 6, 15), (1, 5, 16),
     (2, 7, 31), (1, 3, 32), (1, 4, 200), (1, 2, 1023), (1, 2, 1024), (1, 3, 1027), (1, 1, 2051), (2, 1, 5000)],
)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_fixed_rows_come_back_unchanged(slabs, rows, cols, dtype):
    system, fixed = _nearly_fixed(slabs, rows, cols)
    with system:
        generator = torch.Generator(device="cuda").manual_seed(rows + cols)
        x = torch.randn(system.size, generator=generator, device="cuda", dtype=dtype)
        y = torch.full_like(x, float("nan"))
        low = dtype == torch.float32
        (system.apply_f32_device if low else system.apply_f64_device)(x, y)
        host = (system.apply_f32 if low else system.apply_f64)(x.cpu().numpy())
    y, x = y.cpu().numpy(), x.cpu().numpy()
    np.testing.assert_array_equal(y[fixed], x[fixed])
    assert np.all(np.isfinite(y))
    np.testing.assert_array_equal(host, y)


def test_a_long_strip_is_copied_by_the_whole_device():
    """FP32 actions of a 1 x 100,000 board and of one with as many elements in a
    square: the strip's operator does about as much work, so an action several
    times as long can only be its copies (eleven times, with a warp per row)."""

    def microseconds(rows, cols):
        operator = thermal.MatrixFreeThermalOperator(workloads.board_c1(1, None, rows, cols), preconditioner="jacobi")
        try:
            x = torch.randn(operator.size, device="cuda")
            y = torch.empty_like(x)
            times = []
            for _ in range(25):
                begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                begin.record()
                operator.device_system.apply_f32_device(x, y)
                end.record()
                end.synchronize()
                times.append(1e3 * begin.elapsed_time(end))
        finally:
            operator.close()
        return float(np.median(times))

    assert microseconds(1, 100_000) <= 4.0 * microseconds(316, 316)
