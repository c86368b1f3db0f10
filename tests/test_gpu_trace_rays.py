"""GPU tests of the tracer's ray directions: float32 pairs where their bound
decides, float64 where it does not. Bit-exact with the oracle for cameras near
and far, rays with a component at or near zero, odd frames and extreme scales."""
import numpy as np
import pytest

import dag_compression_fast_gb300 as D
from oracle import oracle as O
from tests.inputs import random_codes

pytestmark = pytest.mark.gpu


def params(camera, ray_min, ddx, ddy, width, height):
    p = D.TraceParams()
    p.debug_level, p.width, p.height = D.TRACE_POSITION_COLORS, width, height
    for k in range(3):
        p.camera[k], p.ray_min[k], p.ray_ddx[k], p.ray_ddy[k] = camera[k], ray_min[k], ddx[k], ddy[k]
    return p


CASES = {
    "inside": ((130.3, 90.1, 77.7), (129.0, 89.2, 78.5), (0.011, 0.0007, -0.003), (0.0002, 0.013, 0.0011), 201, 133),
    "zero_row_and_column": ((128.0, 128.0, -200.0), (127.0, 127.0, -199.0), (0.02, 0, 0), (0, 0.02, 0), 101, 101),
    "far": ((2e7, 1.1e7, -3e7), (2e7 - 1.0, 1.1e7 - 0.55, -3e7 + 1.5), (1e-6, 2e-7, 3e-7), (1e-7, 1e-6, -2e-7), 90, 70),
    "close_to_an_axis": ((120.5, 131.25, -50.0), (120.5001, 131.2501, -49.0), (1e-6, 0, 0), (0, 1e-6, 0), 128, 64),
    "large_steps": ((300.0, 400.0, -500.0), (-4e5, -3e5, 9e5), (9e3, 10.0, 3.0), (5.0, 8e3, 1.0), 96, 96),
    "one_pixel": ((300.0, 400.0, -500.0), (299.8, 399.7, -499.0), (0, 0, 0), (0, 0, 0), 1, 1),
    "out_of_float_range": ((1e20, 2e20, -3e20), (0.0, 0.0, 0.0), (1e17, 0, 0), (0, 1e17, 0), 33, 17),
    "tiny": ((128.0, 128.0, 128.0), (128.0 + 1e-9, 128.0 - 2e-9, 128.0 + 3e-9), (1e-11, 0, 2e-11), (0, 1e-11, 0), 40, 40),
    "no_direction": ((1.0, 1.0, 1.0), (1.0, 1.0, 1.0), (0.5, 0, 0), (0, 0.5, 0), 4, 4),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_ray_directions_bit_exact(ctx, case):
    codes = random_codes(8, 300_000, 11)
    words = ctx.create_final_dag(ctx.create_dag(codes, 8))
    p = params(*CASES[case])
    colors, hits = ctx.trace(words, 8, p)
    ref_c, ref_h, bad = O.trace(words.to_numpy(), 8, p)
    assert bad == 0
    assert np.array_equal(hits, ref_h)
    assert np.array_equal(colors, ref_c)
