"""Source stamps whose mean is summed by a cluster of CTAs, a warp a row:
boxes of one cell, narrower than a warp, wider than one, clipped at every
edge, larger than the field, and more sources than a block culls at once. The
field equals the CPU oracle's bits, with the stamps' e^-u correctly rounded:
the oracle's own stamp calls the host's expf, which misses the nearest float
on about 0.07% of arguments."""
import numpy as np
import pytest

import oceanlib_b200 as ob
from oceanlib_b200.interaction import Disturbance, InteractionDesc, InteractionField
from oracle.iwave import OracleInteraction

pytestmark = pytest.mark.gpu

CELL = 0.25
F = np.float32


class CheckedField(OracleInteraction):
    def _inject(self, d, sub_time, scale):
        n, p, cell = self.n, self.p, self.cell
        sigma = max(F(d.radius), F(0.25) * cell)
        inv = F(1.0) / (F(2.0) * sigma * sigma)
        gx = (F(d.world_x) + F(d.velocity_x) * F(sub_time)) / cell
        gz = (F(d.world_z) + F(d.velocity_z) * F(sub_time)) / cell
        rad = int(np.ceil(F(4.0) * sigma / cell))
        x0, x1 = max(0, int(np.floor(gx)) - rad), min(n - 1, int(np.floor(gx)) + rad)
        z0, z1 = max(0, int(np.floor(gz)) - rad), min(n - 1, int(np.floor(gz)) + rad)
        if x1 < x0 or z1 < z0:
            return
        px = (np.arange(x0, x1 + 1).astype(F) + F(0.5)) - gx
        pz = (np.arange(z0, z1 + 1).astype(F) + F(0.5)) - gz
        u = ((px * px)[None, :] + (pz * pz)[:, None]) * cell * cell * inv
        stamp = (F(1.0) - u) * np.exp(-u.astype(np.float64)).astype(F)
        sh = stamp - F(stamp.astype(np.float64).sum() / stamp.size)
        dd, dv = F(-d.strength) * F(scale) * sh, F(d.velocity_y) * F(scale) * sh
        at = (slice(p + z0, p + z1 + 1), slice(p + x0, p + x1 + 1))
        self.planes[self.cur].reshape(self.rows, self.stride)[at] += dd
        self.planes[self.old].reshape(self.rows, self.stride)[at] += dd - dv * self.dt


CASES = {
    "one cell wide": [(16.0, 16.0, 0.0)],
    "corners": [(0.0, 0.0, 0.3), (32.0, 0.0, 0.3), (0.0, 32.0, 0.3), (32.0, 32.0, 0.3)],
    "outside": [(-3.0, 16.0, 1.0), (35.0, 16.0, 1.0), (16.0, -3.0, 1.0), (16.0, 35.0, 1.0)],
    "around a warp's width": [(16.0, 16.0, r * CELL / 4.0) for r in (15, 16, 17)],
    "around a cluster's rows": [(16.0, 16.0, r * CELL / 4.0) for r in (31, 32, 33)],
    "larger than the field": [(16.0, 16.0, 40.0)],
    "seventy overlapping": [(2.0 + 0.4 * i, 30.0 - 0.37 * i, 0.2 + 0.05 * (i % 9)) for i in range(70)],
}


@pytest.mark.parametrize("name", list(CASES))
def test_stamps(cuda_device, name):
    ob.force_simd_level(None)
    d = InteractionDesc(size=128, extent=128 * CELL, kernel_radius=3, max_sources=80)
    field = InteractionField(d)
    check = CheckedField(d, field.taps(), field.fixed_dt)
    for frame in range(2):
        for i, (x, z, r) in enumerate(CASES[name]):
            s = Disturbance(x, z, r, 0.3, 0.2, 0.7, -0.4, (i + frame) % 2)
            field.add(s)
            check.add(s)
        field.update(1.0 / 60.0)
        check.update(1.0 / 60.0)
    got = field.buffers()["field"]
    assert np.array_equal(np.ascontiguousarray(got).view(np.uint32), check.out.view(np.uint32))
