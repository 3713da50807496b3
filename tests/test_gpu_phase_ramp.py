"""The phase-ramp removal at the end of ML, AP, DM and RAAR calls (PyNX ZeroPhaseRamp), alone:
an AP call of no cycles against the float64 oracle, at every side the engine has and with one and
three modes. The centroid is a double sum of double transforms, so what differs is the single
precision of the arrays: each value rounded once, 6e-8, and 1e-6 holds with room."""
import numpy as np
import pytest

from oracle.ptycho import zero_phase_ramp
from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 96, 128, 192, 256])
@pytest.mark.parametrize("modes", [1, 3])
def test_ramp_of_a_call_without_cycles(n, modes):
    rng = np.random.default_rng(n + modes)
    side = n + 21
    probe = sim.hermite_probe(n, n / 4.0, [0.8, 0.15, 0.05][:modes])
    y, x = np.mgrid[:n, :n] / n
    probe = probe * np.exp(2j * np.pi * (3.3 * y - 1.7 * x))     # off-centre far field
    probe = (probe + 0.05 * (rng.normal(size=probe.shape) + 1j * rng.normal(size=probe.shape))
             * np.abs(probe).max()).astype(np.complex64)
    obj = (1.0 + 0.1 * rng.normal(size=(1, side, side + 6))).astype(np.complex64)
    scan = Scan(np.ones((2, n, n), np.float32), np.zeros(2), np.zeros(2), sim.WAVELENGTH,
                sim.DISTANCE, sim.DETECTOR_PIXEL)
    want_obj, want_probe = zero_phase_ramp(obj.astype(np.complex128), probe.astype(np.complex128))
    with GpuPtycho(scan, obj, probe) as g:
        g.ap(0, zero_phase_ramp=True)
        assert rel_l2(g.probe(), want_probe) < 1e-6
        assert rel_l2(g.object(), want_obj) < 1e-6
