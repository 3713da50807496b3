"""The phase-ramp removal at the end of ML, AP, DM and RAAR calls (PyNX ZeroPhaseRamp), alone:
an AP call of no cycles against the float64 oracle, at every side the engine has and with one and
three modes. The centroid is a double sum of double transforms, so what differs is the single
precision of the arrays: each value rounded once, 6e-8, and 1e-6 holds with room."""
import numpy as np
import pytest

from oracle.ptycho import zero_phase_ramp
from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import far_field, rel_l2
from test_zz_no_alloc import _driver, _pool_used

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


@pytest.mark.parametrize("modes,stack,own", [(1, 1, False), (2, 2, False), (3, 2, False),
                                             (3, 1, True)])
def test_ramp_lies_in_memory_held_anyway(modes, stack, own):
    """The removal takes no device memory of its own, but for several modes with launches of one
    frame (16·K·N² bytes, once)."""
    cu = _driver()
    s = far_field(64, modes, 4, 128, seed=modes)
    scan = Scan(s["counts"], s["y"], s["x"], sim.WAVELENGTH, sim.DISTANCE, sim.DETECTOR_PIXEL)
    obj, probe = s["truth"], s["probe"] * (1 + 0.1j)
    with GpuPtycho(scan, obj, probe, stack_size=stack) as g:
        g.ap(0, zero_phase_ramp=False)
        used = _pool_used(cu)
        g.ap(0, zero_phase_ramp=True)
        want_obj, want_probe = zero_phase_ramp(obj.astype(np.complex64).astype(complex),
                                               probe.astype(np.complex64).astype(complex))
        assert rel_l2(g.probe(), want_probe) < 1e-6
        assert rel_l2(g.object(), want_obj) < 1e-6
        g.ap(0, zero_phase_ramp=True)
        more = _pool_used(cu) - used
    if own:
        assert 16 * modes * 64 ** 2 <= more < 17 * modes * 64 ** 2
    else:
        assert more == 0
