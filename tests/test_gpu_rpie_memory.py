"""Where rPIE keeps a batch's object sums: a call after an LSQML call with the same batches takes
no more device memory (one mode: LSQML's direction arrays; more: the frames' planes that the
batches leave alone, with and without offsets), but for objects larger than those planes, where
several modes get arrays of their own once. Every place is held to the float64 oracle, one epoch,
at the run bound of the other rPIE tests."""
import numpy as np
import pytest

from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import far_field, oracle_state, rel_l2
from test_zz_no_alloc import _driver, _pool_used

pytestmark = pytest.mark.gpu

RUN_TOL = 1e-4


# probe modes, frames, object side; 12 frames of 64² x 2 hold the sums of 128² pixels beside a
# batch of 4 (64 k of 8 bytes against 12·2·16 k bytes), 2 frames hold none of 192²
@pytest.mark.parametrize("modes,nframe,side,own", [(1, 12, 192, False), (2, 12, 128, False),
                                                   (2, 2, 192, True), (4, 2, 192, True)])
@pytest.mark.parametrize("offsets", [False, True])
def test_sums_lie_in_memory_held_anyway(modes, nframe, side, own, offsets):
    cu = _driver()
    s = far_field(64, modes, nframe, side, seed=modes + 66, step=6.0)
    s["object"] = s["truth"] * 0.9 * np.exp(0.1j)
    cpu = oracle_state(s)
    scan = Scan(s["counts"], s["y"], s["x"], sim.WAVELENGTH, sim.DISTANCE, sim.DETECTOR_PIXEL)
    with GpuPtycho(scan, s["object"], s["probe"]) as g:
        if offsets:
            d = np.random.default_rng(4).uniform(-0.6, 0.6, (nframe, 2))
            g.set_positions(d, refine=False)
            cpu.set_positions(d)
        g.lsqml(1, batch_size=4, seed=7)
        g.set_object(s["object"])
        g.set_probe(s["probe"])
        cpu.cycle = g.cycle()
        used = _pool_used(cu)
        g.rpie(1, batch_size=4, seed=7)
        cpu.rpie(1, batch_size=4, seed=7)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL
        g.rpie(1, batch_size=4, seed=7)
        more = _pool_used(cu) - used
    if own:
        assert 12 * modes * side * side <= more < 13 * modes * side * side
    else:
        assert more == 0
