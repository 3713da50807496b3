"""The per-kernel times name what an rPIE call launches: frame passes, the sums (object and probe
together) with their frames, the updates, and nothing else."""
import pytest

from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import far_field

pytestmark = pytest.mark.gpu


def test_names_of_an_rpie_call():
    s = far_field(64, 1, 10, 128, seed=1, step=5.0)
    scan = Scan(s["counts"], s["y"], s["x"], sim.WAVELENGTH, sim.DISTANCE, sim.DETECTOR_PIXEL)
    with GpuPtycho(scan, s["object"], s["probe"]) as g:
        g.set_timing(True)
        g.rpie(2, batch_size=4)
        times, frames = g.kernel_times(), g.kernel_frames()
    assert {k: n for k, (_, n) in times.items()} == {"frame_rpie": 6, "rpie_sums": 6,
                                                     "rpie_updates": 6}
    assert frames == {"frame_rpie": 20, "rpie_sums": 20}
