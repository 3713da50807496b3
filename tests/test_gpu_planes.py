"""The plane transforms (csrc/plane.cuh) at every cluster shape built for every side, with one mode
and the most that fit the cluster (four; three in the two shapes of 64 KB a mode): forward intensities, the Poisson gradients of object and
probe (forward and inverse), and the position gradients (moves and offset derivatives) of two
frames against the float64 oracle. Each is one pass of single-precision transforms: a rounding
error of about 1e-7·log2(N²) per transform, held to 1e-5 as the other single steps are."""
import numpy as np
import pytest

from oracle import ops
from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import far_field, oracle_state, rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("n,cluster,modes", [
    (n, cluster, modes) for n, cluster, most in [(64, 1, 4), (96, 2, 4), (128, 2, 3), (128, 4, 4),
                                                 (192, 8, 4), (256, 8, 3), (256, 16, 4)]
    for modes in (1, most)])
def test_one_pass_of_each_transform(n, cluster, modes):
    # the cluster is taken as asked for: its planes and tables fit a CTA's shared memory
    assert 8 * modes * n * n // cluster + 16 * n + 1280 <= 227 * 1024
    s = far_field(n, modes, 2, n + 45, photons=1e5, seed=n + modes, step=9.0)
    rng = np.random.default_rng(3)
    # a start near the truth everywhere: no detector pixel where 1 − I/model amplifies rounding
    s["counts"] = rng.poisson(20.0, s["counts"].shape).astype(np.float32)
    s["object"] = s["truth"]
    s["probe"] = 20.0 * (rng.normal(size=s["probe"].shape) + 1j * rng.normal(size=s["probe"].shape))
    d = rng.uniform(-0.7, 0.7, (2, 2))
    scan = Scan(s["counts"], s["y"], s["x"], sim.WAVELENGTH, sim.DISTANCE, sim.DETECTOR_PIXEL)
    cpu = oracle_state(s)
    want = ops.icalc_of(cpu.optics.exit_forward(cpu.calc_psi()), cpu.addr.nmode)
    go, gp = cpu.grads()
    with GpuPtycho(scan, s["object"], s["probe"], cluster=cluster) as g:
        assert rel_l2(g.forward_intensity(), want) < TOL
        got = g.gradients(positions=False)
        assert rel_l2(got["object"], go) < TOL
        assert rel_l2(got["probe"], gp) < TOL
        g.set_positions(d, refine=False)
        cpu.set_positions(d)
        go, gp = cpu.grads()
        got = g.gradients()
        assert rel_l2(got["object"], go) < TOL
        assert rel_l2(got["probe"], gp) < TOL
        # ∂L/∂d = Re⟨g, ∂ψ/∂d⟩ cancels: its bound is 1e-6 of ‖g‖·‖∂ψ/∂d‖ (Cauchy-Schwarz on
        # fields that each hold to a few 1e-7), not of the sum itself
        wave = cpu.shifted()
        g_norm = np.linalg.norm(cpu.grad_psi().reshape(2, -1), axis=1)
        bound = np.stack([g_norm * np.linalg.norm(wave.derivatives(cpu.object, a).reshape(2, -1),
                                                  axis=1) for a in (0, 1)], 1)
        assert (np.abs(got["positions"] - cpu.position_grad()) < 1e-6 * bound).all()
