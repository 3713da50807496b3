"""Kernel instances that the other suites' shapes do not reach, against the float64 oracle at their
bounds (one batch 1e-5 where it is a single step, runs 1e-4): the clusters that only the `cluster`
option picks (2 CTAs a frame at 128², 8 at 256²), four probe modes through rPIE, LSQML, DM and the
gathers behind them, and launches of more frames than a gather lists at a time (512) or the
position step takes at a time (1024)."""
import numpy as np
import pytest

from oracle.lsqml import Lsqml
from ptyrs_b200 import GpuPtycho, Scan, sim
from scenarios import far_field, oracle_state, rel_l2
from test_gpu_multislice import gpu_of as slices_gpu_of
from test_gpu_multislice import lsqml_cpu as slices_lsqml_cpu
from test_gpu_multislice import multislice_scan

pytestmark = pytest.mark.gpu

ONE_STEP_TOL = 1e-5
RUN_TOL = 1e-4


def gpu_of(s, **kw):
    scan = Scan(s["counts"], s["y"], s["x"], sim.WAVELENGTH, sim.DISTANCE, sim.DETECTOR_PIXEL)
    return GpuPtycho(scan, s["object"], s["probe"], **kw)


def assert_offsets(got, cpu_offsets, d0):
    moved = cpu_offsets - d0
    assert np.abs(moved).max() > 0
    assert np.abs((got - d0) - moved).max() <= RUN_TOL * 10 * np.abs(moved).max()


def assert_lsqml(s, g, batch, cost):
    """One LSQML epoch: every step size, the object and the probe."""
    cpu = oracle_state(s)
    obj, probe, steps = Lsqml(batch, cost, 7).epoch(cpu.addr, cpu.obs, cpu.optics, cpu.object,
                                                    cpu.probe)
    g.lsqml(1, batch_size=batch, cost=cost, seed=7)
    got = g.lsqml_steps()
    assert [x["frames"] for x in got] == [x["frames"] for x in steps]
    for gs, cs in zip(got, steps):
        for key in ("a_far", "a_obj", "a_probe"):
            a, b = np.array(gs[key]), np.array(cs[key])
            assert np.abs(a - b).max() <= RUN_TOL * np.abs(b).max() + 1e-30, key
    assert rel_l2(g.object(), obj) < RUN_TOL
    assert rel_l2(g.probe(), probe) < RUN_TOL


# (frame side, CTAs a frame, probe modes, frames, object side)
OPTION_CLUSTERS = [(128, 2, 3, 12, 256), (256, 8, 2, 8, 416)]


@pytest.fixture(scope="module", params=OPTION_CLUSTERS, ids=lambda p: f"n{p[0]}c{p[1]}")
def option_cluster(request):
    n, cluster, k, nframe, side = request.param
    # the planes of every mode fit the CTA's shared memory: the option is taken, not replaced
    assert 8 * k * n * n // cluster + 16 * n + 1280 <= 227 * 1024
    s = far_field(n, k, nframe, side, masked=True, seed=n + k)
    s["object"] = s["truth"] * 0.9 * np.exp(0.1j)
    return s, cluster


def test_rpie_at_option_clusters(option_cluster):
    """One batch on the shared probe, then an epoch refining offsets (moves forward and back, the
    window derivatives)."""
    s, cluster = option_cluster
    nframe = len(s["counts"])
    cpu = oracle_state(s)
    cpu.rpie(1, batch_size=nframe, seed=7)
    with gpu_of(s, cluster=cluster) as g:
        g.rpie(1, batch_size=nframe, seed=7)
        assert rel_l2(g.object() - s["object"], cpu.object - s["object"]) < ONE_STEP_TOL
        assert rel_l2(g.probe() - s["probe"], cpu.probe - s["probe"]) < ONE_STEP_TOL
    d0 = np.random.default_rng(7).uniform(-0.6, 0.6, (nframe, 2))
    cpu = oracle_state(s)
    cpu.set_positions(d0, refine=True)
    cpu.rpie(1, batch_size=5, seed=7)
    with gpu_of(s, cluster=cluster) as g:
        g.set_positions(d0, refine=True)
        g.rpie(1, batch_size=5, seed=7)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL
        assert_offsets(g.positions(), cpu.offsets, d0)


@pytest.mark.parametrize("cost", ["poisson", "amplitude"])
def test_lsqml_at_option_clusters(option_cluster, cost):
    s, cluster = option_cluster
    with gpu_of(s, cluster=cluster) as g:
        assert_lsqml(s, g, 5, cost)


@pytest.mark.parametrize("algorithm,kw", [("ap", dict(probe_inertia=0.001)), ("dm", {}),
                                          ("raar", {})])
def test_carried_at_option_clusters(option_cluster, algorithm, kw):
    s, cluster = option_cluster
    cpu = oracle_state(s)
    getattr(cpu, algorithm)(3, calc_llk=1, zero_phase_ramp=False, **kw)
    with gpu_of(s, cluster=cluster) as g:
        getattr(g, algorithm)(3, calc_llk=1, zero_phase_ramp=False, **kw)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL
        want = np.array([r["poisson"] for r in cpu.history])
        assert np.abs(g.history()["poisson"] - want).max() <= RUN_TOL * np.abs(want).max()


def test_ml_at_option_clusters(option_cluster):
    """Two cycles refining offsets: gradients, projection of the kept field, position sums and the
    line search."""
    s, cluster = option_cluster
    d0 = np.random.default_rng(8).uniform(-0.6, 0.6, (len(s["counts"]), 2))
    cpu = oracle_state(s)
    cpu.set_positions(d0, refine=True)
    cpu.ml(2, update_probe=True, zero_phase_ramp=False)
    with gpu_of(s, cluster=cluster) as g:
        g.set_positions(d0, refine=True)
        g.ml(2, update_probe=True, zero_phase_ramp=False)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL
        assert_offsets(g.positions(), cpu.offsets, d0)


@pytest.mark.parametrize("n,cluster,side,gaps", [(128, 2, 256, (1e-6, 1.5e-6)),
                                                 (256, 8, 416, (0.4e-6, 0.6e-6))])
@pytest.mark.parametrize("cost", ["poisson", "amplitude"])
def test_slices_at_option_clusters(n, cluster, side, gaps, cost):
    s = multislice_scan(n, 2, 8, side, gaps, seed=n)
    cpu, run, objs, probe, _ = slices_lsqml_cpu(s, 1, 5, cost)
    with slices_gpu_of(s, cluster=cluster) as g:
        g.lsqml(1, batch_size=5, cost=cost, seed=7)
        got = g.objects()
        for k in range(3):
            assert rel_l2(got[k] - 1.0, objs[k][0] - 1.0) < RUN_TOL, k
        assert rel_l2(g.probe(), probe) < RUN_TOL
        ref = run.llk(cpu.addr, cpu.obs, cpu.optics, objs, probe)
        assert abs(g.llk()["poisson"] - ref.poisson) <= RUN_TOL * abs(ref.poisson)


# (frame side, frames, object side) of the four-mode cases: one and four CTAs a frame
FOUR_MODES = [(64, 24, 160), (128, 12, 256)]


@pytest.fixture(scope="module", params=FOUR_MODES, ids=lambda p: f"n{p[0]}")
def four_modes(request):
    n, nframe, side = request.param
    s = far_field(n, 4, nframe, side, masked=True, seed=n + 4)
    s["object"] = s["truth"] * 0.9 * np.exp(0.1j)
    assert s["probe"].shape[0] == 4
    return s


@pytest.mark.parametrize("step", [dict(), dict(obj_step=None), dict(probe_step=None)],
                         ids=["both", "probe", "object"])
@pytest.mark.parametrize("offsets", [False, True], ids=["shared", "moved"])
def test_rpie_of_four_modes(four_modes, step, offsets):
    """Both updates, the probe's alone and the object's alone (an array without its step stays
    bit for bit)."""
    s = four_modes
    cpu = oracle_state(s)
    d0 = np.random.default_rng(7).uniform(-0.6, 0.6, (len(s["counts"]), 2))
    if offsets:
        cpu.set_positions(d0)
    cpu.rpie(1, batch_size=7, seed=3, **step)
    with gpu_of(s) as g:
        if offsets:
            g.set_positions(d0, refine=False)
        g.rpie(1, batch_size=7, seed=3, **step)
        if "obj_step" in step:
            assert np.array_equal(g.object(), s["object"].astype(np.complex64).astype(complex))
        if "probe_step" in step:
            assert np.array_equal(g.probe(), s["probe"].astype(np.complex64).astype(complex))
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL


@pytest.mark.parametrize("cost", ["poisson", "amplitude"])
def test_lsqml_of_four_modes(four_modes, cost):
    with gpu_of(four_modes) as g:
        assert_lsqml(four_modes, g, 7, cost)


def test_dm_of_four_modes(four_modes):
    cpu = oracle_state(four_modes)
    cpu.dm(3, zero_phase_ramp=False)
    with gpu_of(four_modes) as g:
        g.dm(3, zero_phase_ramp=False)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL


def test_rpie_holds_the_probe_without_its_step():
    """One mode, whole batches of three: the object's blocks of the updates alone."""
    s = far_field(64, 1, 12, 160, masked=True, seed=5)
    cpu = oracle_state(s)
    cpu.rpie(1, probe_step=None, batch_size=5, seed=3)
    with gpu_of(s) as g:
        g.rpie(1, probe_step=None, batch_size=5, seed=3)
        assert np.array_equal(g.probe(), s["probe"].astype(np.complex64).astype(complex))
        assert rel_l2(g.object(), cpu.object) < RUN_TOL


@pytest.fixture(scope="module")
def many_frames():
    """1100 frames of 64² x 2 on a dense spiral: every tile's list spans several chunks, the
    innermost with more than 512 views."""
    s = far_field(64, 2, 1100, 224, seed=12, step=2.0)
    s["object"] = s["truth"] * 0.9 * np.exp(0.1j)
    oy, ox = s["corners"][:, 0], s["corners"][:, 1]
    assert ((oy <= 112) & (oy + 64 > 112) & (ox <= 112) & (ox + 64 > 112)).sum() > 512
    return s


def test_rpie_batch_of_1100_frames(many_frames):
    s = many_frames
    d0 = np.random.default_rng(7).uniform(-0.6, 0.6, (len(s["counts"]), 2))
    cpu = oracle_state(s)
    cpu.set_positions(d0, refine=True)
    cpu.rpie(1, batch_size=1100, seed=7)
    with gpu_of(s) as g:
        g.set_positions(d0, refine=True)
        g.rpie(1, batch_size=1100, seed=7)
        assert rel_l2(g.object() - s["object"], cpu.object - s["object"]) < RUN_TOL
        assert rel_l2(g.probe() - s["probe"], cpu.probe - s["probe"]) < RUN_TOL
        assert_offsets(g.positions(), cpu.offsets, d0)
    cpu = oracle_state(s)
    cpu.rpie(1, batch_size=1100, seed=7)
    with gpu_of(s) as g:
        g.rpie(1, batch_size=1100, seed=7)
        assert rel_l2(g.object() - s["object"], cpu.object - s["object"]) < ONE_STEP_TOL
        assert rel_l2(g.probe() - s["probe"], cpu.probe - s["probe"]) < ONE_STEP_TOL


def test_lsqml_batches_of_550_frames(many_frames):
    with gpu_of(many_frames) as g:
        assert_lsqml(many_frames, g, 550, "poisson")


def test_gradients_and_blend_of_1100_frames(many_frames):
    """ML's gradient in stacks of 512 frames and of the whole scan, and two AP cycles, whose blend
    gathers every frame in one launch."""
    s = many_frames
    cpu = oracle_state(s)
    go, gp = cpu.grads()
    for stack in (0, 1100):
        with gpu_of(s, stack_size=stack) as g:
            got = g.gradients(positions=False)
            assert rel_l2(got["object"], go) < ONE_STEP_TOL
            assert rel_l2(got["probe"], gp) < ONE_STEP_TOL
    cpu.ap(2, probe_inertia=0.001, zero_phase_ramp=False)
    with gpu_of(s) as g:
        g.ap(2, probe_inertia=0.001, zero_phase_ramp=False)
        assert rel_l2(g.object(), cpu.object) < RUN_TOL
        assert rel_l2(g.probe(), cpu.probe) < RUN_TOL
