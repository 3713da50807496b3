"""Host logic of the bench (no GPU): its kernels' byte counts, and of its time-to-target leg the
LLK records to per-iteration traces and the reference's two-target rule."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


def test_llk_after_drops_the_ml_start_record():
    assert bench.llk_after("ml", [9.0, 5.0, 4.0]) == [5.0, 4.0]
    assert bench.llk_after("rpie", [5.0, 4.0]) == [5.0, 4.0]


def test_first_target_when_every_algorithm_reaches_it():
    traces = {"a": [3.0, 2.0, 1.0], "b": [2.5, 1.005, 1.001]}
    (t, iters), = bench.ttt_targets(traces)
    assert t == 1.01 * 1.0
    assert iters == {"a": 3, "b": 2}


def test_second_target_from_the_highest_final_that_misses_the_first():
    traces = {"rpie": [3.0, 2.0, 1.5, 1.4], "lsqml": [2.0, 1.2, 1.1], "ml": [2.0, 1.3, 1.0]}
    targets = bench.ttt_targets(traces)
    assert len(targets) == 2
    (t1, i1), (t2, i2) = targets
    assert i1 == {"rpie": None, "lsqml": None, "ml": 3}
    assert t2 == 1.01 * 1.4
    assert i2 == {"rpie": 4, "lsqml": 2, "ml": 2}


def test_a_diverged_run_sets_no_target():
    nan = float("nan")
    traces = {"rpie": [5.0, 1e9, nan], "lsqml": [2.0, 1.2, 1.1], "ml": [2.0, 1.3, 1.0]}
    targets = bench.ttt_targets(traces)
    assert len(targets) == 2
    (t1, i1), (t2, i2) = targets
    assert t1 == 1.01 * 1.0 and i1 == {"rpie": None, "lsqml": None, "ml": 3}
    assert t2 == 1.01 * 1.1 and i2 == {"rpie": None, "lsqml": 3, "ml": 3}


def test_rpie_bytes_are_those_of_its_launches():
    """rPIE's sums (object and probe in one launch) have their bytes under the name that the
    library times them by; the updates run over object and probe pixels, not frames."""
    from ptyrs_b200 import _lib, build
    build.build()
    lib = _lib.load()
    names = {lib.ptyb_kernel_name(i).decode() for i in range(lib.ptyb_kernel_kinds())}
    assert {"frame_rpie", "rpie_sums", "rpie_updates"} <= names and "object_rpie" not in names
    s = dict(n=64, probe=np.ones((2, 64, 64)), object=np.ones((1, 256, 256)))
    wl = dict(algorithm="rpie")
    assert bench.algorithmic_bytes("rpie_sums", s, wl) == (2 * 8 + 8) * 64 ** 2
    assert bench.algorithmic_bytes("rpie_updates", s, wl) is None
    assert bench.algorithmic_bytes("object_rpie", s, wl) is None
