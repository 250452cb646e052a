"""Far-field pattern of a box with more rows of points than a grid's second axis
holds blocks (65,535), against postproc's FP64 host restatement on the same
accumulators.  The tolerance is that of the other pattern tests."""
import numpy as np
import pytest

from conftest import load_package
from scenarios_small import small_scenario

pkg = load_package()
from special_topics_b200 import postproc  # noqa: E402
from special_topics_b200.backend import Engine  # noqa: E402
from special_topics_b200.scenario import build_problem_from_scenario  # noqa: E402

pytestmark = pytest.mark.gpu


def test_a_long_thin_box():
    steps = 12
    scn = small_scenario(2, "yn", steps=steps)
    scn["boundary"]["air_buffer_xp"] += 33000
    p = build_problem_from_scenario(scn, steps, per_cell=False)
    th, ph = np.array([0.4, 1.3, 2.2]), np.array([0.1, 2.0, 5.0])
    with Engine(p, "f32-table") as eng:
        eng.run(steps)
        acc = eng.farfield()
        radp, dth, dph = eng.farfield_post(th, ph)
    want_p = postproc.radiated_power(acc, p.grid, p.farfield)
    want = postproc.directivity(acc, p.grid, p.farfield, want_p, th, ph)
    assert np.allclose(radp, want_p, rtol=1e-10, atol=0)
    for got, w in zip((dth, dph), want):
        assert np.abs(got - w).max() <= 1e-9 * np.abs(w).max()
