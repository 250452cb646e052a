"""Far-field patterns from row sums (csrc/fdtd_ffpost.cuh): boxes with rows of
odd and even length, longer than the pairs staged at a time, direction lists
with one theta, all thetas different, grids in both orders, and enough thetas for
two runs, against postproc's FP64 host restatement on the same accumulators.
The tolerance is the accumulated rounding of at most a few thousand FP64 terms,
as for the other pattern test.
"""
import numpy as np
import pytest

from conftest import load_package
from scenarios_small import small_scenario

pkg = load_package()
from special_topics_b200 import postproc  # noqa: E402
from special_topics_b200.backend import Engine  # noqa: E402
from special_topics_b200.scenario import build_problem_from_scenario  # noqa: E402

pytestmark = pytest.mark.gpu
STEPS = 40


def _close(got, want):
    assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max()


@pytest.fixture(scope="module", params=[(0, 0), (1, 2), (150, 151)], ids=str)
def engine(request):
    """Rows along y and z longer by (dy, dz) cells."""
    scn = small_scenario(4, "yn", steps=STEPS)
    scn["boundary"]["air_buffer_yp"] += request.param[0]
    scn["boundary"]["air_buffer_zp"] += request.param[1]
    with Engine(build_problem_from_scenario(scn, STEPS), "f64") as eng:
        eng.run(STEPS)
        yield eng, eng.farfield()


def _host(eng, acc, th, ph):
    p = eng.problem
    radp = postproc.radiated_power(acc, p.grid, p.farfield)
    return radp, *postproc.directivity(acc, p.grid, p.farfield, radp, th, ph)


@pytest.mark.parametrize("kind", ["one", "cut", "random", "grid", "grid-phi-first"])
def test_directions_of_every_form(engine, kind):
    eng, acc = engine
    rng = np.random.default_rng(1)
    th, ph = {
        "one": lambda: (np.array([0.7]), np.array([2.1])),
        "cut": lambda: (np.full(37, np.pi / 2), np.radians(np.arange(37) * 10.0)),
        "random": lambda: (rng.uniform(0, np.pi, 131), rng.uniform(0, 2 * np.pi, 131)),
        "grid": lambda: tuple(a.ravel() for a in np.meshgrid(np.linspace(0, np.pi, 9), np.linspace(0, 6, 15), indexing="ij")),
        "grid-phi-first": lambda: tuple(a.ravel() for a in np.meshgrid(np.linspace(0, np.pi, 9), np.linspace(0, 6, 15))),
    }[kind]()
    radp, dth, dph = eng.farfield_post(th, ph)
    want = _host(eng, acc, th, ph)
    assert np.allclose(radp, want[0], rtol=1e-10, atol=0)
    _close(dth, want[1])
    _close(dph, want[2])


def test_many_thetas_in_runs():
    scn = small_scenario(4, "yn", steps=STEPS)
    with Engine(build_problem_from_scenario(scn, STEPS), "f64") as eng:
        eng.run(STEPS)
        th = np.linspace(0, np.pi, 170001)
        ph = np.linspace(0, 40, th.size)
        _, dth, dph = eng.farfield_post(th, ph)
        for part in (slice(0, 40), slice(th.size // 2, th.size // 2 + 40), slice(th.size - 40, None)):
            _, a, b = eng.farfield_post(th[part], ph[part])
            scale = np.abs(dth).max() + np.abs(dph).max()
            assert np.abs(dth[:, part] - a).max() <= 1e-12 * scale and np.abs(dph[:, part] - b).max() <= 1e-12 * scale
