"""A run that goes on after an infinite source sample: the one-pass step leaves
what the half-steps leave alone (the walls, the cells beside a CPML band), so
fields, Psi, traces and far field are the same values, infinities and NaN in the
same places.  Both paths do the same roundings in the same order: the tolerance
is zero.
"""
import numpy as np
import pytest

from conftest import load_package
from test_gpu_one_pass import SHAPES, _problem, _state

pkg = load_package()
from special_topics_b200 import _native as N  # noqa: E402
from special_topics_b200.backend import Batch, Engine  # noqa: E402
from special_topics_b200.scenario import build_problem_from_scenario  # noqa: E402

pytestmark = pytest.mark.gpu
STEPS = 70


def _diverged(run, eng):
    with pytest.raises(N.FdtdError) as ei:
        run(STEPS)
    assert ei.value.code == N.FDTD_ERR_NONFINITE
    return _state(eng)


@pytest.mark.parametrize("precision", ["f64", "f32", "f32-table"])
@pytest.mark.parametrize("shape", [SHAPES[q] for q in (1, 3, 5)], ids=lambda s: "x".join(map(str, s[:3])))
def test_an_infinite_sample_spreads_as_in_the_half_steps(shape, precision):
    p = build_problem_from_scenario(_problem(shape)[0], STEPS)
    p.voltage_sources[0].voltage_per_e_field[3] = np.inf
    for x_wall in (True, False):
        with Engine(p, precision, x_wall=x_wall) as eng, Batch([eng], streams=1) as b:
            want = _diverged(b.run, eng)
        with Engine(p, precision, x_wall=x_wall) as eng:
            got = _diverged(eng.run, eng)
        assert np.isnan(want["Ez"]).any()
        for key in want:
            assert np.array_equal(want[key], got[key], equal_nan=True), (x_wall, key)
