"""Reads between one-pass runs bring over the array that is read and no other:
every field and Psi slot alone, in any order, again, and mixed with saved states
and half-steps, has the values of a handle on the half-steps, bit for bit, and
leaves the run alone."""
import random

import numpy as np
import pytest

from conftest import load_package
from test_gpu_one_pass import FIELDS, SHAPES, _assert_same, _problem, _state

pkg = load_package()
from special_topics_b200.backend import Engine  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32-table"])
@pytest.mark.parametrize("shape", [SHAPES[q] for q in (1, 5)], ids=lambda s: "x".join(map(str, s[:3])))
def test_each_array_alone(shape, precision):
    _, p = _problem(shape)
    rng = random.Random(7)
    reads = [(f, None) for f in FIELDS] + [(q, s) for q, f in enumerate(p.cpml) for s in range(4) if f is not None]
    size = lambda q, s: p.cpml[q].cpsi[s].size  # noqa: E731
    with Engine(p, precision) as a, Engine(p, precision, half_steps=True) as b:
        for n in (3, 4, 5, 4, 3):
            a.run(n)
            b.run(n)
            rng.shuffle(reads)
            for q, s in reads[:9] + reads[:2]:
                x, y = (e.field(q) if s is None else e.psi(q, s, size(q, s)) for e in (a, b))
                assert np.array_equal(x, y), (q, s)
            if n == 5:
                a.load_state(a.save_state())
            a.half_steps = n == 4
        _assert_same(_state(b), _state(a))
