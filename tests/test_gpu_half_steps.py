"""The half-step kernels, which serve what the one-pass step does not (bands that
meet, too many cell classes, little memory), in every form that a handle or a
batch can ask for: fdtd_ctx_set_step_path keeps a handle on them, a batch's tile
group or members per launch a batch.  A profile says which kernels ran: only the
half-steps have an E launch.  FP64 against the oracle, FP32 against the one-pass
step, bit for bit: every path does the same roundings in the same order.
"""
import numpy as np
import pytest

import oracle
from conftest import load_package
from test_gpu_one_pass import FIELDS, SHAPES, STEPS, _assert_same, _problem, _state

pkg = load_package()
from special_topics_b200 import _native as N, autotune  # noqa: E402
from special_topics_b200.backend import Batch, Engine  # noqa: E402

pytestmark = pytest.mark.gpu


def _profile_to_end(target, step):
    """The last two steps, profiled: their E launches' time."""
    target.run(STEPS - 2 - step)
    return target.profile_kernels(2)["e"]


@pytest.mark.parametrize("chunk,rows,pf,width", [(1, 4, 1, 32), (7, 2, 1, 32), (64, 8, 1, 32), (5, 4, 2, 32), (25, 2, 2, 32),
                                                 (4, 2, 1, 16), (5, 16, 2, 16), (1, 8, 1, 16)])
def test_fp64_shapes_match_oracle(chunk, rows, pf, width):
    scn, p = _problem(SHAPES[0])
    o = oracle.Oracle(scn, STEPS)
    o.step(STEPS)
    with Engine(p, "f64", half_steps=True) as eng:
        autotune.set_tiling(eng, min(chunk, p.grid.nx + 1), rows, pf, width)
        assert eng.half_steps and _profile_to_end(eng, 0) > 0
        got = _state(eng)
    for f in FIELDS:
        assert np.array_equal(got[f], o.get(f)), f
    assert np.array_equal(got["V0"], o.get("V:0")) and np.array_equal(got["I0"], o.get("I:0"))


@pytest.mark.parametrize("precision,chunk,rows,pf,width",
                         [("f32-table", *s) for s in ((5, 2, 3, 32), (16, 8, 4, 32), (1, 4, 4, 32), (64, 2, 3, 32),
                                                      (3, 8, 2, 32), (8, 4, 1, 16), (6, 16, 3, 16), (16, 2, 4, 16),
                                                      (8, 4, 5, 32), (1, 2, 5, 32), (64, 8, 5, 32))] +
                         [("f32", *s) for s in ((8, 4, 1, 32), (3, 8, 2, 32), (5, 16, 1, 16))])
def test_fp32_shapes_match_the_one_pass_step(precision, chunk, rows, pf, width):
    """Prefetch 1, 2: planes in registers; 3, 4: staged; 5: staged by bulk copies."""
    _, p = _problem(SHAPES[4])
    with Engine(p, precision) as eng:
        assert _profile_to_end(eng, 0) == 0
        want = _state(eng)
    with Engine(p, precision) as eng:
        eng.run(3)
        eng.half_steps = True            # from here on
        autotune.set_tiling(eng, min(chunk, p.grid.nx + 1), rows, pf, width)
        assert _profile_to_end(eng, 3) > 0
        _assert_same(want, _state(eng))


@pytest.mark.parametrize("precision", ["f64", "f32-table"])
@pytest.mark.parametrize("group,per_launch,half", [(0, 0, True), (3, 0, False), (0, 2, False), (1, 0, True), (0, 3, True)])
@pytest.mark.parametrize("chunk,rows,pf,width", [(8, 4, 1, 32), (5, 16, 2, 16), (1024, 2, 1, 32)])
def test_batch_modes_match_members_alone(precision, group, per_launch, half, chunk, rows, pf, width):
    """A tile group or members per launch select their mode; without them a member
    on the half-steps keeps the batch from chains."""
    probs = [_problem(SHAPES[q])[1] for q in (0, 3, 6)]
    want = []
    for p in probs:
        with Engine(p, precision) as eng:
            eng.run(STEPS)
            want.append(_state(eng))
    engs = [Engine(p, precision, half_steps=half and not q) for q, p in enumerate(probs)]
    try:
        with Batch(engs) as b:
            if not half:
                b.run(2)                 # as chains
            b.set_tiling(chunk, rows, pf, group, width=width, per_launch=per_launch)
            assert _profile_to_end(b, 0 if half else 2) > 0
        for w, e in zip(want, engs):
            _assert_same(w, _state(e))
    finally:
        for e in engs:
            e.close()


def test_the_path_is_set_between_runs():
    _, p = _problem(SHAPES[0])
    with Engine(p, "f32-table") as eng:
        eng.run(STEPS)
        want = _state(eng)
    with Engine(p, "f32-table") as eng:
        for q, half in enumerate((True, False, True, False)):
            eng.half_steps = half
            assert eng.half_steps == half and (eng.profile_kernels(2)["e"] > 0) == half
            eng.run(q)
        eng.run(STEPS - 14)
        _assert_same(want, _state(eng))
        with pytest.raises(N.FdtdError) as ei:
            N.check(N.lib().fdtd_ctx_set_step_path(eng._h, 2))
        assert ei.value.code == N.FDTD_ERR_BADARG


def test_the_tuner_times_what_runs(tmp_path, monkeypatch):
    """One row where the one-pass step serves; batches time its chains once."""
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tiling.json"))
    from scenarios_small import small_scenario
    from special_topics_b200.scenario import build_problem_from_scenario
    p = build_problem_from_scenario(small_scenario(6, "xp"), 3000, per_cell=False)
    res = autotune.tune(p, "f32-table", steps_per_candidate=8)
    assert res["one_pass"] and len(res["table"]) == 1
    engs = [Engine(p, "f32-table") for _ in range(2)]
    try:
        with Batch(engs) as b:
            res = autotune.tune_batch(b, steps_per_candidate=4)
            assert b.step <= autotune.batch_steps_needed(4)
            assert sum(r["chains"] for r in res["table"]) == 1 and len({r["streams"] for r in res["table"]}) > 3
            assert (b.profile_kernels(1)["e"] == 0) == (res["chains"] or res["streams"] == 0 and not res["group"] and not res["per_launch"])
    finally:
        for e in engs:
            e.close()
