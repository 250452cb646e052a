"""The one-pass step (csrc/fdtd_fused.cuh) where its tiles can go wrong: rows
that end at, before and after a tile (68 and 72 columns, 6 rows), chunks of one
plane to all of them, band widths that split a group of columns, odd run
lengths.  FP64 against the oracle, FP32 against the engine's half-step kernels
(a batch of one on member streams), both bit for bit: each path does the same
roundings in the same order, so the tolerance is zero.
"""
import numpy as np
import pytest

import oracle
from conftest import load_package
from scenarios_small import small_scenario

pkg = load_package()
from special_topics_b200.backend import Batch, Engine  # noqa: E402
from special_topics_b200.scenario import FF_NAMES, build_problem_from_scenario  # noqa: E402

pytestmark = pytest.mark.gpu

FIELDS = ("Hx", "Hy", "Hz", "Ex", "Ey", "Ez")
STEPS = 23

# (nx, ny, nz, CPML cells on xn xp yn yp zn zp)
SHAPES = [
    (24, 25, 70, (4, 5, 3, 6, 4, 3)),
    (23, 26, 71, (3, 3, 5, 5, 5, 4)),      # one whole k tile
    (25, 27, 72, (1, 2, 7, 1, 3, 8)),      # a second k tile for one column
    (26, 29, 73, (5, 4, 6, 3, 8, 1)),
    (25, 30, 135, (4, 4, 4, 4, 7, 6)),     # two whole k tiles
    (26, 31, 136, (2, 6, 6, 6, 6, 5)),
    (90, 25, 27, (8, 9, 3, 3, 2, 2)),      # many x chunks
]


def _problem(shape):
    nx, ny, nz, nc = shape
    scn = small_scenario(sum(shape[:3]), ("xp", "yn", "zp")[nz % 3], ncpml=nc, steps=STEPS)
    g = build_problem_from_scenario(scn, STEPS).grid
    for a, (n, n0) in enumerate(zip((nx, ny, nz), (g.nx, g.ny, g.nz))):
        scn["boundary"][f"air_buffer_{'xyz'[a]}p"] += n - n0
        assert scn["boundary"][f"air_buffer_{'xyz'[a]}p"] >= 1
    scn["farfield"]["number_of_cells_from_outer_boundary"] = 4
    p = build_problem_from_scenario(scn, STEPS)
    assert (p.grid.nx, p.grid.ny, p.grid.nz) == (nx, ny, nz)
    return scn, p


def _state(eng):
    out = {f: eng.field(f) for f in FIELDS}
    for q, v in enumerate(eng.voltages()):
        out[f"V{q}"] = v
    for q, v in enumerate(eng.currents()):
        out[f"I{q}"] = v
    for name, (re, im) in eng.farfield().items():
        out[name + " re"], out[name + " im"] = re, im
    for fid, f in enumerate(eng.problem.cpml):
        for s in range(4):
            if f is not None and f.cpsi is not None:
                out[f"psi{fid}:{s}"] = eng.psi(fid, s, f.cpsi[s].size)
    return out


def _assert_same(a, b):
    assert a.keys() == b.keys()
    for key in a:
        assert np.array_equal(a[key], b[key]), key


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[:3])))
def test_fp64_one_pass_matches_oracle(shape):
    scn, p = _problem(shape)
    o = oracle.Oracle(scn, STEPS)
    o.step(STEPS)
    with Engine(p, "f64") as eng:
        eng.run(1)
        eng.run(8)
        eng.field("Ez")                  # a read between runs leaves the state alone
        eng.run(STEPS - 9)
        got = _state(eng)
    for f in FIELDS:
        assert np.array_equal(got[f], o.get(f)), f
    assert np.array_equal(got["V0"], o.get("V:0")) and np.array_equal(got["I0"], o.get("I:0"))
    for fid in range(6):
        for s in range(4):
            assert np.array_equal(got[f"psi{fid}:{s}"], o.get(f"psi:{fid}:{s}")), (fid, s)
    for a in FF_NAMES:
        assert np.array_equal(got[a + " re"], o.get(f"ff:{a}:0")) and np.array_equal(got[a + " im"], o.get(f"ff:{a}:1")), a


@pytest.mark.parametrize("precision", ["f32", "f32-table"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[:3])))
def test_fp32_one_pass_matches_half_steps(shape, precision):
    _, p = _problem(shape)
    for x_wall in (True, False):
        with Engine(p, precision, x_wall=x_wall) as eng, Batch([eng], streams=1) as b:
            b.run(STEPS)
            want = _state(eng)
        with Engine(p, precision, x_wall=x_wall) as eng:
            eng.run(10)
            saved = eng.save_state()
            eng.run(3)
            eng.load_state(saved)        # back to step 10, with both copies of the state stale
            with Batch([eng], streams=1) as b:
                b.run(2)                 # half-steps in between
            eng.run(STEPS - 12)
            _assert_same(want, _state(eng))


@pytest.mark.parametrize("members", [2, 5, 24])
def test_chunks_of_any_length_match(members):
    """A member's share of the device, and so the x planes of its blocks, depends
    on how many there are."""
    _, p = _problem(SHAPES[6])
    with Engine(p, "f32-table") as eng:
        eng.run(STEPS)
        want = _state(eng)
    engs = [Engine(p, "f32-table") for _ in range(members)]
    try:
        with Batch(engs) as b:
            b.run(STEPS)
        for e in (engs[0], engs[-1]):
            _assert_same(want, _state(e))
    finally:
        for e in engs:
            e.close()


@pytest.mark.parametrize("blocks", [(0, 0, 0), (4, 4, 4), (0, 4, 3)], ids=str)
@pytest.mark.parametrize("group,per_launch", [(0, 0), (2, 0), (0, 2)])
def test_batch_chains_match_members_alone(blocks, group, per_launch):
    """Members at different copies of their state; DFT blocks of one length
    (chains) and of several (tile list, persistent grid, grouped launches)."""
    probs = [_problem(SHAPES[q])[1] for q in (0, 3, 6)]
    want = []
    for p, d in zip(probs, blocks):
        with Engine(p, "f32-table", dft_block=d) as eng:
            eng.run(STEPS)
            want.append(_state(eng))
    engs = [Engine(p, "f32-table", dft_block=d) for p, d in zip(probs, blocks)]
    try:
        engs[1].run(1)
        engs[0].run(1)
        with Batch([engs[2]]) as b:
            b.run(1)
        engs[0].load_state(engs[0].save_state())
        with Batch(engs, group=group) as b:
            b.set_tiling(8, 4, 1, group, per_launch=per_launch)
            b.run(6)
            b.run(5)
            engs[1].field("Hx")
            b.run(STEPS - 12)
        for w, e in zip(want, engs):
            _assert_same(w, _state(e))
    finally:
        for e in engs:
            e.close()


@pytest.mark.parametrize("freqs,block,runs", [(1, 2, (5, 18)), (3, 6, (8, 15)), (7, 4, (4, 19)), (8, 33, (23,)), (9, 5, (1, 1, 21)), (17, 7, (9, 14))])
def test_blocked_dft_sums_in_step_order(freqs, block, runs):
    """Compensated FP32 sums are the same bits whether a step's samples are
    added at once or with their block: frequency groups of 8 full and ragged,
    point groups of 32 ragged, blocks closed by a run's end, longer than a run
    and longer than the phasors staged at a time."""
    scn, _ = _problem(SHAPES[1])
    scn["farfield"]["frequencies"] = [1e9 * (2 + q) for q in range(freqs)]
    p = build_problem_from_scenario(scn, STEPS)
    out = []
    for b in (0, block):
        with Engine(p, "f32-table", dft_accumulator="kahan-f32", dft_block=b) as eng:
            for n in runs:
                eng.run(n)
            out.append(eng.farfield())
    for a in FF_NAMES:
        assert np.array_equal(out[0][a][0], out[1][a][0]) and np.array_equal(out[0][a][1], out[1][a][1]), a


def test_memory_held_for_speed_is_given_back():
    """A problem that fits beside another's fields, but not beside the padded
    copies that the other keeps, is accepted, and both go on with the same
    results.  (The rest of the device's memory is taken, so that neither fits
    twice: 128^3 keeps some 110 MB of padded copies, 144^3 needs some 95 MB.)"""
    import torch
    from special_topics_b200.workloads import scaling_box
    probs = [build_problem_from_scenario(scaling_box((n, n, n), seed=3, steps=STEPS), STEPS, per_cell=False)
             for n in (128, 144)]
    want = []
    for p in probs:
        with Engine(p, "f32-table") as eng:
            eng.run(STEPS)
            want.append(_state(eng))
    with Engine(probs[0], "f32-table") as a:
        a.run(9)
        free, _ = torch.cuda.mem_get_info()
        rest = torch.empty(free - (80 << 20), dtype=torch.uint8, device="cuda")
        try:
            with Engine(probs[1], "f32-table") as b:
                b.run(STEPS)
                _assert_same(want[1], _state(b))
            a.run(STEPS - 9)
            _assert_same(want[0], _state(a))
        finally:
            del rest
            torch.cuda.empty_cache()
