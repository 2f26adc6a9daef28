"""Calls that find too little device memory for what only saves time: they take the slower way, give the
same results and leave no buffer to others while a kernel still writes it."""
import pytest

import short_memory

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so(tmp_path_factory):
    return short_memory.build(str(tmp_path_factory.mktemp("short")))


def test_field_points_left_out_pair_set_is_idle_when_given_back(so):
    """Infinite depth: the points' Rankine tables are being filled when the allocation of their influences
    fails; the stream is waited for before the tables go back to the cache."""
    got = short_memory.run(so, """
geom = deck([meshgen.cylinder(5.0, 10.0, 18, 9, 4)])
n, m, beta = 234, 20000, [0.3]
rng = np.random.default_rng(1)
p = np.column_stack([rng.uniform(8.0, 40.0, m), rng.uniform(-30.0, 30.0, m), -rng.uniform(0.5, 30.0, m)])
want = None
for short in (False, True):
    ctx = hams_b200.Context(geom, -1.0, rho=1025.0, g=9.81)
    w = ctx.wave(0.9)
    mem.short_memory_reset()
    if short:
        hams_b200.release_cached()
        mem.short_memory_limit(mem.short_memory_used() + (16 + 8) * n * m)
    ctx.set_field_points(p)
    calls, refused = log(), mem.short_memory_refused()
    mem.short_memory_limit(0)
    ctx.solve_frequency(w, beta)
    pot = ctx.field_potentials(1)
    if want is None: want = pot
    ctx.close()
answer(refused=refused, after=calls[calls.rindex("x") + 1:], err=rel(pot, want))
""")
    assert got["refused"] == 2  # the allocation and its repetition
    after = got["after"]
    assert "S" in after and (after.find("G") < 0 or after.find("S") < after.find("G")), after
    assert got["err"] < 1e-12  # the same influences from k_field_pairs, their sums of 234 terms in another order


@pytest.mark.parametrize("without", ["second block", "copy of the right-hand sides"])
def test_gmres_without_its_second_block(so, without):
    """Memory for everything but the second set of body blocks, or but the copy of the right-hand sides
    beside it: the library's factors, as where no inverse is formed.  Tolerance 1e-11 on the preconditioned
    residual, systems of condition below 1e3: 1e-8."""
    got = short_memory.run(so, f"without = {without!r}" + """
geom = deck([meshgen.cylinder(5.0, 8.0, 24, 9, 4, 30.0 * k, 0.0) for k in range(3)])
n, nn, nrhs = 936, 312, 19
kw = dict(rho=1025.0, g=9.81, solver=hams_b200.SOLVER_GMRES, gmres_restart=40, gmres_maxit=400, gmres_tol=1e-11,
          gmres_dense=1)
w, beta = hams_b200.wave_properties(0.9, -1.0, 9.81), [0.3]
ctx = hams_b200.Context(geom, -1.0, **kw)
want = ctx.solve_frequency(w, beta)
ctx.close()
hams_b200.release_cached()
mem.short_memory_reset()
ctx = hams_b200.Context(geom, -1.0, **kw)
ctx.solve_frequency(w, beta)
peak = mem.short_memory_peak()
ctx.close()
hams_b200.release_cached()
ctx = hams_b200.Context(geom, -1.0, **kw)
block = (16 * 3 * nn * nn + (1 << 21) - 1 >> 21) << 21
tmp = (16 * n * nrhs + 255) // 256 * 256
mem.short_memory_reset()
mem.short_memory_limit(peak - (block if without == "second block" else tmp))
got = ctx.solve_frequency(w, beta)
again = ctx.solve_frequency(w, beta)
lib = hams_b200.load_library()
lib.hams_last_error.restype = ctypes.c_char_p
answer(refused=mem.short_memory_refused(), err=max(rel(a, b) for a, b in zip(got, want)), msg=lib.hams_last_error().decode(),
       same=all(np.array_equal(a, b) for a, b in zip(got, again)))
""")
    assert got["refused"] > 0 and got["err"] < 1e-8 and got["same"] and got["msg"] == ""


ROUGH = """
import test_series
geom = deck(test_series._rough([meshgen.cylinder(4.0, 6.0, 20, 5, 3)], 0.02, 1))
beta, size = [0.3, 1.1], 1 << 20  # size: far below the tables of its 25,600 distances
waves = [hams_b200.wave_properties(v, 45.0, 9.81) for v in (0.6, 1.3)]
def live():
    hams_b200.release_cached()
    return mem.short_memory_used()
"""


def test_context_without_its_radial_tables(so):
    """A table of the distinct distances that does not fit leaves its branch to the pairs' own rows: the
    same numbers, the same operations, the same bits."""
    got = short_memory.run(so, ROUGH + """
def assembled(limit):
    live()
    mem.short_memory_limit(limit)
    ctx = hams_b200.Context(geom, 45.0, rho=1025.0, g=9.81)
    mem.short_memory_limit(0)
    held = live()
    out = [x.copy() for w in waves for x in ctx.assemble(w, beta)]
    ctx.close()
    return out, held
want, held = assembled(0)
got, less = assembled(held - size)
answer(less=held - less, same=all(np.array_equal(a, b) for a, b in zip(got, want)))
""")
    assert got["less"] >= 1 << 20 and got["same"]


def test_batch_lane_without_its_radial_tables(so):
    """The lane of a batch's second frequency finds no room for the tables that its context has."""
    got = short_memory.run(so, ROUGH + """
def batch(limit):
    live()
    ctx = hams_b200.Context(geom, 45.0, rho=1025.0, g=9.81, batch_lanes=2)
    ctx.solve_frequency(waves[0], beta)
    live()
    mem.short_memory_limit(limit)
    out = ctx.solve_batch(waves, beta)
    mem.short_memory_limit(0)
    held = live()
    ctx.close()
    return out, held
want, held = batch(0)
got, less = batch(held - size)
answer(less=held - less, same=all(np.array_equal(a, b) for a, b in zip(got, want)))
""")
    assert got["less"] >= 1 << 20 and got["same"]


# bodies, depth, waves, field points, keywords, and the MB that the call needs without what only saves time,
# 5 % above the least found by bisection
DECKS = {
    "batch": ("test_series._rough([meshgen.cylinder(4.0, 6.0, 24, 8, 4)], 0.02, 1)", 45.0, 4, 0, "", 44),
    "mixed": ("test_series._rough([meshgen.cylinder(4.0, 6.0, 24, 8, 4)], 0.02, 1)", 45.0, 1, 0,
              "precision=hams_b200.PREC_MIXED", 23),
    "field points": ("[meshgen.cylinder(4.0, 6.0, 20, 9, 4)]", 45.0, 3, 4000, "", 140),
    "gmres": ("[meshgen.cylinder(4.0, 6.0, 20, 9, 4, 20.0 * k, 0.0) for k in range(3)]", 45.0, 1, 0,
              "solver=hams_b200.SOLVER_GMRES, gmres_tol=1e-11, gmres_dense=1", 71),
}


@pytest.mark.parametrize("name", list(DECKS))
def test_tables_make_room(so, name):
    """The buffers that a solve allocates as it goes find no room beside the tables: these are given back
    and the call is repeated, down to the memory that it needs without them.  Every limit from there up
    works, with the results of ample memory to the rounding of another order of sums."""
    bodies, depth, nf, field, kw, need = DECKS[name]
    got = short_memory.run(so, f"bodies, depth, nf, field, need, kw = \"{bodies}\", {depth}, {nf}, {field}, {need}, dict({kw})" + """
import test_series
geom = deck(eval(bodies))
rng = np.random.default_rng(1)
p = np.column_stack([rng.uniform(8.0, 30.0, field), rng.uniform(-20.0, 20.0, field), -rng.uniform(0.5, 12.0, field)])
waves = [hams_b200.wave_properties(v, depth, 9.81) for v in np.linspace(0.6, 1.4, nf)]
def solved(limit):
    hams_b200.release_cached()
    mem.short_memory_limit(limit)
    ctx = hams_b200.Context(geom, depth, rho=1025.0, g=9.81, **kw)
    if field: ctx.set_field_points(p)
    out = list(ctx.solve_batch(waves, [0.3]) if nf > 1 else ctx.solve_frequency(waves[0], [0.3]))
    if field: out += [ctx.field_potentials(1, k) for k in range(nf)]
    mem.short_memory_limit(0)
    ctx.close()
    return out
solved(0)
hams_b200.release_cached()
mem.short_memory_reset()
want = solved(0)
peak, errs, refused = mem.short_memory_peak(), [], []
need = int(need * 2 ** 20)
for limit in np.linspace(need, peak, 9).astype(int):
    mem.short_memory_reset()
    errs.append(max(rel(a, b) for a, b in zip(solved(int(limit)), want)))
    refused.append(mem.short_memory_refused())
answer(peak=peak, need=need, errs=errs, refused=refused)
""")
    assert got["need"] < got["peak"] and got["refused"][0] > 0, got
    assert max(got["errs"]) < 1e-9, got


def test_field_points_of_a_batch_take_one_way(so):
    """A lane that finds no room for the mode tables of the points' pair set, though for the influences
    themselves: every frequency has the bits of the pair set, or every one those of the pairs taken singly."""
    got = short_memory.run(so, """
geom = deck([meshgen.cylinder(4.0, 6.0, 6, 3, 1)])
rng, m = np.random.default_rng(1), 20000
p = np.column_stack([rng.uniform(8.0, 30.0, m), rng.uniform(-20.0, 20.0, m), -rng.uniform(0.5, 12.0, m)])
waves = [hams_b200.wave_properties(v, 45.0, 9.81) for v in np.linspace(0.6, 1.4, 6)]
def solved(room):
    ctx = hams_b200.Context(geom, 45.0, rho=1025.0, g=9.81, batch_lanes=2)
    ctx.set_field_points(p)
    ctx.solve_frequency(waves[0], [0.3])
    hams_b200.release_cached()
    mem.short_memory_reset()
    mem.short_memory_limit(mem.short_memory_used() + room if room else 0)
    ctx.solve_batch(waves, [0.3])
    mem.short_memory_limit(0)
    out = [ctx.field_potentials(1, k) for k in range(len(waves))]
    ctx.close()
    hams_b200.release_cached()
    return out
want, ways = solved(0), []
for mb in range(22, 62, 3):
    ways.append([bool(np.array_equal(a, b)) for a, b in zip(solved(mb << 20), want)])
answer(ways=ways)
""")
    assert all(all(w) or not any(w) for w in got["ways"]), got
    assert any(all(w) for w in got["ways"]) and any(not any(w) for w in got["ways"]), got


def test_points_without_their_tables(so):
    """hams_eval_green with room for the points and their results only: a thread per point, the same bits."""
    got = short_memory.run(so, """
ctx = hams_b200.Context(deck([meshgen.cylinder(4.0, 4.0, 8, 2, 2)]), 31.0, g=9.81)
rng, n = np.random.default_rng(1), 5000
r, th = 31.0 * np.exp(rng.uniform(np.log(1e-4), np.log(2.0), n)), rng.uniform(0.0, 6.28, n)
pts = np.zeros((n, 6), order="F")
pts[:, 3], pts[:, 4] = r * np.cos(th), r * np.sin(th)
pts[:, 2], pts[:, 5] = rng.uniform(-12.0, -0.3, n), rng.uniform(-12.0, -0.3, n)
flag, wave = (rng.uniform(size=n) < 0.5).astype(np.int32), ctx.wave(1.3)
want = ctx.eval_green(wave, pts, flag)
hams_b200.release_cached()
same, refused = [], []
for room in (n * (48 + 4 + 64) + 4096, 1 << 20, 4 << 20):
    mem.short_memory_reset()
    mem.short_memory_limit(mem.short_memory_used() + room)
    same.append(bool(np.array_equal(ctx.eval_green(wave, pts, flag), want)))
    refused.append(mem.short_memory_refused())
    hams_b200.release_cached()
answer(same=same, refused=refused)
""")
    assert all(got["same"]) and all(got["refused"]), got


@pytest.mark.parametrize("solver", ["SOLVER_LU", "SOLVER_GMRES"])
def test_a_refused_launch_of_the_lu_is_named(so, solver):
    """The runtime refuses one launch of the complex128 LU: the call's error is the runtime's, and the next
    call works."""
    got = short_memory.run(so, f"solver = hams_b200.{solver}" + """
geom = deck([meshgen.cylinder(5.0, 8.0, 10, 4, 4, 30.0 * k, 0.0) for k in range(2)])
ctx = hams_b200.Context(geom, -1.0, rho=1025.0, g=9.81, solver=solver, gmres_dense=1)
w, msgs = ctx.wave(0.9), []
want = ctx.solve_frequency(w, [0.3])
for k in (0, 1, 2, 3, 12):  # panel, its rows' exchange, update, and one of a later block of columns
    mem.short_memory_fail_launch(k)
    try:
        ctx.solve_frequency(w, [0.3])
        msgs.append("")
    except hams_b200.HamsError as e:
        msgs.append(str(e))
    mem.short_memory_fail_launch(-1)
    again = ctx.solve_frequency(w, [0.3])
    msgs[-1] += "" if all(np.array_equal(a, b) for a, b in zip(again, want)) else " (and then wrong)"
answer(msgs=msgs)
""")
    assert all("-2" in m and m.endswith("invalid configuration argument") for m in got["msgs"]), got
