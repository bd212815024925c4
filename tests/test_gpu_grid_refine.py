"""The grid-wide refinement at the edges of its 256-row diagonal blocks, and
the factor's 128-column steps at the edges of theirs (S of 3,072 and above):
meshes whose S is just above a multiple of the width or below one, against
the plain FP64 form (Zin 1e-6, currents 1e-7 normwise: the mixed form's gates)."""
import numpy as np
import pytest

import bench

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import nec_accel

    return nec_accel


# a grid of nx x ny cells has 3 (nx (ny + 1) + ny (nx + 1)) unknowns
@pytest.mark.parametrize("edges,pivoting", [(512, 0), (513, 0), (597, 0), (598, 1), (683, 0), (720, 1), (1023, 0),
                                            (1024, 0), (1025, 0), (1066, 0), (1067, 0), (1109, 0), (1109, 1)])
def test_mixed_mesh_matches_plain(acc, edges, pivoting):
    w, s, f = bench.mesh_workload(24)
    ant = acc.Antenna(acc.wires_array(w[:edges]), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    plain = acc.HallenBatch([ant]).solve()
    b = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED)
    assert b.units[0]["s"] == 3 * edges
    b.schedule = {"factor_pivoting": pivoting}
    mixed = b.solve()
    assert plain.status[0] == 0 and mixed.status[0] == 0
    x0, x1 = plain.currents[0], mixed.currents[0]
    assert np.linalg.norm(x1 - x0) <= 1e-7 * np.linalg.norm(x0)
    z0, z1 = (complex(r.feeds[0][0][5], r.feeds[0][0][6]) for r in (plain, mixed))
    assert abs(z1 - z0) <= 1e-6 * abs(z0)


def test_wide_steps_of_several_units_beside_small_ones(acc):
    """Two systems that take 128-column steps (one a multiple of 128 tall),
    a mid-size and a small one in one batch: each equals its own solve."""
    w, s, f = bench.mesh_workload(24)
    ants = [acc.Antenna(acc.wires_array(w[:e]), acc.sources_array([(7, 1, 1.0)]), [f], 1) for e in (1024, 300, 1040, 40)]
    both = acc.HallenBatch(ants, precision=acc.PRECISION_MIXED).solve()
    for u, ant in enumerate(ants):
        alone = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED).solve()
        assert both.status[u] == 0 and alone.status[0] == 0
        x0, x1 = alone.currents[0], both.currents[u]
        assert np.linalg.norm(x1 - x0) <= 1e-7 * np.linalg.norm(x0)


def test_server_takes_a_large_request_whose_own_scratch_misses_the_budget(acc):
    """A budget 4 MB below a request's estimate leaves no room for the block
    inverses' scratch (8 KB per row of S = 1,632, 13 MB): the request is still
    taken, planned without it, and its result is the batch's."""
    w, s, f = bench.mesh_workload(16)
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    ref = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED).solve()
    with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=1 << 30) as srv:
        need = srv.shape(ant).device_bytes
    with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=need - (4 << 20)) as srv:
        r = srv.submit(ant, copy_out=True)
        srv.wait(r)
        currents, _, _, status = r.result()
        assert status[0] == 0
        x0, x1 = np.ravel(ref.currents[0]), np.ravel(currents)
        assert np.linalg.norm(x1 - x0) <= 1e-7 * np.linalg.norm(x0)


@pytest.mark.parametrize("ctas", [12, 31, 32])
def test_refinement_on_few_sms(acc, ctas):
    """A partition of fewer than 32 SMs has fewer warps than a diagonal block
    has rows (8 a CTA, 256): the refinement still converges to the plain form
    (its gates), as it does with 32."""
    w, s, f = bench.mesh_workload(16)
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    x0 = acc.HallenBatch([ant]).solve().currents[0]
    acc.test_limit_refinement_ctas(ctas)
    try:
        b = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED)
    finally:
        acc.test_limit_refinement_ctas(0)
    assert b.units[0]["s"] >= 1536
    r = b.solve()
    assert r.status[0] == 0
    assert np.linalg.norm(r.currents[0] - x0) <= 1e-7 * np.linalg.norm(x0)
    assert b.refinement_stats()[0][0] < 24


def test_no_room_for_the_inverses_keeps_the_grid_refinement(acc):
    """A batch whose allocation of the block inverses fails (the last one of
    its planning; injected) still refines grid-wide, in 32-row blocks: it
    runs the launches of a full one but for the four that form the inverses."""
    w, s, f = bench.mesh_workload(16)
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    full = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED)
    ref = full.solve()
    seen = set()
    for after in range(60):
        acc.test_fail_device_allocation(after)
        try:
            b = acc.HallenBatch([ant], precision=acc.PRECISION_MIXED)
        except acc.AccelError as e:
            assert e.code == acc.ERR_OUT_OF_MEMORY
            continue
        finally:
            acc.test_fail_device_allocation(-1)
        if b.info.device_bytes == full.info.device_bytes:
            break  # nothing failed: past the last allocation
        r = b.solve()
        assert r.status[0] == 0
        assert np.linalg.norm(r.currents[0] - ref.currents[0]) <= 1e-7 * np.linalg.norm(ref.currents[0])
        seen.add(full.kernel_launches - b.kernel_launches)
        b.close()
    assert 4 in seen


def _serve(acc, ants, **kw):
    with acc.Server(acc.PRECISION_MIXED, lanes=1, **kw) as srv:
        reqs = [srv.submit(a, copy_out=True) for a in ants]
        for r in reqs:
            srv.wait(r)
        return [r.result() for r in reqs], srv.stats()


def test_request_without_the_optional_scratch_still_refines_grid_wide(acc):
    """The budget of the test above, seen in the launches: the request runs
    all of a full one's but the four that form the block inverses."""
    w, s, f = bench.mesh_workload(16)
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=1 << 30) as srv:
        need = srv.shape(ant).device_bytes
    (full,), s0 = _serve(acc, [ant], hbm_budget_bytes=1 << 30)
    (lean,), s1 = _serve(acc, [ant], hbm_budget_bytes=need - (4 << 20))
    assert full[3][0] == 0 and lean[3][0] == 0
    assert s0["kernel_launches"] - s1["kernel_launches"] == 4
    assert np.linalg.norm(lean[0][0] - full[0][0]) <= 1e-7 * np.linalg.norm(full[0][0])


def test_request_without_the_optional_scratch_leaves_the_others_theirs(acc):
    """S = 9,840, 120, 1,632 and 120, all queued before the only lane may take
    one (results held in place fill its five slabs), on a budget with no room
    for the first one's optional scratch but for its other needs beside all
    of the others.  Two batches: one without the scratch, with the first
    small request in it, and one with it."""
    def ant(w, f):
        return acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)

    w, s, f = bench.mesh_workload(40)
    big, mid, small = ant(w, f), ant(w[:544], f), ant(w[:40], f)
    with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=8 << 30) as srv:
        budget = srv.shape(big).device_bytes - (10 << 20)

    def burst(ants):
        with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=budget) as srv:
            held = [srv.wait(srv.submit(small)) for _ in range(5)]
            srv.stats(reset=True)
            reqs = [srv.submit(a, copy_out=True) for a in ants]
            for r in held:
                r.release()
            for r in reqs:
                srv.wait(r)
            return reqs, srv.stats()

    reqs, st = burst([big, small, mid, small])
    first, s1 = burst([big, small])
    second, s2 = burst([mid, small])
    assert (st["batches"], s1["batches"], s2["batches"]) == (2, 1, 1)
    assert st["kernel_launches"] == s1["kernel_launches"] + s2["kernel_launches"]
    for a, b in zip(reqs, first + second):
        assert a.status[0] == 0 and b.status[0] == 0
        assert np.linalg.norm(a.currents - b.currents) <= 1e-7 * np.linalg.norm(b.currents)


@pytest.mark.parametrize("lanes,short", [(1, 0), (1, 4 << 20), (2, 0)])
def test_submitted_requests_device_bytes_is_what_admission_charges(acc, lanes, short):
    w, s, f = bench.mesh_workload(16)
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(7, 1, 1.0)]), [f], 1)
    with acc.Server(acc.PRECISION_MIXED, lanes=1, hbm_budget_bytes=1 << 30) as srv:
        full = srv.shape(ant).device_bytes
    with acc.Server(acc.PRECISION_MIXED, lanes=lanes, hbm_budget_bytes=full - short) as srv:
        r = srv.wait(srv.submit(ant, copy_out=True))
        assert r.status[0] == 0
        assert r.info.device_bytes == srv.stats()["peak_in_flight_bytes"]
        assert (r.info.device_bytes == full) == (lanes == 1 and short == 0)


@pytest.mark.parametrize("edges", [342, 350, 352])
def test_split_panel_is_the_one_cta_panel(acc, edges):
    """S of 1,026 to 1,056: the first panel is one CTA's when the system is
    alone, and split over many beside a taller one of its size class; the
    same factor, so the same currents, bit for bit."""
    w, s, f = bench.mesh_workload(24)
    ants = [acc.Antenna(acc.wires_array(w[:e]), acc.sources_array([(7, 1, 1.0)]), [f], 1) for e in (edges, 467)]
    alone = acc.HallenBatch(ants[:1], precision=acc.PRECISION_MIXED).solve()
    beside = acc.HallenBatch(ants, precision=acc.PRECISION_MIXED).solve()
    assert alone.status[0] == 0 and beside.status[0] == 0
    assert np.array_equal(alone.currents[0].view(np.uint64), beside.currents[0].view(np.uint64))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("wires,segments,freqs", [(6, 101, 100), (1, 17, 300), (2, 801, 8)])
def test_footprint_of_many_frequencies_bounds_the_batch(acc, precision, wires, segments, freqs):
    """The fill's and the Gram's tile lists hold an entry per tile of every
    frequency's system: the admission estimate counts them all."""
    w = [(t + 1, segments, (2.0 * t, 0.0, -5.0), (2.0 * t, 0.0, 5.0), 1e-3) for t in range(wires)]
    f = [14.0e6 + 1e3 * k for k in range(freqs)]
    ant = acc.Antenna(acc.wires_array(w), acc.sources_array([(1, segments // 2, 1.0)]), f, 0)
    with acc.Server(precision, lanes=1, hbm_budget_bytes=1 << 30) as srv:
        est = srv.shape(ant).device_bytes
    b = acc.HallenBatch([ant], precision=precision)
    assert b.info.device_bytes <= est, (b.info.device_bytes, est)
    b.close()
