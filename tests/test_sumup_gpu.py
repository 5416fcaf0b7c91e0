"""Hartree sum-up on the GPU against the oracle: values within FP64 tolerance
and every branch decision (near / far / skipped, l_atom_max) bit-identical."""
import numpy as np
import pytest
import torch

import oracle
from fast_rpa_eval_b200 import _lib, synth
from gpu_util import dev, host, normwise_rel

pytestmark = pytest.mark.gpu
TOL = 1e-12


def run(plan, p, generic=False, codes=False):
    dv = dev(p.delta_v_hartree)
    c = torch.zeros(p.n_valid_points * p.n_centers_hartree_potential * p.T, dtype=torch.uint8, device="cuda") if codes else None
    plan.execute(p.j_atom_end - p.j_atom_begin + 1, dev(p.l_hartree_max_far_distance, np.int32),
                 dev(p.multipole_radius_sq), dev(p.outer_potential_radius), dev(p.multipole_moments), dev(p.spline),
                 dv, branch_codes=c, force_generic=generic)
    torch.cuda.synchronize()
    out = host(dv, (p.n_full_points, p.T))
    if codes:
        return out, host(c, (p.n_valid_points, p.n_centers_hartree_potential, p.T))
    return out


def delta_rel(out, ref, d0):
    return normwise_rel(out - d0, ref - d0)


@pytest.mark.parametrize("L,T,lh", [(4, 1, None), (6, 1, None), (6, 2, [6, 4, 2, 0]), (8, 1, [8, 7, 5, 3]), (8, 2, None)])
def test_sumup_fast_matches_oracle(L, T, lh):
    p = synth.make_sumup_problem(n_atoms=24, n_points=6000, l_pot_max=L, T=T, seed=50 + L + T,
                                 l_hartree_per_species=lh, extra_full_points=64)
    plan = _lib.SumupPlan(p)
    assert plan.fast
    out, codes = run(plan, p, codes=True)
    ref, rcodes = oracle.sumup(p, branch_codes=True)
    assert np.array_equal(codes, rcodes)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL
    # untouched full points keep their input value exactly
    untouched = np.setdiff1d(np.arange(p.n_full_points), p.i_valid_point_2_i_full_points_map)
    assert np.array_equal(out[untouched], p.delta_v_hartree[untouched])


@pytest.mark.parametrize("centers", ["identity", "permuted"])
def test_sumup_generic_matches_oracle(centers):
    p = synth.make_sumup_problem(n_atoms=20, n_points=3000, l_pot_max=6, T=2, seed=61, centers=centers,
                                 l_hartree_per_species=[6, 5, 3, 6])
    plan = _lib.SumupPlan(p)
    assert plan.fast == (centers == "identity")
    out, codes = run(plan, p, generic=True, codes=True)
    ref, rcodes = oracle.sumup(p, branch_codes=True)
    assert np.array_equal(codes, rcodes)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL


@pytest.mark.skipif(not oracle.ref_available(1), reason="reference library not built")
def test_sumup_matches_reference_cpu_code():
    p = synth.make_sumup_problem(n_atoms=30, n_points=8000, l_pot_max=6, T=1, seed=71, l_hartree_per_species=[6, 6, 4, 2])
    out = run(_lib.SumupPlan(p), p)
    ref = oracle.sumup(p, use_reference=True)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL


def test_sumup_config3_shape_far_field_only():
    # the benchmark recipe at reduced size: no l truncation, near field rare
    p = synth.config3(l_max=8, n_atoms=60, n_points=20000, seed=5)
    out = run(_lib.SumupPlan(p), p)
    ref = oracle.sumup(p, n_threads=8)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL


def test_sumup_dropin_symbol_matches_oracle():
    p = synth.make_sumup_problem(n_atoms=16, n_points=2000, l_pot_max=6, T=2, seed=81)
    out = _lib.dropin_sumup(p)
    ref = oracle.sumup(p)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL


def test_sumup_session_cu_host_matches_oracle():
    r = synth.make_rho1_problem(T=1, seed=3, n_batches=8)
    p = synth.make_sumup_problem(n_atoms=16, n_points=1500, l_pot_max=6, T=1, seed=82)
    # share the full-point count (the session holds both paths)
    p.n_full_points = r.n_full_points = max(r.n_full_points, p.n_full_points)
    pad = p.n_full_points - p.coord_points.shape[1]
    p.coord_points = np.asfortranarray(np.concatenate([p.coord_points, np.zeros((3, pad))], axis=1))
    p.delta_v_hartree = np.asfortranarray(np.concatenate([p.delta_v_hartree, np.zeros((pad, 1))], axis=0))
    p.partition_tab = np.concatenate([p.partition_tab, np.ones(pad)])
    r.partition_tab = p.partition_tab
    r.i_valid_point_2_i_full_points_map = np.concatenate(
        [r.i_valid_point_2_i_full_points_map, np.arange(len(r.i_valid_point_2_i_full_points_map), p.n_full_points)]).astype(np.int32)
    with _lib.Session(r, p) as s:
        out = s.sumup()
        ref = oracle.sumup(p)
        assert delta_rel(out, ref, p.delta_v_hartree) < TOL
        out2 = s.sumup(delta_v=out)
        ref2 = oracle.sumup(p, delta_v=ref)
        assert delta_rel(out2, ref2, p.delta_v_hartree) < TOL


@pytest.mark.parametrize("atoms,points,T,L,outer", [
    (1, 1, 1, 0, None),         # one record, one point
    (7, 33, 1, 3, 6.0),         # one record less than a chunk, a warp and one lane
    (8, 129, 1, 4, 6.0),        # a whole chunk
    (9, 1000, 2, 8, 5.0),       # a chunk and one record; one point per thread, records over 4 warps
    (33, 300, 1, 2, None),      # a chunk of the low degrees and one record
    (25, 900, 2, 6, 6.0),       # two chunks of this degree and one record
    (20, 20_000, 4, 6, 6.0),    # two points per thread
    (16, 40_001, 4, 5, 6.0),    # four points per thread, records over 4 warps
    (3, 152_001, 4, 2, None),   # four points per thread, all records in one warp
])
def test_sumup_dispatch_edges_match_oracle(atoms, points, T, L, outer):
    """Sizes at the edges of the far- and near-field launches' rules."""
    p = synth.make_sumup_problem(n_atoms=atoms, n_points=points, l_pot_max=L, T=T, seed=90 + atoms, outer_radius=outer,
                                 l_hartree_per_species=[L, max(0, L - 1), L, max(0, L - 2)], extra_full_points=5)
    out = run(_lib.SumupPlan(p), p)
    ref = oracle.sumup(p, n_threads=8)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL
    untouched = np.setdiff1d(np.arange(p.n_full_points), p.i_valid_point_2_i_full_points_map)
    assert np.array_equal(out[untouched], p.delta_v_hartree[untouched])


@pytest.mark.parametrize("points", [700, 40_000])
def test_sumup_extreme_records_match_generic_kernel(points):
    """Moments too large (or infinite) at an l that only near-by points reach, a
    vanishing near radius and a point without finite coordinates: the same
    points stay finite as in the table loop, with the same values."""
    p = synth.make_sumup_problem(n_atoms=12, n_points=points, l_pot_max=6, T=4, seed=33, outer_radius=4.0)
    p.multipole_moments[40, 0, :] = np.inf       # l = 6
    p.multipole_moments[30, 1, 1:] = 1e200       # l = 5
    p.multipole_radius_sq[2, :] = 1e-50          # every point far
    bad = int(p.i_valid_point_2_i_full_points_map[3])
    p.coord_points[1, bad] = np.nan
    p.coord_points[0, int(p.i_valid_point_2_i_full_points_map[5])] = np.inf
    plan = _lib.SumupPlan(p)
    fast, generic = run(plan, p), run(plan, p, generic=True)
    assert np.array_equal(fast[bad], p.delta_v_hartree[bad])
    ok = np.isfinite(generic)
    assert np.array_equal(ok, np.isfinite(fast)) and ok.mean() > 0.5
    small = ok & (np.abs(generic) < 1e6)
    assert np.max(np.abs(fast - generic)[small]) < TOL * np.max(np.abs(generic[small]))
    big = ok & ~small
    assert np.all(np.abs(fast - generic)[big] < TOL * np.abs(generic[big]) * 1e2)


@pytest.mark.parametrize("captured", [False, True])
def test_sumup_calls_in_a_row_equal_calls_one_by_one(captured):
    """The three launches of a call overlap their start-up; calls queued without
    a wait, with other moments each time, give the bits of separate calls."""
    p = synth.make_sumup_problem(n_atoms=20, n_points=3000, l_pot_max=4, T=2, seed=97, extra_full_points=5)
    plan = _lib.SumupPlan(p)
    a = [dev(p.l_hartree_max_far_distance, np.int32), dev(p.multipole_radius_sq), dev(p.outer_potential_radius)]
    moments = [dev(p.multipole_moments), dev(-0.7 * p.multipole_moments)]
    spline, na = dev(p.spline), p.j_atom_end - p.j_atom_begin + 1
    dv = [dev(p.delta_v_hartree) for _ in range(2)]
    for i in range(40):
        plan.execute(na, *a, moments[i & 1], spline, dv[0])
        torch.cuda.synchronize()

    def queue():
        for i in range(40):
            plan.execute(na, *a, moments[i & 1], spline, dv[1])

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            queue()
        graph.replay()
    else:
        queue()
    torch.cuda.synchronize()
    assert torch.equal(dv[0], dv[1])


def test_sumup_inverse_distance_of_a_point_charge():
    """One centre with a monopole: delta_v is c / r.  Distances over the whole
    far field, dense around powers of four in r^2, and the centre itself
    (infinite, as in the table loop).  The points lie on the x axis, so r^2 has
    one rounding (that of x x, repeated here) and the rest is one inverse square
    root (CUDA: 1 ulp) and one multiplication (half an ulp): 2 ulp."""
    p = synth.make_sumup_problem(n_atoms=1, n_points=5000, l_pot_max=0, seed=5, outer_radius=None)
    rng = np.random.default_rng(5)
    powers = 2.0 ** np.arange(-60, 14)
    near_powers = np.concatenate([np.nextafter(powers, 0), powers, np.nextafter(powers, np.inf)])
    x = np.concatenate([[0.0], near_powers, 10.0 ** rng.uniform(-19.5, 3.99, 5000 - 1 - near_powers.size)])
    p.coords_center[:] = 0.0
    p.coord_points[:] = 0.0
    p.coord_points[0, p.i_valid_point_2_i_full_points_map] = x * rng.choice([-1.0, 1.0], x.size)
    p.multipole_radius_sq[:] = 0.0
    p.multipole_moments[:] = 1.0
    p.delta_v_hartree[:] = 0.0
    plan = _lib.SumupPlan(p)
    v = run(plan, p)[p.i_valid_point_2_i_full_points_map, 0]
    assert v[0] == np.inf == run(plan, p, generic=True)[p.i_valid_point_2_i_full_points_map[0], 0]
    want = p.cc[0] / np.sqrt((x[1:] * x[1:]).astype(np.longdouble))
    assert float(np.max(np.abs(v[1:] - want) / want)) < 2 * 2.0**-52


@pytest.mark.parametrize("atoms,points,T,L,outer", [
    (1, 64, 1, 2, 3.0),        # one centre at a low l: inline, few points
    (2, 4095, 1, 4, 3.0),      # the near field in its own launch
    (2, 4096, 1, 4, 3.0),      # inline: one point per thread
    (8, 65_536, 1, 6, 3.0),    # the most centres above l 5, as few points each as that takes
    (8, 65_535, 1, 6, 3.0),    # one point less
    (4, 40_000, 1, 7, 3.0),    # not at this l
    (2, 131_072, 2, 6, 3.0),   # as many points and perturbations as that takes
    (2, 20_000, 2, 6, 3.0),    # as few
    (1, 2100, 2, 8, 3.0),      # the highest l; one centre at most
    (2, 5000, 1, 6, None),     # own launch at this l
    (16, 33_000, 1, 5, 4.0),   # the most centres of l 5, records over 4 warps
    (17, 36_000, 1, 5, 4.0),   # one more
    (128, 262_144, 1, 0, None),  # two points per thread, several chunks of records
    (3, 152_001, 2, 1, 2.5),   # two points per thread, all records in one warp
])
def test_sumup_dense_points_match_oracle(atoms, points, T, L, outer):
    """Both sides of the rule that puts the near field into the far field's
    launch, with radii cut inside and outside the near sphere."""
    p = synth.make_sumup_problem(n_atoms=atoms, n_points=points, l_pot_max=L, T=T, seed=120 + atoms, outer_radius=outer,
                                 l_hartree_per_species=[L, max(0, L - 1), L, max(0, L - 2)], extra_full_points=5)
    out = run(_lib.SumupPlan(p), p)
    ref = oracle.sumup(p, n_threads=8)
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL
    untouched = np.setdiff1d(np.arange(p.n_full_points), p.i_valid_point_2_i_full_points_map)
    assert np.array_equal(out[untouched], p.delta_v_hartree[untouched])


@pytest.mark.parametrize("atoms,points,T,L", [
    (9, 1000, 2, 8),       # one point per thread, records over 4 warps; centres shared by 8 near-field warps
    (20, 20_000, 4, 6),    # two points per thread
    (16, 40_001, 4, 5),    # four points per thread, records over 4 warps
    (40, 160_000, 1, 5),   # four points per thread
    (3, 7000, 1, 3),       # near field inline, one point per thread
    (3, 152_001, 2, 2),    # near field inline, two points per thread
])
def test_sumup_branch_codes_are_those_of_the_plain_call(atoms, points, T, L):
    """The codes are written by the launches of a call without codes (same bits of
    delta_v) and equal the table loop's decisions, with points exactly at a near
    radius, at an outer radius of every l and at the end of the far field, and the
    next representable distances on both sides."""
    p = synth.make_sumup_problem(n_atoms=atoms, n_points=points, l_pot_max=L, T=T, seed=140 + atoms, outer_radius=4.0,
                                 l_hartree_per_species=[L, max(0, L - 1), L, max(0, L - 2)], extra_full_points=5)
    rng = np.random.default_rng(atoms)
    slot = 0
    free = p.i_valid_point_2_i_full_points_map[rng.permutation(points)]

    def at_distance(a, d):
        """Three points on the x axis through centre a; the middle one's squared distance."""
        nonlocal slot
        c = p.coords_center[:, a]
        x = c[0] + d
        for v in (np.nextafter(x, -np.inf), x, np.nextafter(x, np.inf)):
            p.coord_points[:, free[slot]] = (v, c[1], c[2])
            slot += 1
        return (x - c[0]) * (x - c[0])

    for a in range(min(atoms, 6)):
        for t in range(T):
            p.multipole_radius_sq[a, t] = at_distance(a, rng.uniform(1.5, 2.5))
            for l in range(1, L + 1):  # falling with l, around and outside the near sphere
                p.outer_potential_radius[l, a, t] = at_distance(a, 1.0 + 6.0 * (L + 1 - l) / L * rng.uniform(0.9, 1.0))
        at_distance(a, 1e4)
        at_distance(a, -1e4)
    assert slot < points
    plan = _lib.SumupPlan(p)
    out, codes = run(plan, p, codes=True)
    ref, rcodes = oracle.sumup(p, branch_codes=True)
    assert np.array_equal(codes, rcodes)
    assert np.any(rcodes == 0) and np.any((rcodes > 0) & (rcodes < 16)) and np.any(rcodes >= 16)
    assert np.array_equal(out, run(plan, p))
    assert delta_rel(out, ref, p.delta_v_hartree) < TOL


def test_sumup_dropin_calls_of_alternating_sizes():
    """The host-array entry keeps its plan's memory between calls: smaller and
    larger problems, l and tiles in turn give the bits of a plan of their own, and
    the memory in use does not grow."""
    cases = [synth.make_sumup_problem(n_atoms=a, n_points=n, l_pot_max=L, T=T, seed=200 + a, extra_full_points=3,
                                      centers=c)
             for a, n, L, T, c in ((5, 300, 4, 1, "identity"), (30, 20_000, 6, 2, "identity"), (9, 2000, 8, 1, "identity"),
                                   (12, 900, 3, 1, "permuted"))]
    free = None
    for turn in range(3):
        for p in cases:
            out = _lib.dropin_sumup(p)
            assert np.array_equal(out, run(_lib.SumupPlan(p), p))
            if turn == 0:
                assert delta_rel(out, oracle.sumup(p), p.delta_v_hartree) < TOL
        torch.cuda.empty_cache()
        now = torch.cuda.mem_get_info()[0]
        assert free is None or now == free
        free = now if turn else None
