"""First-order H on the GPU (evaluate_first_order_h_reduce_memory_c_v2_ and
frpa_rho1_first_order_h) against the reference's own CPU code compiled in
oracle/_ref, with every exchange-correlation term non-zero, and the
determinism of the fixed-point accumulation it shares with the rho1 adjoint:
two runs give the same bits."""
import numpy as np
import pytest
import torch

import oracle
from fast_rpa_eval_b200 import _lib, synth
from gpu_util import dev, host, normwise_rel

pytestmark = pytest.mark.gpu
TOL = 1e-12  # normwise relative, FP64 against the reference's FP64


def _case(T, seed, n_atoms=6, n_batches=16, j_begin=1, n_active=None):
    p = synth.make_rho1_problem(T=T, seed=seed, n_atoms=n_atoms, n_batches=n_batches, pad_value=np.nan,
                                n_active=T if n_active is None else n_active)
    p.j_atom_begin = j_begin
    p.j_atom_end = j_begin + (T if n_active is None else n_active) - 1
    xc = synth.first_order_h_inputs(p, seed=seed + 1, pad_value=np.nan)
    v = np.asfortranarray(np.random.default_rng(seed + 2).normal(size=(p.n_full_points, T)))
    return p, xc, v


def _reference(p, v, xc, j_coord, H0):
    return H0 + oracle.first_order_h(p, v, use_reference=oracle.ref_available(p.T), xc=xc, j_coord=j_coord)


@pytest.mark.parametrize("T,j_coord,j_begin", [(1, 1, 1), (2, 2, 1), (2, 3, 3), (4, 1, 2)])
def test_first_order_h_dropin_matches_reference(T, j_coord, j_begin):
    p, xc, v = _case(T, 100 + 7 * T + j_coord, j_begin=j_begin, n_active=min(T, p_atoms(6, j_begin)))
    H0 = np.asfortranarray(np.random.default_rng(9).normal(size=(p.n_basis, p.n_basis, T)))
    got = _lib.dropin_first_order_h(p, v, xc, H=H0, j_coord=j_coord)
    ref = _reference(p, v, xc, j_coord, H0)
    assert np.all(np.isfinite(got))
    assert normwise_rel(got - H0, ref - H0) < TOL


def p_atoms(n_atoms, j_begin):
    return n_atoms - j_begin + 1


def test_first_order_h_partial_tile_leaves_other_perturbations():
    # tile of 3 with 2 atoms active: the third slice of H is left as it was
    p, xc, v = _case(3, 131, n_active=2)
    H0 = np.asfortranarray(np.random.default_rng(4).normal(size=(p.n_basis, p.n_basis, 3)))
    got = _lib.dropin_first_order_h(p, v, xc, H=H0, j_coord=2)
    ref = _reference(p, v, xc, 2, H0)
    assert normwise_rel(got[:, :, :2] - H0[:, :, :2], ref[:, :, :2] - H0[:, :, :2]) < TOL
    assert np.array_equal(got[:, :, 2], H0[:, :, 2])


def _device_inputs(p, xc, v):
    d = {k: dev(a) for k, a in xc.items()}
    return d, dev(v), dev(p.partition_tab), dev(p.atom_valid_n_compute_c_batches, np.int32)


def test_first_order_h_plan_is_bit_identical_across_runs():
    p, xc, v = _case(2, 141, n_atoms=12, n_batches=60)
    plan = _lib.Rho1Plan(p)
    d, vd, pt, av = _device_inputs(p, xc, v)
    w, gw, hw = dev(p.wave), dev(p.gradient_wave), d["hessian_wave"]
    outs = []
    for _ in range(3):
        H = torch.zeros(p.n_basis * p.n_basis * 2, dtype=torch.float64, device="cuda")
        plan.first_order_h(2, p.n_atoms, 1, 1, av, w, gw, hw, d, vd, pt, H)
        torch.cuda.synchronize()
        outs.append(H.clone())
    assert plan.device_flags() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    ref = oracle.first_order_h(p, v, use_reference=oracle.ref_available(2), xc=xc, j_coord=1)
    assert normwise_rel(host(outs[0], ref.shape), ref) < TOL


def test_adjoint_dP1_is_bit_identical_across_runs():
    p = synth.make_rho1_problem(T=2, seed=151, n_atoms=12, n_batches=60, with_bias=True)
    plan = _lib.Rho1Plan(p)
    rng = np.random.default_rng(3)
    g_rho = dev(rng.normal(size=(p.n_full_points, 2)))
    g_grad = dev(rng.normal(size=(3, p.n_max_batch_size, p.n_my_batches_work, 2)))
    w, gw = dev(p.wave), dev(p.gradient_wave)
    outs = []
    for _ in range(3):
        dP1 = torch.zeros(p.n_basis * p.n_basis * 2, dtype=torch.float64, device="cuda")
        plan.adjoint_p1(2, w, gw, g_rho, g_grad, dP1)
        torch.cuda.synchronize()
        outs.append(dP1.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert float(outs[0].abs().max()) > 0


def test_first_order_h_flags_a_range_outside_its_batch():
    p, xc, v = _case(1, 161)
    av = p.atom_valid_n_compute_c_batches.copy()
    b = int(np.argmax(p.n_compute_c_batches))
    av[1, b] = p.n_compute_c_batches[b] + 5  # atom 1's range runs past the batch's compute functions
    plan = _lib.Rho1Plan(p)
    d, vd, pt, _ = _device_inputs(p, xc, v)
    H = torch.zeros(p.n_basis * p.n_basis, dtype=torch.float64, device="cuda")
    plan.device_flags()
    plan.first_order_h(1, p.n_atoms, 1, 1, dev(av, np.int32), dev(p.wave), dev(p.gradient_wave),
                       d["hessian_wave"], d, vd, pt, H)
    torch.cuda.synchronize()
    assert plan.device_flags() & 8
    assert torch.isfinite(H).all()


@pytest.mark.parametrize("nc,np_range,shift,T", [
    (1, (1, 3), 0, 1),        # one function, fewer points than a chunk
    (63, (15, 17), 0, 2),     # one tile, either side of a 16-point chunk
    (66, (31, 64), 1, 1),     # two tiles of 40 and 26 rows; odd wave offsets (8-byte copies)
    (130, (257, 260), 0, 1),  # three tiles of 48, 48 and 34; points past one coefficient stage
])
def test_tile_edges_match_oracle(nc, np_range, shift, T):
    """Adjoint (g_rho only, both, g_grad only) and first-order H at the edges of
    tiles, chunks and copy widths.  Sums of at most 260 x 12 terms a batch."""
    p = synth.make_rho1_problem(T=T, seed=200 + nc, n_atoms=8, n_batches=12, np_range=np_range, nc_range=(nc, nc),
                                pad_value=np.nan, with_bias=True)
    xc = synth.first_order_h_inputs(p, seed=5, pad_value=np.nan)
    if shift:
        p.wave = np.concatenate([np.full(shift, np.nan), p.wave])
        p.gradient_wave = np.concatenate([np.full(3 * shift, np.nan), p.gradient_wave])
        xc["hessian_wave"] = np.concatenate([np.full(6 * shift, np.nan), xc["hessian_wave"]])
        p.i_batch_2_wave_offset = (p.i_batch_2_wave_offset + shift).astype(np.int32)
    rng = np.random.default_rng(nc)
    v = np.asfortranarray(rng.normal(size=(p.n_full_points, T)))
    plan = _lib.Rho1Plan(p)
    d, vd, pt, av = _device_inputs(p, xc, v)
    w, gw, n = dev(p.wave), dev(p.gradient_wave), p.n_basis * p.n_basis * T
    H = torch.zeros(n, dtype=torch.float64, device="cuda")
    plan.first_order_h(T, p.n_atoms, 1, 2, av, w, gw, d["hessian_wave"], d, vd, pt, H)
    ref = oracle.first_order_h(p, v, use_reference=oracle.ref_available(T), xc=xc, j_coord=2)
    assert normwise_rel(host(H, ref.shape), ref) < TOL
    # the adjoint, per batch in numpy
    gr = rng.normal(size=(p.n_full_points, T))
    gg = rng.normal(size=(3, p.n_max_batch_size, p.n_my_batches_work, T))
    for use_r, use_g in ((True, False), (True, True), (False, True)):
        want = np.zeros((p.n_basis, p.n_basis, T))
        for b in range(p.n_my_batches_work):
            o, npb, ncp = int(p.i_batch_2_wave_offset[b]), int(p.n_point_batches[b]), (nc + 3) // 4 * 4
            phi = p.wave[o:o + ncp * npb].reshape(npb, ncp)[:, :nc]
            gphi = p.gradient_wave[3 * o:3 * (o + ncp * npb)].reshape(npb, 3, ncp)[:, :, :nc]
            pre = p.n_point_batches_prefix_sum[b]
            ib = p.i_basis_batches[:nc, b] - 1
            for t in range(T):
                a = np.zeros((npb, nc))
                if use_r:
                    a += gr[p.i_valid_point_2_i_full_points_map[pre:pre + npb], t][:, None] * phi
                if use_g:
                    a += 2.0 * np.einsum("kp,pki->pi", gg[:, :npb, b, t], gphi)
                want[np.ix_(ib, ib, [t])] += (a.T @ phi)[:, :, None]
        dP1 = torch.zeros(n, dtype=torch.float64, device="cuda")
        plan.adjoint_p1(T, w, gw, dev(gr) if use_r else None, dev(gg) if use_g else None, dP1)
        assert normwise_rel(host(dP1, want.shape), want) < TOL
    assert plan.device_flags() == 0


def test_adjoint_over_several_scratch_groups_equals_the_sum_of_its_parts():
    """A problem whose A(i, p) exceeds the scratch (several groups of batches)
    against its two halves, each within it."""
    from fast_rpa_eval_b200 import parallel

    p = synth.config2(seed=3, n_batches=1250)
    assert 8 * p.wave_len > (512 << 20)
    n = p.n_basis * p.n_basis
    rng = np.random.default_rng(1)
    g_rho = dev(rng.normal(size=p.n_full_points))

    def run(q):
        w = torch.empty(q.wave_len, dtype=torch.float64, device="cuda")
        gw = torch.empty(3 * q.wave_len, dtype=torch.float64, device="cuda")
        _lib.synth_basis_values(q, dev(np.asfortranarray(q.valid_points_xyz.T)), w, gw)
        plan, out = _lib.Rho1Plan(q), torch.zeros(n, dtype=torch.float64, device="cuda")
        for _ in range(2):  # the second call starts from the accumulator the first one left
            plan.adjoint_p1(1, w, gw, g_rho, None, out)
        assert plan.device_flags() == 0
        return out

    whole = run(p)
    halves = [parallel.select_batches(p, np.arange(a, b)) for a, b in ((0, 600), (600, 1250))]
    assert all(8 * h.wave_len < (512 << 20) for h in halves)
    parts = run(halves[0]) + run(halves[1])
    assert float((whole - parts).abs().max()) < 1e-13 * float(parts.abs().max())
    assert float(parts.abs().max()) > 0


def _adjoint_reference(p, gr, gg):
    want = np.zeros((p.n_basis, p.n_basis, p.T))
    for b in range(p.n_my_batches_work):
        nc, npb, o = (int(v) for v in (p.n_compute_c_batches[b], p.n_point_batches[b], p.i_batch_2_wave_offset[b]))
        ncp, pre = (nc + 3) // 4 * 4, int(p.n_point_batches_prefix_sum[b])
        phi = p.wave[o:o + ncp * npb].reshape(npb, ncp)[:, :nc]
        gphi = p.gradient_wave[3 * o:3 * (o + ncp * npb)].reshape(npb, 3, ncp)[:, :, :nc]
        ib = p.i_basis_batches[:nc, b] - 1
        for t in range(p.T):
            a = 2.0 * np.einsum("kp,pki->pi", gg[:, :npb, b, t], gphi)
            if t < p.j_atom_end - p.j_atom_begin + 1:
                a += gr[p.i_valid_point_2_i_full_points_map[pre:pre + npb], t][:, None] * phi
            want[np.ix_(ib, ib, [t])] += (a.T @ phi)[:, :, None]
    return want


@pytest.mark.parametrize("n_batches,np_range,nc_range,n_atoms,T,n_active", [
    (60, (100, 200), (40, 120), 8, 2, 1),   # several batches a group, one perturbation of two active
    (60, (100, 200), (40, 120), 8, 3, 3),
    (5, (290, 310), (480, 500), 30, 1, 1),  # every batch a group of its own (more than 1 MiB each)
])
def test_scratch_groups_match_oracle_and_one_group(n_batches, np_range, nc_range, n_atoms, T, n_active):
    """First-order H and the adjoint (g_rho and g_grad) with the points' A rows in
    groups of 1 MiB, against the oracle and, bit for bit, against one group: the
    scale and every contribution are the same.  At most 310 x 60 terms an entry."""
    p = synth.make_rho1_problem(T=T, seed=300 + n_batches, n_atoms=n_atoms, box=None, density=0.037,
                                n_batches=n_batches, np_range=np_range, nc_range=nc_range, pad_value=np.nan,
                                with_bias=True, n_active=n_active)
    xc = synth.first_order_h_inputs(p, seed=5, pad_value=np.nan)
    rng = np.random.default_rng(n_batches)
    v = np.asfortranarray(rng.normal(size=(p.n_full_points, T)))
    gr = rng.normal(size=(p.n_full_points, T))
    gg = rng.normal(size=(3, p.n_max_batch_size, p.n_my_batches_work, T))
    plan = _lib.Rho1Plan(p)
    assert plan.tuning()["h1_scratch_mb"] == 512
    d, vd, pt, av = _device_inputs(p, xc, v)
    w, gw, n = dev(p.wave), dev(p.gradient_wave), p.n_basis * p.n_basis * T
    out = []
    for mb in (512, 1, 2):
        plan.set_tuning(h1_scratch_mb=mb)
        H, dP1 = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
        for _ in range(2):  # the second call starts from the accumulator the first one left
            plan.first_order_h(n_active, p.n_atoms, 1, 3, av, w, gw, d["hessian_wave"], d, vd, pt, H)
            plan.adjoint_p1(n_active, w, gw, dev(gr), dev(gg), dP1)
        out.append((H, dP1))
    assert plan.device_flags() == 0
    ref = oracle.first_order_h(p, v, use_reference=oracle.ref_available(T), xc=xc, j_coord=3)
    want = _adjoint_reference(p, gr, gg)
    assert normwise_rel(0.5 * host(out[0][0], ref.shape), ref) < TOL
    assert normwise_rel(0.5 * host(out[0][1], want.shape), want) < TOL
    for H, dP1 in out[1:]:
        assert torch.equal(H, out[0][0]) and torch.equal(dP1, out[0][1])
    with pytest.raises(_lib.FrpaError):
        plan.set_tuning(h1_scratch_mb=0)


def test_dropin_calls_of_alternating_sizes():
    """The host-array entry keeps its device buffers, A among them, between calls:
    smaller and larger problems in turn give the bits of their first call, and the
    memory in use does not grow."""
    cases = [_case(1, 171, n_batches=6), _case(3, 172, n_batches=40), _case(2, 173, n_batches=12)]
    first, free = [], None
    for turn in range(3):
        for i, (p, xc, v) in enumerate(cases):
            H = _lib.dropin_first_order_h(p, v, xc, j_coord=2)
            if turn == 0:
                first.append(H)
                assert normwise_rel(H, _reference(p, v, xc, 2, 0.0)) < TOL
            assert np.array_equal(H, first[i])
        now = torch.cuda.mem_get_info()[0]
        assert free is None or now == free
        free = now if turn else None


def test_scratch_shrinks_where_it_cannot_be_allocated():
    """With less free memory than one group's A rows take (170 MB), the call goes
    through smaller groups; the accumulator alone (0.4 MB) always fits."""
    p = synth.make_rho1_problem(T=1, seed=310, n_batches=1500, np_range=(150, 200), nc_range=(60, 100), eval_phi=False)
    assert 8 * p.wave_len > 150 << 20
    w = torch.empty(p.wave_len, dtype=torch.float64, device="cuda")
    gw = torch.empty(3 * p.wave_len, dtype=torch.float64, device="cuda")
    _lib.synth_basis_values(p, dev(np.asfortranarray(p.valid_points_xyz.T)), w, gw)
    gr = dev(np.random.default_rng(3).normal(size=p.n_full_points))
    out = [torch.zeros(p.n_basis * p.n_basis, dtype=torch.float64, device="cuda") for _ in range(2)]
    plans = [_lib.Rho1Plan(p) for _ in range(2)]
    plans[0].adjoint_p1(1, w, gw, gr, None, out[0])
    torch.cuda.synchronize()
    plans[0].close()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        plans[1].adjoint_p1(1, w, gw, gr, None, out[1])
        torch.cuda.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert plans[1].device_flags() == 0
    assert torch.equal(out[0], out[1])
