"""The calls a DFPT program makes of this library, as timed cases.

Every case goes through the public Python mirror of the C ABI: plans on device
arrays (`_lib.Rho1Plan`, `_lib.SumupPlan`), the autograd pairs
(`autograd.rho1`, `autograd.sumup`) and the reference-named host entry point
(`_lib.dropin_rho1`).  Inputs are drawn on the GPU from the seed: atoms on a
jittered lattice, Cartesian Gaussian functions, grid batches in a ball around
an atom with the strongest functions over that ball, sizes as in the
workloads of bench.py and of the tests.

`exact` restates each path in plain torch, FP64, from the same inputs.
"""

from __future__ import annotations

import math
import types

import numpy as np
import torch

from fast_rpa_eval_b200 import _lib, autograd, tables

F64 = torch.float64
POINT_RADIUS = 3.0  # A, ball of a batch's points around its atom

# (degree, exponents of x, y, z) of an atom's functions, shell by shell: a
# shell shares one Gaussian exponent
SHELLS = {
    10: [[(0, 0, 0)]] * 3 + [[(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (0, 2, 1), (1, 0, 2), (1, 1, 1)]],
    20: [[(0, 0, 0)]] * 4 + [[(1, 0, 0), (0, 1, 0), (0, 0, 1)]] * 2
    + [[(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (0, 1, 1)]] * 2,
}


# ------------------------------------------------------------------- cases


def listed():
    adjoint = dict(atoms=200, functions=20, density=0.1, batches=1600, np_lo=100, np_hi=200, nc_lo=40, nc_hi=120,
                   log=False, T=1)
    return [
        # a small molecule's density response (8 atoms, 64 batches): latency and launches
        dict(name="rho1_small", op="rho1", mode="fp64", atoms=8, functions=20, density=0.037, batches=64, np_lo=100,
             np_hi=200, nc_lo=40, nc_hi=120, log=False, T=1),
        # four perturbations at once on very uneven batches (the benchmark sweep's spread)
        dict(name="rho1_tile4", op="rho1", mode="fp64", atoms=200, functions=20, density=0.037, batches=800, np_lo=50,
             np_hi=400, nc_lo=50, nc_hi=800, log=True, T=4),
        # the benchmark's 1,000-atom step with as many batches as fit the card three times over
        dict(name="rho1_large", op="rho1", mode="fp64", atoms=1000, functions=10, density=0.1, batches=8000,
             np_lo=100, np_hi=300, nc_lo=100, nc_hi=600, log=False, T=1),
        # the same step in the split-precision mode
        dict(name="rho1_i8", op="rho1", mode="i8", atoms=1000, functions=10, density=0.1, batches=8000, np_lo=100,
             np_hi=300, nc_lo=100, nc_hi=600, log=False, T=1),
        # forward and backward of rho1 and its gradient, 200 atoms: dL/dP1 of a training step
        dict(name="rho1_step", op="rho1_step", mode="fp64", **adjoint),
        # the first-order H integration with every exchange-correlation term, 200 atoms
        dict(name="first_order_h", op="h", mode="fp64", **adjoint),
        # the density-matrix bias of four atoms, before every rho1 step of a CPSCF cycle
        dict(name="bias_part2", op="bias", mode="fp64", atoms=1000, functions=10, density=0.1, batches=4000,
             np_lo=100, np_hi=300, nc_lo=100, nc_hi=600, log=False, T=4),
        # the reference's host-array entry point on a small molecule: plan, copies and kernel in one call
        dict(name="rho1_dropin", op="dropin", mode="fp64", atoms=8, functions=20, density=0.037, batches=64,
             np_lo=100, np_hi=200, nc_lo=40, nc_hi=120, log=False, T=1),
        # a small molecule's Hartree potential
        dict(name="sumup_small", op="sumup", atoms=20, points=2000, L=4, T=1, outer=0.0),
        # the benchmark's potential: 500 atoms, 2 million points
        dict(name="sumup_large", op="sumup", atoms=500, points=2_000_000, L=6, T=1, outer=0.0),
        # four perturbations, highest l, moments cut off with distance
        dict(name="sumup_tile4", op="sumup", atoms=150, points=60_001, L=8, T=4, outer=8.0),
        # forward and backward of the potential, 100 atoms: dL/dQ of a training step
        dict(name="sumup_step", op="sumup_step", atoms=100, points=200_000, L=6, T=1, outer=8.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["rho1", "rho1", "rho1", "rho1_step", "h", "bias", "dropin", "sumup", "sumup", "sumup_step"])
    if op.startswith("sumup"):
        L = rng.choice([4, 5, 6, 7, 8])
        T = rng.choice([1, 1, 2, 3, 4])
        atoms = _log_int(rng, 12, 500)
        top = 4e8 if op == "sumup" else 2e7
        points = max(500, min(_log_int(rng, 1000, 2_000_000), int(top / (atoms * T * (L + 1) ** 2 / 49))))
        return dict(op=op, atoms=atoms, points=points, L=L, T=T, outer=rng.choice([0.0, round(rng.uniform(5.0, 10.0), 3)]))
    mode = rng.choice(["fp64", "fp64", "i8"]) if op == "rho1" else "fp64"
    functions = rng.choice([10, 20])
    atoms = _log_int(rng, 8, 16 if op == "dropin" else 400)
    n_basis = atoms * functions
    nc_lo = rng.randint(20, min(100, n_basis // 2))
    nc_hi = min(n_basis, _log_int(rng, nc_lo + 10, 120 if op in ("h", "rho1_step", "dropin") else 800))
    np_lo = rng.randint(50, 120)
    np_hi = rng.randint(np_lo + 1, 400)
    T = rng.choice([1, 1, 1, 2, 3, 4])
    if op in ("h", "rho1_step"):
        T = min(T, 2)
    if op == "dropin":
        T = 1
    # at most about the listed cases' arrays and products
    top = 0.4e9 if op == "rho1" else 0.2e9 if op != "dropin" else 4e5
    batches = _log_int(rng, 40, 6000)
    batches = max(20, min(batches, int(top / (nc_hi * np_hi * T))))
    return dict(op=op, mode=mode, atoms=atoms, functions=functions, density=rng.choice([0.037, 0.1]), batches=batches,
                np_lo=np_lo, np_hi=np_hi, nc_lo=nc_lo, nc_hi=nc_hi, log=rng.random() < 0.5, T=T)


# ------------------------------------------------------------- rho1 inputs


def _span(rng, lo, hi, log, size):
    if log:
        v = np.floor(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), size))).astype(np.int64)
        return v.clip(lo, hi)
    return rng.integers(lo, hi + 1, size)


def _batch_shapes(case):
    """Points and functions of every batch: part of the case, not of the seed,
    so that every problem of a case has arrays of the same sizes."""
    rng = np.random.default_rng([case[k] for k in ("batches", "np_lo", "np_hi", "nc_lo", "nc_hi")])
    npts = _span(rng, case["np_lo"], case["np_hi"], case["log"], case["batches"])
    ncs = _span(rng, case["nc_lo"], case["nc_hi"], case["log"], case["batches"])
    return npts, np.minimum(ncs, case["atoms"] * case["functions"])


def _lattice(n, spacing, rng):
    side = int(math.ceil(round(n ** (1.0 / 3.0), 6)))
    cells = rng.permutation(side**3)[:n]
    grid = np.stack([cells // (side * side), cells // side % side, cells % side], axis=1).astype(np.float64)
    return (grid + 0.5 + rng.uniform(-0.25, 0.25, (n, 3))) * spacing, side * spacing


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=F64)


def _uniform(gen, lo, hi, *shape):
    return torch.rand(shape, generator=gen, device="cuda", dtype=F64) * (hi - lo) + lo


def _rho1_inputs(case, seed):
    """Geometry (host), wave arrays and density matrix (device) of one problem,
    in the reference's layouts."""
    rng = np.random.default_rng(seed)
    gen = _gen(seed)
    A, F, nb, T = case["atoms"], case["functions"], case["batches"], case["T"]
    g = types.SimpleNamespace(T=T, n_atoms=A, n_basis=A * F, n_my_batches_work=nb)
    atoms, _ = _lattice(A, case["density"] ** (-1.0 / 3.0), rng)
    shells = SHELLS[F]
    alpha = np.exp(rng.uniform(math.log(0.1), math.log(10.0), (A, len(shells))))
    alpha = np.concatenate([np.repeat(alpha[:, s : s + 1], len(sh), axis=1) for s, sh in enumerate(shells)], axis=1)
    power = np.array([m for sh in shells for m in sh], dtype=np.float64)  # (F, 3)

    npts, ncs = _batch_shapes(case)
    centre = rng.integers(0, A, nb)
    nc_max = int(ncs.max())

    # the strongest functions of each batch by their radial envelope over its ball
    at = torch.from_numpy(atoms).cuda()
    al = torch.from_numpy(alpha).cuda().reshape(-1)
    deg = torch.from_numpy(np.tile(power.sum(axis=1), A)).cuda()
    rstar = torch.sqrt(deg / (2.0 * al))
    nc_t = torch.from_numpy(ncs).cuda()
    ib = torch.empty((nb, nc_max), dtype=torch.int64, device="cuda")
    for b0 in range(0, nb, 2048):
        c = at[torch.from_numpy(centre[b0 : b0 + 2048]).cuda()]
        d = torch.linalg.norm(c[:, None, :] - at[None, :, :], dim=2).repeat_interleave(F, dim=1)
        r = torch.minimum(torch.maximum(rstar, (d - POINT_RADIUS).clamp(min=0.0)), d + POINT_RADIUS)
        score = deg * torch.log(r.clamp(min=1e-30)) - al * r * r
        top = torch.topk(score, nc_max, dim=1).indices
        keep = torch.arange(nc_max, device="cuda")[None, :] < nc_t[b0 : b0 + 2048, None]
        ib[b0 : b0 + 2048] = torch.where(keep, top, g.n_basis).sort(dim=1).values
    g.ib = ib  # (nb, nc_max), 0-based, ascending; n_basis past n_compute
    g.ncs, g.npts = ncs, npts

    prefix = np.zeros(nb + 1, np.int64)
    prefix[1:] = np.cumsum(npts)
    n_valid = int(prefix[-1])
    g.n_full_points = n_valid + n_valid // 16 + 1
    perm = rng.permutation(g.n_full_points).astype(np.int32)
    ncp = (ncs + 3) // 4 * 4
    off = np.zeros(nb + 1, np.int64)
    off[1:] = np.cumsum(ncp * npts)
    g.wave_len, g.off, g.ncp = int(off[-1]), off, ncp
    g.n_max_batch_size = int(npts.max())
    g.n_centers_basis_I = nc_max
    g.n_point_batches = npts.astype(np.int32)
    g.n_point_batches_prefix_sum = prefix.astype(np.int32)
    g.i_valid_point_2_i_full_points_map = perm
    g.n_compute_c_batches = ncs.astype(np.int32)
    one_based = torch.where(ib < g.n_basis, ib + 1, 0).to(torch.int32).cpu().numpy()
    g.i_basis_batches = one_based.T  # (nc_max, nb), Fortran order
    g.i_batch_2_wave_offset = off.astype(np.int32)
    g.map = torch.from_numpy(perm).cuda().long()

    # points: uniform in the ball; phi and grad phi of the Cartesian Gaussians
    u = _randn(gen, n_valid, 3)
    u = u / torch.linalg.norm(u, dim=1, keepdim=True)
    owner = torch.repeat_interleave(torch.arange(nb, device="cuda"), torch.from_numpy(npts).cuda())
    pts = at[torch.from_numpy(centre).cuda()[owner]] + POINT_RADIUS * u * _uniform(gen, 0.0, 1.0, n_valid, 1) ** (1.0 / 3.0)
    g.wave = torch.empty(g.wave_len, dtype=F64, device="cuda")
    g.gwave = torch.empty(3 * g.wave_len, dtype=F64, device="cuda")
    pw = torch.from_numpy(power).cuda()
    off_t, ncp_t, pre_t = (torch.from_numpy(a).cuda() for a in (off, ncp, prefix))
    b0 = 0
    while b0 < nb:  # whole batches, about 2^25 elements at a time
        b1 = max(b0 + 1, int(np.searchsorted(off, off[b0] + (1 << 25), side="right")) - 1)
        b1 = min(b1, nb)
        lo, hi = int(off[b0]), int(off[b1])
        b = torch.repeat_interleave(torch.arange(b0, b1, device="cuda"), (off_t[b0 + 1 : b1 + 1] - off_t[b0:b1]))
        e = torch.arange(lo, hi, device="cuda") - off_t[b]
        p, i = e // ncp_t[b], e % ncp_t[b]
        live = i < nc_t[b]
        f = torch.where(live, ib[b, torch.where(live, i, 0)], 0)
        x = pts[pre_t[b] + p] - at[f // F]
        n = pw[f % F]
        a = al[f]
        gauss = torch.where(live, torch.exp(-a * (x * x).sum(dim=1)), 0.0)
        m = torch.pow(x, n)
        dm = n * torch.pow(x, (n - 1.0).clamp(min=0.0)) - 2.0 * a[:, None] * x * m
        g.wave[lo:hi] = m.prod(dim=1) * gauss
        at3 = 3 * off_t[b] + 3 * p * ncp_t[b] + i
        for d in range(3):
            g.gwave[at3 + d * ncp_t[b]] = dm[:, d] * m[:, (d + 1) % 3] * m[:, (d + 2) % 3] * gauss
        b0 = b1

    scale = 1.0 / math.sqrt(2.0 * float(ncs.mean()))
    P1 = []
    for _ in range(T):
        a = _randn(gen, g.n_basis, g.n_basis) * scale
        P1.append(a + a.T)
    g.P1 = torch.stack(P1)  # (T, n, n) C order = (n, n, T) Fortran order, symmetric
    del P1, a
    nmb = g.n_max_batch_size
    g.bias = _uniform(gen, -1.0, 1.0, T, nb, nmb)
    g.gbias = _uniform(gen, -1.0, 1.0, T, nb, nmb, 3)
    g.gen = gen
    return g


def _atom_valid(g, F):
    """(n_atoms + 1, n_batches) Fortran: running counts of a batch's functions by atom."""
    edge = (torch.arange(g.n_atoms + 1, device="cuda") * F).expand(g.n_my_batches_work, -1).contiguous()
    return torch.searchsorted(g.ib, edge).to(torch.int32).contiguous()


def _h_inputs(g):
    gen, nb, nmb, nf, T = g.gen, g.n_my_batches_work, g.n_max_batch_size, g.n_full_points, g.T
    xc = dict(vsigma=0.5 * _randn(gen, nb, nmb, 3), gradient_rho=_randn(gen, nf, 3), H_prefactor1=_randn(gen, T, nb, nmb),
              first_order_gradient_rho=_randn(gen, T, nb, nmb, 3), first_order_rho=_randn(gen, T, nf),
              v2rho2=0.3 * _randn(gen, nb, nmb, 3), v2rhosigma=0.2 * _randn(gen, nb, nmb, 6),
              v2sigma2=0.1 * _randn(gen, nb, nmb, 6))
    hess = 0.3 * _randn(gen, 6 * g.wave_len)
    return xc, hess, _randn(gen, T, nf), _uniform(gen, 0.01, 1.0, nf)


# ----------------------------------------------------------- sum-up inputs


def _sumup_inputs(case, seed):
    rng = np.random.default_rng(seed)
    gen = _gen(seed)
    A, nv, L, T = case["atoms"], case["points"], case["L"], case["T"]
    L2, ngrid, nsp = (L + 1) ** 2, 1301, 4
    s = types.SimpleNamespace(T=T, n_atoms=A, n_valid_points=nv, l_pot_max=L, n_hartree_grid=ngrid, n_species=nsp,
                              n_full_points=nv + nv // 16 + 1, n_centers=A, n_centers_hartree_potential=A,
                              hartree_force_l_add=1, l_max_analytic_multipole=L + 1)
    atoms, box = _lattice(A, 0.1 ** (-1.0 / 3.0), rng)
    s.coords_center = np.asfortranarray(atoms.T)
    s.coord_points = np.asfortranarray(rng.uniform(-3.0, box + 3.0, (s.n_full_points, 3)).T)
    s.i_valid_point_2_i_full_points_map = rng.permutation(s.n_full_points)[:nv].astype(np.int32)
    s.species = rng.integers(1, nsp + 1, A).astype(np.int32)
    s.species_center = s.species.copy()
    s.l_hartree = np.full(nsp, L, np.int32)
    if case["outer"] > 0.0:
        s.l_hartree[1] = max(1, L - 1)
        s.l_hartree[2] = max(1, L - 2)
    s.n_grid = np.full(nsp, ngrid, np.int32)
    s.r_grid_min = 1e-4 * rng.uniform(0.5, 2.0, nsp)
    s.log_r_grid_inc = math.log(1e6) / (ngrid - 1) * rng.uniform(0.95, 1.05, nsp)
    s.center_to_atom = np.arange(1, A + 1, dtype=np.int32)
    s.centers_hartree_potential = np.arange(1, A + 1, dtype=np.int32)
    i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()  # noqa: E731
    s.lhmfd = i32(np.tile(s.l_hartree[s.species - 1], (T, 1)))  # (T, A)
    s.mrs = 4.0 * _uniform(gen, 0.9, 1.1, T, A)
    if case["outer"] > 0.0:
        base = case["outer"] * _uniform(gen, 0.8, 1.2, T, A, 1)
        s.opr = (base / (1.0 + 0.15 * torch.arange(L + 1, device="cuda", dtype=F64))) ** 2
    else:
        s.opr = torch.full((T, A, L + 1), 1e30, dtype=F64, device="cuda")
    decay = torch.cat([torch.full((2 * l + 1,), 10.0**-l, dtype=F64) for l in range(L + 1)]).cuda()
    s.Q = _randn(gen, T, A, L2) * decay
    s.Q[torch.rand((T, A, L2), generator=gen, device="cuda") < 0.02] = 1e-12
    s.spline = _uniform(gen, -0.01, 0.01, T, A, ngrid, 2, L2)
    s.dv0 = _uniform(gen, -1.0, 1.0, T, s.n_full_points)
    s.g = _uniform(gen, 0.01, 1.0, s.n_full_points) * _randn(gen, T, s.n_full_points)
    return s


# ----------------------------------------------------------------- prepare


def prepare(case, seed):
    op = case["op"]
    if op.startswith("sumup"):
        s = _sumup_inputs(case, seed)
        s.index_cc, s.cc, s.n_cc_lm_ijk, s.index_ijk_max_cc = tables.multipole_tables(s.l_max_analytic_multipole)
        s.index_cc_dim_0 = int(s.n_cc_lm_ijk[-1])
        s.case, s.plan = case, _lib.SumupPlan(s)
        s.dv = torch.empty_like(s.dv0)
        if op == "sumup_step":
            s.Q.requires_grad_(True)
        else:
            del s.g, s.dv0
        return s
    g = _rho1_inputs(case, seed)
    g.case = case
    T, nb, nmb = g.T, g.n_my_batches_work, g.n_max_batch_size
    if op == "dropin":  # host arrays, as the caller of the reference's entry point holds them
        h = lambda t: t.cpu().numpy().ravel()  # noqa: E731
        g.j_atom_begin, g.j_atom_end, g.j_coord = 1, T, 1
        g.n_max_compute_ham, g.batch_sizes = int(g.ncs.max()), g.n_point_batches
        g.atom_valid_n_compute_c_batches = h(_atom_valid(g, case["functions"]))
        g.basis_atom = (np.arange(g.n_basis) // case["functions"] + 1).astype(np.int32)
        g.partition_tab, g.density_matrix = np.ones(g.n_full_points), None
        g.wave, g.gradient_wave = h(g.wave), h(g.gwave)
        g.first_order_density_matrix, g.first_order_rho_bias_part2 = h(g.P1), h(g.bias)
        g.first_order_gradient_rho_bias = h(g.gbias)
        g.rho, g.grad = np.zeros(g.n_full_points * T), np.zeros(3 * nmb * nb * T)
        return g
    g.plan = _lib.Rho1Plan(g)
    if op == "rho1":
        g.rho = torch.empty(T, g.n_full_points, dtype=F64, device="cuda")
        g.grad = torch.empty(T, nb, nmb, 3, dtype=F64, device="cuda")
        g.mode = _lib.RHO1_SPLIT_I8 if case["mode"] == "i8" else _lib.RHO1_FP64
    elif op == "rho1_step":
        g.P1 = g.P1.reshape(-1).requires_grad_(True)
        g.g_rho, g.g_grad = _step_upstream(g)
    elif op == "h":
        g.xc, g.hess, g.vhg, g.ptab = _h_inputs(g)
        g.atom_valid = _atom_valid(g, case["functions"])
        g.H = torch.empty(T, g.n_basis, g.n_basis, dtype=F64, device="cuda")
    else:  # bias: P1 stands in for the ground-state density matrix
        g.atom_valid = _atom_valid(g, case["functions"])
        g.dm = g.P1[0].contiguous()
        g.out = torch.zeros(T, nb, nmb, dtype=F64, device="cuda")
        del g.P1, g.bias, g.gbias
    return g


def _step_upstream(g):
    """Upstream gradients of a loss over both outputs (drawn after the inputs)."""
    w = _uniform(g.gen, 0.01, 1.0, g.n_full_points)
    return ((w * _randn(g.gen, g.T, g.n_full_points)).reshape(-1),
            _randn(g.gen, 3 * g.n_max_batch_size * g.n_my_batches_work * g.T))


def _first_atom(g):
    return 1 + (g.n_atoms - g.T) // 2  # a perturbation tile in the middle of the atoms


# --------------------------------------------------------------------- run


def run(s):
    op = s.case["op"]
    if op == "rho1":
        s.plan.execute(s.T, s.wave, s.gwave, s.P1, s.bias, s.gbias, s.rho, s.grad, mode=s.mode)
        return {"rho1": s.rho, "grad": s.grad}
    if op == "rho1_step":
        s.P1.grad = None
        rho, grad = autograd.rho1(s.P1, s.plan, s.wave, s.gwave, s.bias, s.gbias, s.T)
        torch.autograd.backward((rho, grad), (s.g_rho, s.g_grad))
        return {"rho1": rho.detach(), "grad": grad.detach(), "dP1": s.P1.grad}
    if op == "h":
        s.H.zero_()
        s.plan.first_order_h(s.T, s.n_atoms, _first_atom(s), 1, s.atom_valid, s.wave, s.gwave, s.hess, s.xc, s.vhg,
                             s.ptab, s.H)
        return {"H": s.H}
    if op == "bias":
        j = _first_atom(s)
        s.plan.bias_part2(s.T, s.n_atoms, j, j + s.T - 1, 1, s.atom_valid, s.wave, s.gwave, s.dm, s.out)
        return {"bias": s.out}
    if op == "dropin":
        rho, grad = _lib.dropin_rho1(s, rho=s.rho, grad=s.grad)
        return {"rho1": rho, "grad": grad}
    if op == "sumup":
        s.dv.zero_()
        s.plan.execute(s.T, s.lhmfd, s.mrs, s.opr, s.Q, s.spline, s.dv)
        return {"delta_v": s.dv}
    s.Q.grad = None
    dv = autograd.sumup(s.Q, s.plan, s.lhmfd, s.mrs, s.opr, s.spline, s.dv0, s.T)
    torch.autograd.backward((dv,), (s.g,))
    return {"delta_v": dv.detach(), "dQ": s.Q.grad}


# -------------------------------------------------------------------- work


def work(case):
    op, T = case["op"], case["T"]
    if op.startswith("sumup"):
        A, nv, L = case["atoms"], case["points"], case["L"]
        L2 = (L + 1) ** 2
        pairs = float(A) * nv * T
        back = 2 if op == "sumup_step" else 1
        # points in and out, moments, radii; of the spline what the near pairs
        # read (4 L2 values a pair, at most the table)
        near = min(1301.0 * 2 * L2 * A * T, 0.1 * 33.5 * nv * T * 4 * L2)
        return {"bytes": back * 8.0 * (nv * (3 + 2 * T) + A * T * (L2 + L + 3)) + 8.0 * near, "flops": back * pairs * 2 * L2}
    n_basis = case["atoms"] * case["functions"]
    pt, nc = (v.astype(np.float64) for v in _batch_shapes(case))
    matrix = 8.0 * T * min(float(n_basis) ** 2, float((nc * nc).sum()))
    pairs = float((nc * pt).sum())
    phi, rows = 8.0 * pairs, 8.0 * float(pt.sum())
    gemm = 2.0 * T * float((nc * nc * pt).sum())
    if op in ("rho1", "dropin"):
        return {"bytes": 4 * phi + matrix + 8 * T * rows, "flops": gemm + 8.0 * T * pairs}
    if op == "rho1_step":
        return {"bytes": 8 * phi + matrix + 8.0 * T * float(n_basis) ** 2 + 12 * T * rows, "flops": 2 * gemm + 16.0 * T * pairs}
    if op == "h":
        return {"bytes": 4 * phi + 8.0 * T * float(n_basis) ** 2 + (8 + 6 * T) * rows, "flops": gemm + 8.0 * T * pairs}
    # bias: the batches that hold one of the tile's atoms (about nc / functions of them each)
    held = T * float(nc.mean()) / n_basis  # of one batch, over the tile's atoms
    share = min(1.0, held)
    return {"bytes": share * phi + T * rows + 8.0 * T * case["functions"] * n_basis,
            "flops": 2.0 * held * case["functions"] * pairs}


# ------------------------------------------------------------------- exact


def _batch_blocks(g):
    for b in range(g.n_my_batches_work):
        nc, npb, ncp, o = int(g.ncs[b]), int(g.npts[b]), int(g.ncp[b]), int(g.off[b])
        phi = g.wave[o : o + ncp * npb].view(npb, ncp)[:, :nc]
        gphi = g.gwave[3 * o : 3 * (o + ncp * npb)].view(npb, 3, ncp)[:, :, :nc]
        pre = int(g.n_point_batches_prefix_sum[b])
        yield b, nc, npb, ncp, g.ib[b, :nc], phi, gphi, g.map[pre : pre + npb]


def _exact_rho1(g):
    rho = torch.zeros(g.T, g.n_full_points, dtype=F64, device="cuda")
    grad = torch.zeros(g.T, g.n_my_batches_work, g.n_max_batch_size, 3, dtype=F64, device="cuda")
    for b, nc, npb, ncp, ib, phi, gphi, full in _batch_blocks(g):
        for t in range(g.T):
            w = phi @ g.P1[t][ib[:, None], ib[None, :]]
            rho[t, full] = (phi * w).sum(dim=1) + g.bias[t, b, :npb]
            grad[t, b, :npb] = 2.0 * (gphi * w[:, None, :]).sum(dim=2) - g.gbias[t, b, :npb]
    return rho, grad


def _exact_dP1(g, g_rho, g_grad):
    d = torch.zeros(g.T, g.n_basis, g.n_basis, dtype=F64, device="cuda")
    for b, nc, npb, ncp, ib, phi, gphi, full in _batch_blocks(g):
        for t in range(g.T):
            a = g_rho[t, full][:, None] * phi + 2.0 * (g_grad[t, b, :npb][:, :, None] * gphi).sum(dim=1)
            # entry (i, j) of the Fortran-ordered matrix: position j n + i
            d[t][ib[:, None], ib[None, :]] += phi.T @ a
    return d


def _exact_h(g, F):
    xc, hess, vhg, ptab = _h_inputs(g)
    av = _atom_valid(g, F).cpu().numpy()
    H = torch.zeros(g.T, g.n_basis, g.n_basis, dtype=F64, device="cuda")
    j0 = _first_atom(g)
    for b, nc, npb, ncp, ib, phi, gphi, full in _batch_blocks(g):
        o = int(g.off[b])
        hx = hess[6 * o : 6 * (o + ncp * npb)].view(npb, 6, ncp)[:, :3, :nc]  # d_k d_x for k = x, y, z
        vsig, v2r2 = xc["vsigma"][b, :npb, 0], xc["v2rho2"][b, :npb, 0]
        v2rs, v2s2 = xc["v2rhosigma"][b, :npb, 0], xc["v2sigma2"][b, :npb, 0]
        gr, w = xc["gradient_rho"][full], ptab[full]
        for t in range(g.T):
            fog, r1 = xc["first_order_gradient_rho"][t, b, :npb], xc["first_order_rho"][t, full]
            lfos = 2.0 * (fog * gr).sum(dim=1)
            inner = v2rs * r1 + v2s2 * lfos
            c_grad = 2.0 * w[:, None] * (gr * inner[:, None] + vsig[:, None] * fog)
            pf3 = w * (vhg[t, full] + v2r2 * r1 + v2rs * lfos)
            c_phi = 0.5 * (xc["H_prefactor1"][t, b, :npb] + pf3)
            a = c_phi[:, None] * phi + (c_grad[:, :, None] * gphi).sum(dim=1)
            v0, v1 = int(av[b, j0 + t - 1]), int(av[b, j0 + t])
            if v1 > v0:
                a[:, v0:v1] += ((-2.0 * vsig * w)[:, None, None] * gr[:, :, None] * hx[:, :, v0:v1]).sum(dim=1)
            m = a.T @ phi
            H[t][ib[:, None], ib[None, :]] += m + m.T
    return H


def _exact_bias(g, F):
    av = _atom_valid(g, F).cpu().numpy()
    out = torch.zeros(g.T, g.n_my_batches_work, g.n_max_batch_size, dtype=F64, device="cuda")
    dm, j0 = g.P1[0], _first_atom(g)
    for b, nc, npb, ncp, ib, phi, gphi, full in _batch_blocks(g):
        for t in range(g.T):
            v0, v1 = int(av[b, j0 + t - 1]), int(av[b, j0 + t])
            if v1 > v0:
                k = ib[v0:v1]
                S = dm[ib[:, None], k[None, :]] + dm[k[None, :], ib[:, None]]
                out[t, b, :npb] = -((phi @ S) * gphi[:, 0, v0:v1]).sum(dim=1)
    return out


def _harmonics(x, y, z, L):
    """Real spherical harmonics Y_lm of unit vectors, l-major, one tensor each."""
    Y = [None] * (L + 1) ** 2
    C, S, dfact = torch.ones_like(x), torch.zeros_like(x), 1.0
    for m in range(L + 1):
        if m > 0:
            C, S = x * C - y * S, x * S + y * C
            dfact *= 2 * m - 1
        q1 = q2 = None
        for l in range(m, L + 1):
            q = torch.full_like(x, dfact) if l == m else ((2 * l - 1) * z * q1 - ((l + m - 1) * q2 if q2 is not None else 0.0)) / (l - m)
            q1, q2 = q, q1
            k = math.sqrt((2 * l + 1) / (4.0 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                Y[l * l + l] = k * q
            else:
                k *= math.sqrt(2.0)
                Y[l * l + l + m] = (-k if m & 1 else k) * q * C
                Y[l * l + l - m] = k * q * S
    return Y


def _exact_sumup(s, backward):
    A, L, T = s.n_atoms, s.l_pot_max, s.T
    L2 = (L + 1) ** 2
    at = torch.from_numpy(np.ascontiguousarray(s.coords_center.T)).cuda()
    full = torch.from_numpy(s.i_valid_point_2_i_full_points_map).cuda().long()
    pts = torch.from_numpy(np.ascontiguousarray(s.coord_points.T)).cuda()[full]
    sp = torch.from_numpy(s.species.astype(np.int64)).cuda() - 1
    lam0 = torch.from_numpy(s.l_hartree.astype(np.int64)).cuda()[sp]
    rgm, linc = torch.from_numpy(s.r_grid_min).cuda()[sp], torch.from_numpy(s.log_r_grid_inc).cuda()[sp]
    l_of = torch.tensor([l for l in range(L + 1) for _ in range(2 * l + 1)], device="cuda")
    dv = (s.dv0.clone() if backward else torch.zeros_like(s.dv0))
    dQ = torch.zeros(T, A, L2, dtype=F64, device="cuda")
    step = max(1, int(4e6) // A)
    for p0 in range(0, s.n_valid_points, step):
        f = full[p0 : p0 + step]
        d = pts[p0 : p0 + step, None, :] - at[None, :, :]
        d2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]
        r = torch.sqrt(d2)
        Y = _harmonics(d[..., 0] / r, d[..., 1] / r, d[..., 2] / r, L)
        for t in range(T):
            keep = (s.Q[t].abs() > 1e-10) & (l_of[None, :] <= s.lhmfd[t][:, None])
            Q = torch.where(keep, s.Q[t], 0.0)
            lam = lam0[None, :].expand_as(d2).clone()
            for l in range(L, 0, -1):
                lam = torch.where((lam == l) & (s.opr[t, :, l][None, :] < d2), l - 1, lam)
            near = d2 < s.mrs[t][None, :]
            v = torch.zeros_like(d2)
            rl = torch.where(near | (d2 >= 1e8), 0.0, 1.0 / r)
            for l in range(L + 1):
                rlm = torch.where(lam >= l, rl, 0.0)
                part = sum(Y[k] * Q[:, k][None, :] for k in range(l * l, (l + 1) * (l + 1)))
                v += rlm * part
                if backward:
                    gr = s.g[t, f][:, None] * rlm
                    for k in range(l * l, (l + 1) * (l + 1)):
                        dQ[t, :, k] += (gr * Y[k]).sum(dim=0)
                rl = rl / r
            ip, ia = torch.nonzero(near, as_tuple=True)
            if len(ip):
                x = 1.0 + torch.log(r[ip, ia] / rgm[ia]) / linc[ia]
                i = x.long().clamp(1, s.n_hartree_grid - 1)
                u = x - i
                h = ((u - 1) ** 2 * (1 + 2 * u), (u - 1) ** 2 * u, u * u * (3 - 2 * u), u * u * (u - 1))
                n0, n1 = s.spline[t, ia, i - 1], s.spline[t, ia, i]  # (pairs, 2, L2)
                c = n0[:, 0] * h[0][:, None] + n0[:, 1] * h[1][:, None] + n1[:, 0] * h[2][:, None] + n1[:, 1] * h[3][:, None]
                ys = torch.stack([y[ip, ia] for y in Y], dim=1)
                v[ip, ia] += torch.where(l_of[None, :] <= lam[ip, ia][:, None], c * ys, 0.0).sum(dim=1)
            dv[t, f] += v.sum(dim=1)
            if backward and p0 + step >= s.n_valid_points:
                dQ[t] = torch.where(keep, dQ[t], 0.0)
    return dv, dQ


def exact(case, seed):
    op = case["op"]
    if op.startswith("sumup"):
        s = _sumup_inputs(case, seed)
        dv, dQ = _exact_sumup(s, op == "sumup_step")
        return {"delta_v": dv, "dQ": dQ} if op == "sumup_step" else {"delta_v": dv}
    g = _rho1_inputs(case, seed)
    if op == "h":
        return {"H": _exact_h(g, case["functions"])}
    if op == "bias":
        return {"bias": _exact_bias(g, case["functions"])}
    rho, grad = _exact_rho1(g)
    if op == "dropin":  # (n_full, T) and (3, n_max_batch_size, n_batches, T)
        return {"rho1": rho.T.cpu().numpy(), "grad": grad.permute(3, 2, 1, 0).cpu().numpy()}
    if op == "rho1_step":
        g_rho, g_grad = _step_upstream(g)
        d = _exact_dP1(g, g_rho.view(g.T, -1), g_grad.view(g.T, g.n_my_batches_work, g.n_max_batch_size, 3))
        return {"rho1": rho.reshape(-1), "grad": grad.reshape(-1), "dP1": d.reshape(-1)}
    return {"rho1": rho, "grad": grad}
