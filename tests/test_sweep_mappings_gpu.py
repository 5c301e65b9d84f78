"""The sweep's mappings of energies and columns to threads, its shortened
interior step and the paths beside it, the batch's merged launches and the
adjoint's bounded buffer, at the sizes where each can go wrong.  FP64 against
the CPU oracle to 1e-10 (the tolerance of the other parity tests); mixed
precision to 1e-5 of the bulk gap, the bound that FP32 stepping keeps
elsewhere."""
import copy

import numpy as np
import pytest

from tests import configs

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(np.max(np.abs(b)), 1e-300))


def _grain(temperature=0.1, disc=False, ppxi=5.0, size=None, angles=12):
    cfg = configs.small_disc() if disc else configs.small_square_d()
    cfg["physics"]["temperature"] = temperature
    cfg["numerics"]["points_per_coherence_length"] = ppxi
    cfg["numerics"]["num_fermi_momenta"] = angles
    shape = cfg["geometry"][0]
    if disc:
        shape["disc"]["radius"] = size or 3.0
    else:
        shape["regular_polygon"]["side_length"] = size or 5.0
    return cfg


def _pair(cfg, mode="fp64", scale=1.0):
    import superconga_b200 as sb
    from oracle import oracle as O
    o = O.Oracle(cfg)
    s = o.setup
    db = O.delta_bulk(s.temperature, s.symmetries[0])
    d, a = configs.seeded_state(s.n_comp, s.n0, db * scale, 7, 0.05, True, 0.05)
    e = sb.Context(cfg, mode=mode)
    o.set_state(d, a)
    e.set_state(d, a)
    return o, e, db


# Energy counts around the kernels' energies per thread (1, 2, 4, 5, 6, 7 in
# FP64; pairs in FP32) and their powers of two of threads: (temperature, count).
COUNTS = [(0.95, 5), (0.7, 6), (0.5, 7), (0.3, 8), (0.25, 9), (0.2, 10), (0.15, 12), (0.12, 13), (0.06, 18),
          (0.017, 34), (0.005, 63)]


@pytest.mark.parametrize("temperature,count", COUNTS)
@pytest.mark.parametrize("disc", [False, True])
def test_energy_counts(engine_lib, temperature, count, disc):
    cfg = _grain(temperature, disc)
    o, e, db = _pair(cfg)
    m = _pair(cfg, "mixed")[1]
    assert abs(e.dims.n_energies - count) <= 1
    for _ in range(2):
        o.compute()
        e.compute(1)
        m.compute(1)
    d_o, j_o, a_o = o.results()
    d_e, j_e, a_e = e.results()
    assert _rel(d_e, d_o) < TOL and _rel(j_e, j_o) < TOL and _rel(a_e, a_o) < TOL
    for which in range(4):
        assert _rel(e.boundary(which), o.boundary(which)) < TOL
    assert np.max(np.abs(m.results()[0] - d_o)) / db < 1e-5


@pytest.mark.parametrize("groups", ["1", "2", "8", "16"])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_threads_per_column(engine_lib, monkeypatch, groups, mode):
    """Every group size with an odd number of energies, on a rotated square
    (columns of even and odd length in one warp)."""
    monkeypatch.setenv("SCB_ENERGY_GROUPS", groups)
    cfg = _grain(0.12, ppxi=4.0, angles=14)
    o, e, db = _pair(cfg, mode)
    for _ in range(2):
        o.compute()
        e.compute(1)
    d_o, j_o, _ = o.results()
    d_e, j_e, _ = e.results()
    if mode == "fp64":
        assert _rel(d_e, d_o) < TOL and _rel(j_e, j_o) < TOL
    else:
        assert np.max(np.abs(d_e - d_o)) / db < 1e-5


def test_energy_passes_in_one_launch_and_many(engine_lib, monkeypatch):
    """89 energies: one launch with 16 threads per column, and the passes of 32
    that larger grains take."""
    cfg = _grain(0.0025)
    o, e, db = _pair(cfg)
    monkeypatch.setenv("SCB_ENERGY_GROUPS", "8")
    p = _pair(cfg)[1]
    assert e.dims.n_energies > 64
    for _ in range(2):
        o.compute()
        e.compute(1)
        p.compute(1)
    for c in (e, p):
        assert _rel(c.results()[0], o.results()[0]) < TOL
        for which in range(4):
            assert _rel(c.boundary(which), o.boundary(which)) < TOL


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_fields_too_large_for_the_short_step(engine_lib, mode):
    """An order parameter of 20 bulk gaps on two lattice points per xi0: no
    interior site allows the shortened step (0.625 h |Delta| > 1/4)."""
    o, e, db = _pair(_grain(0.3, ppxi=2.0, size=8.0), mode, scale=20.0)
    o.compute()
    e.compute(1)
    d_o, d_e = o.results()[0], e.results()[0]
    # mixed: the FP32 scalar steps keep about 1e-6 of the largest value
    assert _rel(d_e, d_o) < (TOL if mode == "fp64" else 1e-5)


def test_entering_values_outside_the_unit_disc(engine_lib):
    """Columns entered with |gamma| > 1 keep to the general step, whose root
    has a branch: the same outgoing values as the oracle's."""
    o, e, _ = _pair(_grain(0.3))
    rng = np.random.default_rng(5)
    for c in (o, e):
        getattr(c, "set_boundary_initial" if c is o else "boundary_initial")()
    for which in (0, 2):
        v = o.boundary(which)
        v = v * np.where(rng.uniform(size=v.shape) < 0.3, 1.5 / np.maximum(np.abs(v), 1e-3), 1.0)
        o.set_boundary(which, v)
        e.set_boundary(which, v)
    o.compute()
    e.compute(1)
    assert _rel(e.boundary(1), o.boundary(1)) < 1e-8  # values that grow along the column amplify rounding
    assert _rel(e.boundary(3), o.boundary(3)) < 1e-8


@pytest.mark.parametrize("per_block", [80, 132])
def test_ldos_blocks_in_one_pass_and_two(engine_lib, per_block):
    """Blocks of 80 and 132 real energies on a small grain: one pass, and two
    of 66 whose slice of the frame is not 16-byte aligned; mixed against FP64
    (1e-4 of the largest value, the bound of the other LDOS tests), FP64 against
    the passes of 32 (another order of nothing but the boundary: 1e-12)."""
    import os
    import superconga_b200 as sb
    sim = _grain(0.3, True, angles=16)
    out = {}
    for key, mode, env in (("fp64", "fp64", None), ("passes", "fp64", "8"), ("mixed", "mixed", None)):
        if env:
            os.environ["SCB_ENERGY_GROUPS"] = env
        try:
            e = sb.LdosContext(sim, configs.ldos_postprocess(0.2, n_energies=per_block, per_block=per_block, n_angles=16),
                               mode=mode)
        finally:
            os.environ.pop("SCB_ENERGY_GROUPS", None)
        d, a = configs.seeded_state(1, e.dims.n0, 0.2, 3, 0.05, True, 0.02)
        e.set_state(d, a)
        e.begin_block(0)
        e.burn_in(1)
        e.iterate(2)
        out[key] = e.ldos()
    assert _rel(out["passes"], out["fp64"]) < 1e-12
    assert _rel(out["mixed"], out["fp64"]) < 1e-4


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_batch_of_unlike_grains(engine_lib, mode):
    """Merged launches over grains whose kernels differ: one and two
    components, CongAcc, Anderson and Polyak, with and without a vector
    potential, energy passes; equal to the grains run alone."""
    import superconga_b200 as sb
    cfgs = [_grain(0.3), configs.chiral_annulus(), _grain(0.5, True), _grain(0.0025, size=4.0), _grain(0.2, True)]
    cfgs[2]["accelerator"] = {"name": "anderson"}
    cfgs[3]["accelerator"] = {"name": "polyak", "step_size": 0.5}
    cfgs[4]["physics"]["penetration_depth"] = -1.0
    for c in cfgs:
        c["numerics"]["convergence_criterion"] = 1e-30
    b = sb.Batch(copy.deepcopy(cfgs), mode=mode)
    alone = [sb.Context(c, mode=mode) for c in cfgs]
    for k, (g, s) in enumerate(zip(b.grains, alone)):
        d, a = configs.seeded_state(g.dims.n_comp, g.dims.n0, 0.2, 20 + k, 0.05, True, 0.02)
        g.set_state(d, a)
        s.set_state(d, a)
    b.compute(4)
    for g, s in zip(b.grains, alone):
        s.compute(4)
        # mixed: another number of threads per column adds the FP64 sums in
        # another order, which can move single FP32 roundings of the fields
        assert _rel(g.results()[0], s.results()[0]) < (1e-11 if mode == "fp64" else 1e-6)
        assert _rel(g.state()[0], s.state()[0]) < (1e-11 if mode == "fp64" else 1e-6)


@pytest.mark.parametrize("temperature", [0.3, 0.01])
def test_adjoint_in_many_launches(engine_lib, monkeypatch, temperature):
    """The buffer of the adjoint bounded to a few tiles, and more energies than
    one pass of 32 takes: the same gradients."""
    cfg = _grain(temperature, True)
    e = _pair(cfg)[1]
    e.boundary_initial()
    beta = np.random.default_rng(3).standard_normal((2, e.dims.n0, e.dims.n0))
    want = e.adjoint(0.7, beta)
    monkeypatch.setenv("SCB_SCRATCH_MB", "1")
    f = _pair(cfg)[1]
    f.boundary_initial()
    got = f.adjoint(0.7, beta)
    for x, y in zip(got, want):
        assert _rel(x, y) < 1e-11


def test_autograd_takes_tensors_of_any_place_and_layout(engine_lib):
    """CPU tensors, a conjugated view and a broadcast weight give the gradients
    of contiguous GPU tensors, on the tensors' own devices."""
    import superconga_b200 as sb
    import torch
    from superconga_b200 import autograd
    e = sb.Context(_grain(0.3, True), mode="fp64")
    n0 = e.dims.n0
    d, a = configs.seeded_state(1, n0, 0.2, 4, 0.05, True, 0.02)
    e.set_state(d, a)
    e.boundary_initial()
    row = np.random.default_rng(1).standard_normal((2, 1, n0))
    beta, spread = np.repeat(row, n0, axis=1), np.broadcast_to(row, (2, n0, n0))
    z = torch.from_numpy(d[:, 0] + 1j * d[:, 1])

    def grads(delta, av, b, weight=beta):
        loss = autograd.FreeEnergy.apply(delta, av, b, e, 1.0, weight)
        return (loss, *torch.autograd.grad(loss, [delta, av, b]))

    b0 = e.external_field()
    ref = grads(z.cuda().requires_grad_(), torch.from_numpy(a).cuda().requires_grad_(),
                torch.tensor(b0, dtype=torch.float64, device="cuda", requires_grad=True))
    cpu = grads(z.clone().requires_grad_(), torch.from_numpy(a).clone().requires_grad_(),
                torch.tensor(b0, dtype=torch.float64, requires_grad=True))
    view = z.conj().resolve_conj().cuda().conj().detach().requires_grad_()  # lazily conjugated
    at = torch.from_numpy(a).cuda().transpose(1, 2).contiguous().transpose(1, 2).detach().requires_grad_()
    got = grads(view, at, torch.tensor(b0, dtype=torch.float64, device="cuda", requires_grad=True), spread)
    for r, c, g in zip(ref, cpu, got):
        assert c.device.type == "cpu" and g.device.type == "cuda"
        assert _rel(c.detach().numpy(), r.detach().cpu().numpy()) < 1e-12
        assert _rel(g.detach().cpu().numpy(), r.detach().cpu().numpy()) < 1e-12


@pytest.mark.parametrize("broadening", [0.05, 0.02, 0.008])
def test_short_step_rounds_like_the_general_one(engine_lib, broadening):
    """The LDOS of a disc in FP64 against the oracle, which takes the general
    step everywhere.  A step rounds at about 2^-53 in both, a column remembers
    the last 1 / (2 h delta) sites (broadening delta), and independent errors
    add up as the square root of their number; the bound is 1.5 of that (B200:
    0.2).  An error that all steps of an energy share adds up in proportion to
    the sites (a rounded 1 + h e: 2 to 2.9)."""
    from oracle import oracle as O
    import superconga_b200 as sb
    points = 12.0
    sim = _grain(0.5, True, ppxi=points, size=6.0, angles=16)
    db = O.delta_bulk(0.5, "s")
    pp = configs.ldos_postprocess(db, n_energies=12, per_block=12, n_angles=16, broadening=broadening)
    L = O.LdosOracle(sim, pp)
    e = sb.LdosContext(sim, pp, mode="fp64")
    d, a = configs.seeded_state(1, e.dims.n0, db, 6, 0.05, True, 0.02)
    for c in (L, e):
        c.set_state(d, a)
        c.begin_block(0)
    L.iterate()
    e.iterate(1)
    diff = np.linalg.norm(e.ldos() - L.ldos) / np.linalg.norm(L.ldos)
    assert diff < 1.5 * 2.0 ** -53 * np.sqrt(points / (2.0 * broadening))


def test_the_adjoints_buffer_grows_when_memory_is_there(engine_lib, monkeypatch):
    """A first gradient with room for a few tiles only takes many launches; once
    the room is there, the next one takes as many as a context that always had
    it, and they agree."""
    cfg = _grain(0.3, True)
    e, f = _pair(cfg)[1], _pair(cfg)[1]
    for c in (e, f):
        c.boundary_initial()
    beta = np.random.default_rng(3).standard_normal((2, e.dims.n0, e.dims.n0))

    def gradient(c):
        n = c.launch_count()
        out = c.adjoint(0.7, beta)
        return out, c.launch_count() - n

    monkeypatch.setenv("SCB_SCRATCH_MB", "0.05")
    first, bounded = gradient(e)
    still, held = gradient(e)
    monkeypatch.delenv("SCB_SCRATCH_MB")
    again, free = gradient(e)
    want, launches = gradient(f)
    assert bounded == held > launches and free == launches
    for got in (first, still, again):
        for x, y in zip(got, want):
            assert _rel(x, y) < 1e-11


@pytest.mark.parametrize("per_block,groups", [(13, 4), (16, 4), (18, 8), (32, 8), (66, 8)])
def test_ldos_frames_of_four_energies_a_thread(engine_lib, monkeypatch, per_block, groups):
    """FP64 LDOS with four energies a thread: blocks whose sites are 32-byte
    aligned in the frame and blocks whose sites are not, a last thread with
    fewer than four, and a last pass of two: against the oracle (1e-10, as in
    the other parity tests)."""
    from oracle import oracle as O
    import superconga_b200 as sb
    monkeypatch.setenv("SCB_ENERGY_GROUPS", str(groups))
    sim = _grain(0.5, True, angles=16)
    db = O.delta_bulk(0.5, "s")
    pp = configs.ldos_postprocess(db, n_energies=per_block, per_block=per_block, n_angles=16)
    L = O.LdosOracle(sim, pp)
    e = sb.LdosContext(sim, pp, mode="fp64")
    d, a = configs.seeded_state(1, e.dims.n0, db, 6, 0.05, True, 0.02)
    for c in (L, e):
        c.set_state(d, a)
        c.begin_block(0)
    L.burn_in()
    e.burn_in(1)
    L.iterate()
    e.iterate(1)
    assert _rel(e.ldos(), L.ldos) < TOL
