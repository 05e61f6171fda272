"""Parity of the sm_100a engine with the FP64 oracle and the reference's golden vectors.

Tolerances: the double-precision engine agrees with the oracle to ~1e-10 relative; mixed precision
(FP32 pair/PME kernels, FP64 reductions) is held to 1e-6 relative in energy and 1e-5 RMS relative
in forces and induced dipoles, the bar the reference states for its mixed path against float64.
"""

import numpy as np
import pytest
import torch
from conftest import SMALL_BOX_SETTINGS

pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402


def ff_for(system, H, prec="double", **kw):
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField

    st = dict(SMALL_BOX_SETTINGS)
    st.update(kw)
    return PGMForceField(system, H, MDSettings(precision=prec, **st))


def rms_rel(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.sqrt(np.mean((a - b) ** 2)) / np.sqrt(np.mean(b**2)))


@pytest.fixture(scope="module")
def box(small_box_system, golden_small_box):
    s, pos, H = small_box_system
    o = O.Oracle(s, SMALL_BOX_SETTINGS)
    return s, pos, H, o, o.compute(pos, H)


@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_field_of_charges_and_dipoles(box, prec):
    """The field sweep (rows + PME + self term) against the oracle's _field."""
    s, pos, H, o, _ = box
    rng = np.random.default_rng(3)
    d = rng.normal(scale=0.01, size=(s.n, 3))
    ref = o.field(pos, H, s.q, d)
    ff = ff_for(s, H, prec)
    got = ff.field(pos, H, d, charges=True).cpu().numpy()
    tol = 1e-10 if prec == "double" else 2e-6
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max(), np.abs(got - ref).max() / np.abs(ref).max()
    ref0 = o.field(pos, H, None, d)
    got0 = ff.field(pos, H, d, charges=False).cpu().numpy()
    assert np.abs(got0 - ref0).max() <= tol * np.abs(ref0).max()


@pytest.mark.parametrize("grid", [(32, 32, 32), (36, 48, 48), (32, 32, 48), (30, 36, 32)])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_field_through_every_fft_route(box, grid, prec):
    """The field sweep on meshes that take each route of the reciprocal-space chain: the plane
    passes (K2 = K3: 32^3 and 36 x 48^2) and separate k3 and k2 passes (32 x 32 x 48, 30 x 36 x 32),
    against the oracle.  The
    oracle transforms the full spectrum, the engine (as pme.py:370-376) the rfft half: on this
    triclinic box the influence function is not mirror-symmetric on the Nyquist planes, which
    separates the two by up to ~2e-10 of the field on the coarse 30 x 36 x 32 mesh (white-noise
    grids: 7e-12), hence 1e-9 for FP64 here."""
    s, pos, H, _, _ = box
    st = dict(SMALL_BOX_SETTINGS, pme_grid=grid)
    o = O.Oracle(s, st)
    rng = np.random.default_rng(5)
    d = rng.normal(scale=0.01, size=(s.n, 3))
    ref = o.field(pos, H, s.q, d)
    got = ff_for(s, H, prec, pme_grid=grid).field(pos, H, d, charges=True).cpu().numpy()
    tol = 1e-9 if prec == "double" else 2e-6
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max(), np.abs(got - ref).max() / np.abs(ref).max()


def test_compute_double_matches_golden(box, golden_small_box):
    """FP64 engine: ff_small_box energies, forces, dipoles, iterations, virial (reference golden)."""
    s, pos, H, o, r = box
    g = golden_small_box
    ff = ff_for(s, H, "double")
    res = ff.compute(pos, H, None, ff.init_induction())
    assert int(res.status[0]) & ~0x2 == 0
    for k in ("elec", "vdw", "total"):
        ref = float(g[f"double.energy.{k}"])
        assert abs(float(res.energy[k][0]) - ref) <= 1e-9 * abs(ref), (k, float(res.energy[k][0]), ref)
    assert int(res.iterations[0]) == int(g["double.iterations"])
    F = res.forces.cpu().numpy()
    assert np.abs(F - g["double.forces"]).max() <= 1e-8 * np.abs(g["double.forces"]).max()
    mu = res.induction.mu.cpu().numpy()
    assert np.abs(mu - g["double.mu"]).max() <= 1e-9 * np.abs(g["double.mu"]).max()
    W = res.virial[0].cpu().numpy()
    assert np.abs(W - g["double.strain"]).max() <= 1e-7 * np.abs(g["double.strain"]).max()


def test_compute_mixed_within_tolerance(box, golden_small_box):
    """Mixed precision against the float64 golden: 1e-6 energy, 1e-5 RMS forces / dipoles."""
    s, pos, H, o, r = box
    g = golden_small_box
    ff = ff_for(s, H, "mixed")
    res = ff.compute(pos, H, None, ff.init_induction())
    for k in ("elec", "total"):
        ref = float(g[f"double.energy.{k}"])
        assert abs(float(res.energy[k][0]) - ref) <= 1e-6 * abs(ref), (k, float(res.energy[k][0]), ref)
    assert abs(float(res.energy["vdw"][0]) - float(g["double.energy.vdw"])) <= 1e-5 * abs(float(g["double.energy.vdw"]))
    assert rms_rel(res.forces.cpu().numpy(), g["double.forces"]) <= 1e-5
    assert rms_rel(res.induction.mu.cpu().numpy(), g["double.mu"]) <= 1e-5
    assert abs(int(res.iterations[0]) - int(g["mixed.iterations"])) <= 2


@pytest.mark.parametrize("elec", ["q", "qp", "qi", "qpi"])
def test_elec_levels_match_oracle(small_box_system, elec):
    s, pos, H = small_box_system
    st = dict(SMALL_BOX_SETTINGS, elec=elec)
    r = O.Oracle(s, st).compute(pos, H)
    ff = ff_for(s, H, "double", elec=elec)
    res = ff.compute(pos, H)
    assert abs(float(res.energy["total"][0]) - r["energy"]["total"]) <= 1e-9 * abs(r["energy"]["total"])
    assert np.abs(res.forces.cpu().numpy() - r["forces"]).max() <= 1e-8 * np.abs(r["forces"]).max()
    assert int(res.iterations[0]) == r["iterations"]


def test_candidate_rows_equal_cell_list(box):
    """Rows from the caller's candidate list (the reference's idx) equal the engine's cell list."""
    s, pos, H, o, r = box
    ff = ff_for(s, H, "double")
    idx = ff.rows_for(pos, H)
    a = ff.compute(pos, H, None)
    b = ff.compute(pos, H, idx)
    assert abs(float(a.energy["total"][0]) - float(b.energy["total"][0])) <= 1e-11 * abs(float(a.energy["total"][0]))
    assert np.abs(a.forces.cpu().numpy() - b.forces.cpu().numpy()).max() <= 1e-9 * float(a.forces.abs().max())


def test_energy_and_fixed_mu_paths(box):
    """energy() (CG from the state's mu) and energy_fixed_mu() agree with compute()."""
    s, pos, H, o, r = box
    ff = ff_for(s, H, "double")
    res = ff.compute(pos, H)
    E, ind, it, ov = ff.energy(pos, H, None, res.induction)
    assert abs(float(E[0]) - float(res.energy["total"][0])) <= 1e-8 * abs(float(E[0]))
    Ef, parts = ff.energy_fixed_mu(pos, H, res.induction.mu)
    assert abs(float(Ef[0]) - float(res.energy["total"][0])) <= 1e-11 * abs(float(Ef[0]))
    assert np.abs(parts["forces"].cpu().numpy() - res.forces.cpu().numpy()).max() <= 1e-9 * float(res.forces.abs().max())
    ref = o.energy_fixed_mu(pos, H, res.induction.mu.cpu().numpy())
    assert abs(float(Ef[0]) - ref["total"]) <= 1e-10 * abs(ref["total"])


@pytest.mark.parametrize("prec,pred", [("double", "mu4"), ("mixed", "mu4"), ("double", "mu1")])
def test_predictor_steps_match_oracle(small_box_system, prec, pred):
    """Six steps with a predictor (mu4, or mu1: the previous step's dipoles) and the fused start
    (history, count, norm carried)."""
    s, pos, H = small_box_system
    st = dict(SMALL_BOX_SETTINGS, dipole_tol=1e-8, norm_refresh=5, predictor=pred)
    o = O.Oracle(s, st)
    ff = ff_for(s, H, prec, dipole_tol=1e-8, norm_refresh=5, predictor=pred)
    ind_o = o.init_induction()
    ind_g = ff.init_induction()
    rng = np.random.default_rng(1)
    x = pos.copy()
    for step in range(6):
        x = x + rng.normal(scale=2e-4, size=x.shape)
        ro = o.compute(x, H, ind_o)
        ind_o = ro["induction"]
        rg = ff.compute(x, H, None, ind_g)
        ind_g = rg.induction
        e_ref = ro["energy"]["total"]
        tol_e = 1e-10 if prec == "double" else 1e-6
        assert abs(float(rg.energy["total"][0]) - e_ref) <= tol_e * abs(e_ref), (step, float(rg.energy["total"][0]), e_ref)
        if prec == "double":
            assert int(rg.iterations[0]) == ro["iterations"], (step, int(rg.iterations[0]), ro["iterations"])
        else:
            assert abs(int(rg.iterations[0]) - ro["iterations"]) <= 1
        assert rms_rel(rg.forces.cpu().numpy(), ro["forces"]) <= (1e-9 if prec == "double" else 1e-5)
    assert int(ind_g.count[0]) == 6 == ind_o["count"]


def test_batch_equals_separate_systems(small_box_system):
    """A batch of uneven systems (two boxes, different sizes and grids) equals separate evaluations."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import small_box

    s0, p0, H0 = small_box_system
    s1, p1, H1 = small_box(5, nw=40, nm=2)
    st = MDSettings(precision="double", **dict(SMALL_BOX_SETTINGS, dipole_tol=1e-8))
    grids = [(32, 32, 32), (36, 30, 32)]
    fb = PGMForceField([s0, s1], [H0, H1], st, pme_grids=grids)
    rb = fb.compute(np.concatenate([p0, p1]), np.stack([H0, H1]))
    for k, (s, p, H, g) in enumerate([(s0, p0, H0, grids[0]), (s1, p1, H1, grids[1])]):
        f = PGMForceField(s, H, st, pme_grids=[g])
        r = f.compute(p, H)
        assert abs(float(rb.energy["total"][k]) - float(r.energy["total"][0])) <= 1e-10 * abs(float(r.energy["total"][0]))
        assert int(rb.iterations[k]) == int(r.iterations[0])
        sl = slice(int(fb.offsets[k]), int(fb.offsets[k + 1]))
        assert np.abs(rb.forces[sl].cpu().numpy() - r.forces.cpu().numpy()).max() <= 1e-9 * float(r.forces.abs().max())


def test_water512_fp64_matches_oracle():
    """512 pGM3P-25 waters (24.83 A box, 9 A cutoff, PME 48^3 order 6, beta 0.4/A, tol 1e-8), FP64."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(8, 2.483, seed=0)
    st = dict(cutoff=0.9, ewald_beta=4.0, pme_grid=(48, 48, 48), pme_order=6, dipole_tol=1e-8, max_iter=100)
    r = O.Oracle(s, st).compute(pos, H)
    ff = PGMForceField(s, H, MDSettings(precision="double", **st))
    g = ff.compute(pos, H)
    assert abs(float(g.energy["total"][0]) - r["energy"]["total"]) <= 1e-9 * abs(r["energy"]["total"])
    assert rms_rel(g.forces.cpu().numpy(), r["forces"]) <= 1e-9
    assert int(g.iterations[0]) == r["iterations"]
    assert np.abs(g.virial[0].cpu().numpy() - r["virial"]).max() <= 1e-7 * np.abs(r["virial"]).max()
    ffm = PGMForceField(s, H, MDSettings(precision="mixed", **st))
    m = ffm.compute(pos, H)
    assert abs(float(m.energy["total"][0]) - r["energy"]["total"]) <= 1e-6 * abs(r["energy"]["total"])
    assert rms_rel(m.forces.cpu().numpy(), r["forces"]) <= 1e-5
    assert rms_rel(m.induction.mu.cpu().numpy(), r["mu"]) <= 1e-5


def test_row_overflow_is_reported_and_recovers():
    """A capacity below the largest row sets the overflow bit; growing it repeats the step correctly.

    (The driver's resize-and-repeat of the reference, driver.py:117-151, forcefield.py:1286.)
    """
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(8, 2.483, seed=0)
    st = dict(cutoff=0.9, ewald_beta=4.0, pme_grid=(48, 48, 48), pme_order=6, dipole_tol=1e-8, max_iter=100)
    ff = PGMForceField(s, H, MDSettings(precision="double", **st))
    ref = ff.compute(pos, H)
    assert not bool(ref.overflow[0])
    big = ff.capacity
    ff.set_capacity(64)
    res = ff.compute(pos, H)
    assert bool(res.overflow[0]) and ff.capacity == 64
    ff.grow_rows(big)
    res = ff.compute(pos, H)
    assert not bool(res.overflow[0])
    assert abs(float(res.energy["total"][0]) - float(ref.energy["total"][0])) <= 1e-10 * abs(float(ref.energy["total"][0]))


def test_cg_max_iter_status(box):
    s, pos, H, o, r = box
    ff = ff_for(s, H, "double", max_iter=3)
    res = ff.compute(pos, H)
    assert int(res.iterations[0]) == 3 and int(res.status[0]) & 0x2


@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_split_rows_match_oracle(small_box_system, prec):
    """elec_cutoff 0.45 < cutoff 0.6 (split rows): the field sweeps stream only the electrostatic
    part of every row, the LJ term keeps every pair; energies, forces, dipoles and iterations as the
    oracle's split rows, and an overflow of either part is reported and recovered by grow_rows."""
    s, pos, H = small_box_system
    st = dict(SMALL_BOX_SETTINGS, dipole_tol=1e-8, elec_cutoff=0.45)
    ro = O.Oracle(s, st).compute(pos, H)
    ff = ff_for(s, H, prec, dipole_tol=1e-8, elec_cutoff=0.45)
    rg = ff.compute(pos, H)
    assert int(rg.status[0]) == 0
    e = float(rg.energy["total"][0])
    assert abs(e - ro["energy"]["total"]) <= (1e-10 if prec == "double" else 1e-6) * abs(ro["energy"]["total"])
    assert rms_rel(rg.forces.cpu().numpy(), ro["forces"]) <= (1e-9 if prec == "double" else 1e-5)
    assert rms_rel(rg.induction.mu.cpu().numpy(), ro["mu"]) <= (1e-9 if prec == "double" else 1e-5)
    if prec == "double":
        assert int(rg.iterations[0]) == ro["iterations"]
        full = ff_for(s, H, prec, dipole_tol=1e-8)
        full.compute(pos, H)
        assert int(full._lib.pgm_row_pairs(full._h)) > int(ff._lib.pgm_row_pairs(ff._h))  # fewer pairs streamed
        # overflow of the LJ part, then recovery
        small = ff_for(s, H, prec, dipole_tol=1e-8, elec_cutoff=0.45)
        small.set_capacity(small.elec_capacity + 32)
        e_cap = small.elec_capacity
        small.set_elec_capacity(32)
        r1 = small.compute(pos, H)
        if int(small._lib.pgm_max_row_count(small._h)) > 32:
            assert int(r1.status[0]) & 0x1
        small.grow_rows(small.capacity)
        r2 = small.compute(pos, H)
        assert int(r2.status[0]) == 0 and small.elec_capacity >= 32 and e_cap > 0
        assert abs(float(r2.energy["total"][0]) - ro["energy"]["total"]) <= 1e-10 * abs(ro["energy"]["total"])


def test_compute_host_with_the_state_on_the_device():
    """pgm_compute_host with ind = NULL (the induction state kept in the handle, only positions in
    and outputs out) gives, step after step, what the same call with the state in host buffers
    gives, and switching between the two continues from the handle's state."""
    import ctypes as C

    from pgm_jax_b200 import _lib
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(4, 1.25, seed=11)
    kw = dict(cutoff=0.6, ewald_beta=5.0, pme_grid=(32, 32, 32), dipole_tol=1e-7, max_iter=100)
    fa = ff_for(s, H, "mixed", **kw)  # state on the device
    fb = ff_for(s, H, "mixed", **kw)  # state in host buffers
    n = s.n
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731

    def outputs():
        arrs = [np.zeros((1, 3)), np.zeros((n, 3)), np.zeros((1, 3, 3)), np.zeros(1, np.int32), np.zeros(1),
                np.zeros(1, np.int32)]
        return arrs, _lib.PgmOutputs(*[p(a).value for a in arrs])

    arrs_a, outa = outputs()  # the arrays stay referenced: the library writes into them
    arrs_b, outb = outputs()
    Ea, Fa, _va, ita, _ra, sta = arrs_a
    Eb, Fb, _vb, itb, _rb, stb = arrs_b
    mu, hist = np.zeros((n, 3)), np.zeros((4, n, 3))
    cnt, norm = np.zeros(1, np.int32), np.ones(1)
    ind = _lib.PgmInduction(p(mu).value, p(hist).value, p(cnt).value, p(norm).value)
    rng = np.random.default_rng(5)
    x = pos.copy()
    hb = np.ascontiguousarray(H[None])
    for step in range(6):
        x = x + rng.normal(scale=2e-4, size=x.shape)
        xc = np.ascontiguousarray(x)
        # at step 3 the device-state handle is given the host state from before this step (the
        # values it holds itself): it loads it and carries on from it
        ia = None
        if step == 3:
            mu_b, hist_b, cnt_b, norm_b = mu.copy(), hist.copy(), cnt.copy(), norm.copy()
            ind_prev = _lib.PgmInduction(p(mu_b).value, p(hist_b).value, p(cnt_b).value, p(norm_b).value)
            ia = C.byref(ind_prev)
        _lib.check(fb._lib.pgm_compute_host(fb._h, p(xc), p(hb), C.byref(ind), C.byref(outb)))
        _lib.check(fa._lib.pgm_compute_host(fa._h, p(xc), p(hb), ia, C.byref(outa)))
        assert sta[0] == 0 and stb[0] == 0
        # mixed precision: the two handles differ only by the order of FP32 atomic additions
        assert abs(Ea[0, 2] - Eb[0, 2]) <= 1e-7 * abs(Eb[0, 2]), step
        assert np.abs(Fa - Fb).max() <= 1e-5 * np.abs(Fb).max(), step
        assert abs(int(ita[0]) - int(itb[0])) <= 1, step


def test_compute_host_matches_device_calls():
    """pgm_compute_host (host buffers; from the second call a replayed captured graph) gives the
    device path's energies, forces and dipole history over consecutive steps, also after the row
    capacity changed (the captured graph is rebuilt)."""
    import ctypes as C

    from pgm_jax_b200 import _lib
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(4, 1.25, seed=9)
    kw = dict(cutoff=0.6, ewald_beta=5.0, pme_grid=(32, 32, 32), dipole_tol=1e-7, max_iter=100)
    fd = ff_for(s, H, "mixed", **kw)
    fh = ff_for(s, H, "mixed", **kw)
    ind_d = fd.init_induction()
    n = s.n
    mu, hist = np.zeros((n, 3)), np.zeros((4, n, 3))
    cnt, norm = np.zeros(1, np.int32), np.ones(1)
    E, F, V = np.zeros((1, 3)), np.zeros((n, 3)), np.zeros((1, 3, 3))
    it, res, stt = np.zeros(1, np.int32), np.zeros(1), np.zeros(1, np.int32)
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    ind = _lib.PgmInduction(p(mu).value, p(hist).value, p(cnt).value, p(norm).value)
    out = _lib.PgmOutputs(p(E).value, p(F).value, p(V).value, p(it).value, p(res).value, p(stt).value)
    rng = np.random.default_rng(3)
    x = pos.copy()
    hb = np.ascontiguousarray(H[None])
    for step in range(7):
        if step == 4:
            fh.set_capacity(fh.capacity + 32)
            fd.set_capacity(fd.capacity + 32)
        x = x + rng.normal(scale=2e-4, size=x.shape)
        xc = np.ascontiguousarray(x)
        _lib.check(fh._lib.pgm_compute_host(fh._h, p(xc), p(hb), C.byref(ind), C.byref(out)))
        rd = fd.compute(x, H, None, ind_d)
        ind_d = rd.induction
        assert stt[0] == 0
        # mixed precision: the two handles differ only by the order of FP32 atomic additions
        assert abs(E[0, 2] - float(rd.energy["total"][0])) <= 1e-7 * abs(E[0, 2]), step
        assert np.abs(F - rd.forces.cpu().numpy()).max() <= 1e-5 * np.abs(F).max(), step
        assert np.abs(hist - ind_d.hist.cpu().numpy()).max() <= 1e-5 * np.abs(hist).max(), step
        assert abs(int(it[0]) - int(rd.iterations[0])) <= 1 and int(cnt[0]) == int(ind_d.count[0]) == step + 1


@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_pgm3p25_512_matches_reference_golden(pgm3p25_512_system, golden_pgm3p25_512, prec):
    """The reference's ff_pgm3p25_512 regression point (examples/water512 frame, truncated
    octahedron, default settings, 30^3 mesh): FP64 against its float64 record (energy 1e-9, forces
    1e-8 RMS, iterations equal, virial 1e-6); mixed precision against its mixed record (energy
    1e-6) and its float64 record (forces and dipoles 1e-5 RMS relative; 2e-5 against its mixed one)."""
    from conftest import PGM3P25_512_SETTINGS

    from pgm_jax_b200.forcefield import MDSettings, PGMForceField

    g = golden_pgm3p25_512
    ff = PGMForceField(pgm3p25_512_system, g["box"], MDSettings(precision=prec, **PGM3P25_512_SETTINGS))
    res = ff.compute(g["pos"], g["box"], None, ff.init_induction())
    assert int(res.status[0]) == 0
    # mixed: the FP32 LJ pair sum carries ~1e-6 of the van der Waals term (the reference's own mixed
    # record is 5e-7 from its float64 one), so that component is held to 1e-5 as on the small box
    tol_e = {"elec": 1e-9, "vdw": 1e-9, "total": 1e-9} if prec == "double" else {"elec": 1e-6, "vdw": 1e-5, "total": 1e-6}
    for k in ("elec", "vdw", "total"):
        ref = float(g[f"{prec}.energy.{k}"])
        assert abs(float(res.energy[k][0]) - ref) <= tol_e[k] * abs(ref), (k, float(res.energy[k][0]), ref)
    tol = 1e-8 if prec == "double" else 1e-5
    # FP32 kernels against the float64 record; against the reference's own mixed record (its FP32
    # path's rounding added to ours) at twice that
    assert rms_rel(res.forces.cpu().numpy(), g["double.forces"]) <= tol
    assert rms_rel(res.induction.mu.cpu().numpy(), g["double.mu"]) <= tol
    if prec == "mixed":
        assert rms_rel(res.forces.cpu().numpy(), g["mixed.forces"]) <= 2 * tol
        assert rms_rel(res.induction.mu.cpu().numpy(), g["mixed.mu"]) <= 2 * tol
    if prec == "double":
        assert int(res.iterations[0]) == int(g["double.iterations"])
        W = g["double.strain"]
        assert np.abs(res.virial[0].cpu().numpy() - W).max() <= 1e-6 * np.abs(W).max()
    else:
        assert abs(int(res.iterations[0]) - int(g["mixed.iterations"])) <= 1


@pytest.mark.parametrize("grid", [(64, 64, 64), (72, 72, 72), (96, 96, 96), (192, 192, 192), (64, 96, 72)])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_field_on_the_workload_meshes(grid, prec):
    """The field sweep on the mesh lengths of the benchmark workloads: 64^3 and 72^3 (the uneven
    boxes and the path-integral beads), 96^3 (4,096 waters) and 192^3 (32,768 waters: K > 128 takes
    the five-pass chain), and a mixed 64 x 96 x 72 mesh (the separate passes, each axis's compiled
    plan), against the oracle's full-spectrum FFT on 512 pGM3P-25 waters."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(8, 2.483, seed=2)
    st = dict(cutoff=0.9, ewald_beta=4.0, pme_grid=grid, pme_order=6, dipole_tol=1e-8, max_iter=100)
    rng = np.random.default_rng(7)
    d = rng.normal(scale=0.01, size=(s.n, 3))
    ref = O.Oracle(s, st).field(pos, H, s.q, d)
    got = PGMForceField(s, H, MDSettings(precision=prec, **st)).field(pos, H, d, charges=True).cpu().numpy()
    tol = 1e-9 if prec == "double" else 2e-6
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max(), np.abs(got - ref).max() / np.abs(ref).max()


@pytest.mark.parametrize("edges", [(1.25, 1.25, 1.25), (1.4, 2.1, 3.3), (2.9, 2.5, 1.9), (4.4, 1.3, 2.2)])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_candidate_list_of_rectangular_boxes_is_complete(edges, prec):
    """The engine's candidate list against candidate rows of all other atoms given by the caller (the cutoff is tested in
    the engine either way: a third of the atoms sit on cell faces, many pairs at the cutoff to rounding), on
    rectangular boxes with few and many cells per axis, positions outside the box: the same pairs (exact
    counts), the same forces."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import Molecule, System

    rng = np.random.default_rng(23)
    n, cutoff, L = 420, 0.6, np.array(edges)
    pos = rng.uniform(0, 1, size=(n, 3)) * L
    cells = np.floor(L / (0.5 * cutoff))
    pos[: n // 3] = np.round(pos[: n // 3] / L * cells) / cells * L
    pos += rng.normal(scale=1e-9, size=pos.shape)
    s = System([Molecule("X", ["O"], [q], [0.05], [1e-3]) for q in rng.normal(size=n)])
    ff = PGMForceField(s, np.diag(L), MDSettings(precision=prec, elec="q", cutoff=cutoff, ewald_beta=6.0, pme_grid=(24, 24, 24)),
                       row_capacity=416)
    ff.set_list_capacity(512)
    others = (np.arange(n)[:, None] + np.arange(1, n)) % n
    given = ff.compute(pos, np.diag(L), others.astype(np.int32))
    pairs = int(ff._lib.pgm_row_pairs(ff._h))
    for shift in (0, 1):  # the second call rebuilds the list at positions a lattice vector away
        own = ff.compute(pos + shift * L, np.diag(L))
        assert int(ff._lib.pgm_row_pairs(ff._h)) == pairs
        assert not bool(own.overflow.any())
        assert rms_rel(own.forces.cpu().numpy(), given.forces.cpu().numpy()) <= (1e-10 if prec == "double" else 1e-5)


@pytest.mark.parametrize("edge", [4.0, 60.0, 1000.0])
@pytest.mark.parametrize("skew", [0.0, 0.3])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_candidate_list_of_large_boxes_is_complete(edge, skew, prec):
    """Pairs a hair closer than cutoff + skin when the list is built, then moved together by a hair less than the
    skin, so that the list must still hold every one: the same pairs as from the caller's rows of all other
    atoms (the cutoff is tested in the engine either way), in boxes whose FP32 coordinates are good to 2e-7 to
    6e-5 nm."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import Molecule, System

    rng = np.random.default_rng(31)
    n, cutoff, skin = 400, 0.6, 0.1
    H = np.diag([edge] * 3) + edge * np.array([[0, 0, 0], [skew, 0, 0], [-skew, skew, 0]])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    a = rng.uniform(0, 1, size=(n, 3)) @ H
    b = a + u * (cutoff + skin - rng.uniform(0, 2e-8 * edge, size=(n, 1)))
    move = 0.5 * skin * (1 - 1e-9) * u
    start, end = np.concatenate([a, b]), np.concatenate([a + move, b - move])
    s = System([Molecule("X", ["O"], [q], [0.05], [1e-3]) for q in rng.normal(size=2 * n)])
    st = MDSettings(precision=prec, elec="q", cutoff=cutoff, skin=skin, ewald_beta=6.0, pme_grid=(24, 24, 24))
    own, given = (PGMForceField(s, H, st, row_capacity=128) for _ in range(2))
    own.set_list_capacity(256)
    own.compute(start, H)
    built = own.list_rebuilds()
    own.compute(end, H)
    assert own.list_rebuilds() == built
    others = (np.arange(2 * n)[:, None] + np.arange(1, 2 * n)) % (2 * n)
    given.compute(end, H, others.astype(np.int32))
    assert int(own._lib.pgm_row_pairs(own._h)) == int(given._lib.pgm_row_pairs(given._h))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("skew", [0.0, 0.3])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_non_finite_position_is_a_status_not_a_fault(prec, skew, value):
    """A coordinate that is not a number ends the call with the status bit, in rectangular and triclinic boxes with
    several cells per axis; the next call with finite positions gives what a new handle gives."""
    from pgm_jax_b200 import _lib
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(6, 1.8624, seed=2)
    H = H + np.array([[0, 0, 0], [skew, 0, 0], [0, skew, 0]])
    kw = dict(cutoff=0.5, pme_grid=(24, 24, 24), dipole_tol=1e-8 if prec == "double" else 1e-6)
    ff = ff_for(s, H, prec, **kw)
    for atom, axis in ((0, 2), (s.n - 1, 0), (s.n // 2, 1)):
        x = pos.copy()
        x[atom, axis] = value
        assert int(ff.compute(x, H).status[0]) & _lib.STATUS_NONFINITE
    got, ref = ff.compute(pos, H), ff_for(s, H, prec, **kw).compute(pos, H)
    assert not int(got.status[0]) & _lib.STATUS_NONFINITE
    assert rms_rel(got.forces.cpu().numpy(), ref.forces.cpu().numpy()) <= (1e-10 if prec == "double" else 2e-6)


@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_degenerate_box_is_a_status_not_a_fault(prec):
    """Boxes without volume, with a negative edge or with entries that are not finite end the call with a
    status bit (box or non-finite energy); the next call with a good box gives what a new handle gives."""
    from pgm_jax_b200 import _lib
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(6, 1.8624, seed=2)
    kw = dict(cutoff=0.5, pme_grid=(24, 24, 24), dipole_tol=1e-8 if prec == "double" else 1e-6, max_iter=40)
    ff = ff_for(s, H, prec, **kw)
    bad = [np.zeros((3, 3)), -H, np.diag([1.8624, 1.8624, 0.0]), np.diag([1.8624, -1.8624, 1.8624]), np.full((3, 3), np.nan)]
    bad += [np.diag([1.8624, 1.8624, v]) for v in (np.nan, np.inf)]
    bad.append(H + np.array([[0, 0, 0], [0.3, 0, 0], [0, np.nan, 0]]))
    for box in bad:
        assert int(ff.compute(pos, box).status[0]) & (_lib.STATUS_BAD_BOX | _lib.STATUS_NONFINITE), box
    got, ref = ff.compute(pos, H), ff_for(s, H, prec, **kw).compute(pos, H)
    assert not int(got.status[0]) & (_lib.STATUS_BAD_BOX | _lib.STATUS_NONFINITE)
    assert rms_rel(got.forces.cpu().numpy(), ref.forces.cpu().numpy()) <= (1e-10 if prec == "double" else 2e-6)


@pytest.mark.parametrize("prec,beta", [("double", b) for b in (1.0, 4.0, 8.0, 14.0)] + [("mixed", b) for b in (1.0, 4.0, 8.0)])
def test_pair_kernels_over_their_ranges(prec, beta):
    """The field of charges and dipoles of single atoms at all distances from 0.02 nm (both arguments of the
    pair kernels small) to the cutoff (the Gaussians screened out), with widths on both sides of beta,
    against the oracle.  Tolerances as for the field of the small box.  At beta 14 / nm the field is a small
    difference of the row, mesh and self parts (137, 155 and 52 of 80 e/nm^2), whose FP32 mesh part alone is
    above the mixed tolerance: FP64 only."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import Molecule, System

    rng = np.random.default_rng(17)
    n, edge = 80, 1.3
    mols = [Molecule("X", ["O"], [q], [r], [1e-3]) for q, r in zip(rng.normal(size=n), rng.uniform(0.03, 0.12, size=n))]
    s, H = System(mols), np.eye(3) * edge
    pos = rng.uniform(0, edge, size=(n, 3))
    u = rng.normal(size=(n // 2, 3))  # every second atom beside its neighbour, 0.02 .. 0.3 nm away
    pos[1::2] = pos[::2] + u / np.linalg.norm(u, axis=1)[:, None] * np.linspace(0.02, 0.3, n // 2)[:, None]
    d = rng.normal(scale=0.01, size=(n, 3))
    st = dict(cutoff=0.6, ewald_beta=beta, pme_grid=(24, 24, 24), pme_order=6)
    ref = O.Oracle(s, st).field(pos, H, s.q, d)
    got = PGMForceField(s, H, MDSettings(precision=prec, **st)).field(pos, H, d, charges=True).cpu().numpy()
    tol = 1e-10 if prec == "double" else 2e-6
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max(), np.abs(got - ref).max() / np.abs(ref).max()


@pytest.mark.parametrize("size", [1, 8, 9, 10, 33, 70])
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_molecules_of_many_sizes(prec, size):
    """One rigid molecule of `size` atoms (no partners, up to the partners that two threads share, one above, more
    than a chunk of 32 and than two) among waters, in a box where some of its atoms are beyond the cutoff of
    others: energy, forces and virial of charges and permanent dipoles against the oracle.  Tolerances as for the small
    box."""
    from pgm_jax_b200.systems import Molecule, System, pgm3p25_water, water_box

    s, pos, H = water_box(5, 1.552, seed=8)
    rng = np.random.default_rng(size)
    q = rng.normal(scale=0.3, size=size)
    big = Molecule("B", ["C"] * size, q, rng.uniform(0.05, 0.07, size), np.full(size, 1e-3), [], np.full(size, 0.15), np.full(size, 0.4))
    first = 3 * -(-size // 3)  # the molecule takes the places of the first waters' atoms
    sy = System([big] + [pgm3p25_water()] * ((s.n - first) // 3))
    x = np.concatenate([pos[:size], pos[first:]])
    kw = dict(cutoff=0.5, pme_grid=(30, 30, 30), elec="qp")
    r = O.Oracle(sy, dict(SMALL_BOX_SETTINGS, **kw)).compute(x, H)
    g = ff_for(sy, H, prec, **kw).compute(x, H)
    e, f, w = (1e-9, 1e-8, 1e-7) if prec == "double" else (1e-6, 1e-5, 1e-4)
    assert abs(float(g.energy["elec"][0]) - r["energy"]["elec"]) <= e * abs(r["energy"]["elec"])
    assert rms_rel(g.forces.cpu().numpy(), r["forces"]) <= f
    assert np.abs(g.virial[0].cpu().numpy() - r["virial"]).max() <= w * np.abs(r["virial"]).max()


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_mixed_energy_is_as_good_as_its_charges(seed):
    """The mixed engine's energy of 512 waters at given dipoles (none, and the solved ones) against the FP64 engine's.
    Rounding the parameters to FP32 (the self energy keeps the FP64 charges) moves the oracle's energy by 2.6e-8;
    the sums' own error has to stay below half of that again: 4e-8 in all.  A bias of the pair kernels or of
    the charge products, the same for all pairs of a kind, is 2e-8 and above."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(8, 2.4832, seed=seed)
    d, m = (PGMForceField(s, H, MDSettings(precision=p, pme_grid=(48, 48, 48), dipole_tol=1e-8)) for p in ("double", "mixed"))
    mu = d.compute(pos, H).induction.mu
    for given in (torch.zeros_like(mu), mu):
        ref = float(d.energy_fixed_mu(pos, H, given)[0][0])
        assert abs(float(m.energy_fixed_mu(pos, H, given)[0][0]) - ref) <= 4e-8 * abs(ref)


MESH_LENGTHS = [K for K in range(8, 257, 2) if 2**8 * 3**5 * 5**3 % K == 0]


@pytest.mark.parametrize("L", MESH_LENGTHS)
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_field_on_every_mesh_length(L, prec):
    """Every mesh length the engine takes, along each axis in turn (the last tiles of lines and columns
    are ragged) and as a plane (K2 = K3), on 64 waters in a cubic box with order 4, against the oracle.
    Tolerances as on the workload meshes."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(4, 1.2416, seed=3)
    d = np.random.default_rng(11).normal(scale=0.01, size=(s.n, 3))
    tol = 1e-9 if prec == "double" else 2e-6
    for grid in [(L, 8, 10), (10, L, 8), (8, 10, L), (8, L, L)]:
        st = dict(cutoff=0.6, ewald_beta=6.0, pme_grid=grid, pme_order=4)
        ref = O.Oracle(s, st).field(pos, H, s.q, d)
        got = PGMForceField(s, H, MDSettings(precision=prec, **st)).field(pos, H, d, charges=True).cpu().numpy()
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max(), (grid, np.abs(got - ref).max() / np.abs(ref).max())


@pytest.mark.parametrize("L", MESH_LENGTHS)
@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_energy_and_virial_on_every_mesh_length(L, prec):
    """The energy form of the k1 pass (its block reductions, the weights of the half spectrum and the influence
    part of the virial) for every mesh length along k1 and along k3, on charges and permanent dipoles,
    against the oracle.  Tolerances as for the molecules of many sizes.  On the k1 Nyquist plane m1 has one sign in
    the engine's half spectrum (as in the reference's rfft), while its products with m2 and m3 cancel in the oracle's
    full one: the xy and xz elements are compared where that plane's exp(-(pi m1 / beta L)^2) is
    below 2e-8 (lengths from 20)."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(4, 1.2416, seed=3)
    e, f, w = (1e-9, 1e-8, 1e-7) if prec == "double" else (1e-6, 1e-5, 1e-4)
    for grid in [(L, 24, 20), (20, 24, L)]:
        st = dict(cutoff=0.6, ewald_beta=6.0, pme_grid=grid, pme_order=4, elec="qp")
        r = O.Oracle(s, st).compute(pos, H)
        g = PGMForceField(s, H, MDSettings(precision=prec, **st)).compute(pos, H)
        assert abs(float(g.energy["elec"][0]) - r["energy"]["elec"]) <= e * abs(r["energy"]["elec"]), grid
        assert rms_rel(g.forces.cpu().numpy(), r["forces"]) <= f, grid
        dW = np.abs(g.virial[0].cpu().numpy() - r["virial"])
        if grid[0] < 20:
            dW[0, 1:] = dW[1:, 0] = 0.0
        assert dW.max() <= w * np.abs(r["virial"]).max(), grid


def test_water4096_frame_matches_oracle():
    """The 4,096-water benchmark frame (12,288 atoms, 4.966 nm box, PME 96^3, cutoff 0.9 nm,
    Ewald 4.0/nm) as a single point at tol 1e-8: the FP64 engine against the oracle (energy 1e-9,
    forces 1e-8 RMS, iterations equal, virial 1e-7); mixed precision at tol 1e-6 against the same
    oracle point (energy 1e-6, forces and dipoles 1e-5 RMS)."""
    from pgm_jax_b200.forcefield import MDSettings, PGMForceField
    from pgm_jax_b200.systems import water_box

    s, pos, H = water_box(16, 4.966, seed=0)
    st = dict(cutoff=0.9, ewald_beta=4.0, pme_grid=(96, 96, 96), pme_order=6, dipole_tol=1e-8, max_iter=100)
    r = O.Oracle(s, st).compute(pos, H)
    g = PGMForceField(s, H, MDSettings(precision="double", **st)).compute(pos, H)
    assert int(g.status[0]) == 0
    assert abs(float(g.energy["total"][0]) - r["energy"]["total"]) <= 1e-9 * abs(r["energy"]["total"])
    assert rms_rel(g.forces.cpu().numpy(), r["forces"]) <= 1e-8
    assert rms_rel(g.induction.mu.cpu().numpy(), r["mu"]) <= 1e-8
    assert int(g.iterations[0]) == r["iterations"]
    assert np.abs(g.virial[0].cpu().numpy() - r["virial"]).max() <= 1e-7 * np.abs(r["virial"]).max()
    m = PGMForceField(s, H, MDSettings(precision="mixed", **dict(st, dipole_tol=1e-6))).compute(pos, H)
    assert abs(float(m.energy["total"][0]) - r["energy"]["total"]) <= 1e-6 * abs(r["energy"]["total"])
    assert rms_rel(m.forces.cpu().numpy(), r["forces"]) <= 1e-5
    assert rms_rel(m.induction.mu.cpu().numpy(), r["mu"]) <= 1e-5


@pytest.mark.parametrize("prec,niter", [("double", 1), ("double", 2), ("mixed", 1), ("double", 3)])
def test_local_preconditioner_steps_match_oracle(pgm3p25_512_system, golden_pgm3p25_512, prec, niter):
    """The local preconditioner (local_niter inner CG iterations on the row entries closer than
    local_cut = 0.3 nm, forcefield.py:1766-1811) over five mu4 steps of the pGM3P-25 512-water frame
    with small displacements: FP64 energy, forces and dipoles as the oracle's, and the same outer
    iterations; fewer outer iterations than Jacobi; mixed precision within its tolerance."""
    from conftest import PGM3P25_512_SETTINGS

    from pgm_jax_b200.forcefield import MDSettings, PGMForceField

    s, g = pgm3p25_512_system, golden_pgm3p25_512
    tol = 1e-8 if prec == "double" else 1e-6
    st = dict(PGM3P25_512_SETTINGS, dipole_tol=tol, max_iter=100, local_cut=0.3, local_niter=niter)
    o = O.Oracle(s, st)
    oj = O.Oracle(s, dict(st, local_niter=0))
    ff = PGMForceField(s, g["box"], MDSettings(precision=prec, **st))
    ind_o, ind_j, ind_g = o.init_induction(), oj.init_induction(), ff.init_induction()
    rng = np.random.default_rng(5)
    x = g["pos"].copy()
    its, its_j = [], []
    for step in range(5):
        x = x + rng.normal(scale=2e-4, size=x.shape)
        ro = o.compute(x, g["box"], ind_o)
        ind_o = ro["induction"]
        rj = oj.compute(x, g["box"], ind_j)
        ind_j = rj["induction"]
        rg = ff.compute(x, g["box"], None, ind_g)
        ind_g = rg.induction
        assert int(rg.status[0]) == 0
        e_ref = ro["energy"]["total"]
        assert abs(float(rg.energy["total"][0]) - e_ref) <= (1e-10 if prec == "double" else 1e-6) * abs(e_ref)
        assert rms_rel(rg.forces.cpu().numpy(), ro["forces"]) <= (1e-8 if prec == "double" else 1e-5)
        assert rms_rel(rg.induction.mu.cpu().numpy(), ro["mu"]) <= (1e-8 if prec == "double" else 1e-5)
        if prec == "double":
            assert int(rg.iterations[0]) == ro["iterations"], (step, int(rg.iterations[0]), ro["iterations"])
        else:
            assert abs(int(rg.iterations[0]) - ro["iterations"]) <= 1
        its.append(ro["iterations"])
        its_j.append(rj["iterations"])
    assert sum(its) < sum(its_j), (its, its_j)


@pytest.mark.parametrize("prec", ["double", "mixed"])
def test_pmemd_pgm_single_point(pgm3p25_512_system, golden_pgm3p25_512, golden_pmemd_pbc_512, prec):
    """The engine against the independent pmemd-pgm single point (PME 72^3 order 8, 10 A cutoff, no
    LJ tail) on the water512 frame: FP64 as tight as the oracle (EELEC 1e-9, forces at pmemd's FP32
    storage, dipoles 1e-9 e A RMS); mixed precision at its tolerance."""
    from conftest import PMEMD_PBC_SETTINGS, pmemd_compare

    from pgm_jax_b200.forcefield import MDSettings, PGMForceField

    s, g = pgm3p25_512_system, golden_pgm3p25_512
    st = dict(PMEMD_PBC_SETTINGS, dipole_tol=1e-10 if prec == "double" else 1e-6)
    r = PGMForceField(s, g["box"], MDSettings(precision=prec, **st)).compute(g["pos"], g["box"])
    re_ = PGMForceField(s, g["box"], MDSettings(precision=prec, **dict(st, vdw="none"))).compute(g["pos"], g["box"])
    assert int(r.status[0]) == 0
    de, dv, df, dmu = pmemd_compare(float(r.energy["elec"][0]), float(r.energy["vdw"][0]), re_.forces.cpu().numpy(),
                                    r.forces.cpu().numpy(), r.induction.mu.cpu().numpy(), golden_pmemd_pbc_512)
    if prec == "double":
        assert de <= 1e-9 and dv <= 1e-4 and df <= 2e-6 and dmu <= 1e-9, (de, dv, df, dmu)
    else:
        assert de <= 1e-6 and dv <= 1e-3 and df <= 36.0 * 1e-5 and dmu <= 0.12 * 1e-5, (de, dv, df, dmu)

