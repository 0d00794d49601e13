"""GPU tests of the specialised stage kernels against the general ones they
stand in for, over the forms they accept.

A deck and the same deck on the general path give the same physics: two
materials with the same constants keep the TDGL and column kernels from the
single-material form, an identity frame rotation (if_OrientRotate with Tg2c = 1) keeps the elastic
stage on k_elastic_tile, and a Drude pole in a material that no cell has keeps
the Yee update on k_em_fused.  The convolution is compared with the numpy
restatement (oracle/restate_fm.py).

Tolerances: the paths order the same sums differently, so fields differ by a
few rounding errors of their terms.  After three steps an FP64 field carries
of order 1e-15 x the cancellation in a stress or curl difference (up to ~1e2
for the random fields here): 1e-12.  FP32: 1e-7 x the same: 2e-5.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 2e-5}
FIELDS = ("m", "m_afm1", "p", "q", "u", "v", "force_store", "Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _run(gf, d, precision, steps=3):
    out = {}
    with gf.Engine.from_params(d, device=0, precision=precision) as e:
        e.advance(steps)
        for f in FIELDS:
            try:
                out[f] = e.download(f)
            except gf.GFError:
                pass
        e.check_finite()
    return out


def _same(a, b, tol):
    assert a.keys() == b.keys()
    for f in a:
        n = np.linalg.norm(b[f])
        d = np.linalg.norm(a[f] - b[f])
        assert np.isfinite(d) and d <= tol * n, (f, d / n if n else d)


def _unit(rng, shape):
    v = rng.standard_normal((3,) + shape)
    return v / np.linalg.norm(v, axis=0)


def _moving(d, seed):
    """Random displacement, velocity and order parameters of the deck's cells."""
    rng = np.random.default_rng(seed)
    sh = (d.nx, d.ny, d.nz)
    mc = d.material_cell()
    solid = mc != 0
    if d.elastic:
        d.u0 = 1e-13 * rng.standard_normal((3,) + sh) * solid
        d.v0 = 1e-2 * rng.standard_normal((3,) + sh) * solid

    def has(flag):
        return np.isin(mc, [q + 1 for q, m in enumerate(d.materials) if getattr(m, flag)])
    d.m0 = d.p0 = d.q0 = None
    if has("fm").any():
        d.m0 = _unit(rng, sh) * has("fm")
    if has("afm").any():
        d.afm0 = np.concatenate([_unit(rng, sh) * has("afm"), _unit(rng, sh) * has("afm")])
    if has("fe").any():
        d.p0 = 0.05 * rng.standard_normal((3,) + sh) * has("fe")
        d.q0 = np.zeros_like(d.p0)
    return d


def _fe(gf, nx, ny, nz, **kw):
    d = gf.decks.preset_ferroelectric(nx=nx, ny=ny, nz=nz, steps=10)
    for k, v in kw.items():
        setattr(d, k, v)
    return d


def _me(gf, nx, ny, nz, sub, film, **kw):
    d = gf.decks.preset_magnetoelastic(nx=nx, ny=ny, nz=nz, sub=sub, film=film, steps=10)
    for k, v in kw.items():
        setattr(d, k, v)
    return d


def _scattered(gf, nx, ny, nz, mats, seed, **kw):
    d = _fe(gf, nx, ny, nz)
    d.materials = mats
    rng = np.random.default_rng(seed)
    d.struct = rng.integers(0, len(mats) + 1, (nx, ny, nz)).astype(np.uint8)
    d.layers = [(nz, 1)]
    for k, v in kw.items():
        setattr(d, k, v)
    return d


def _elastic_decks(gf):
    D = gf.decks
    damped = dataclasses.replace(D.pto(), mass_damping=1e10, stiff_damping=1e-13, er=7.0)
    flexo = dataclasses.replace(D.pto(), f11=6.0, f12=3.5, f44=2.5)
    afm = D.afm_uniaxial(magnetoelastic=True)
    yig = D.yig(1e-2, magnetoelastic=True)
    return {
        # one material, the whole z axis in one tile, tile edges in y, smallest and odd sides
        "fe_uniform": _fe(gf, 9, 21, 13),
        "fe_small": _fe(gf, 1, 5, 5),
        "fe_two_planes": _fe(gf, 2, 7, 6),
        # several tiles along z and y, with remainders
        "fe_wide": _fe(gf, 5, 141, 139),
        # open x and y; periodic z needs ny = nz
        "fe_open_xy": _fe(gf, 10, 17, 11, periodic=(False, False, False)),
        "fe_periodic_z": _fe(gf, 6, 12, 12, periodic=(True, True, True), abc_1D=True),
        # film on a substrate under vacuum, Liao boundary and source
        "me_film": _me(gf, 7, 20, 20, 9, 7),
        "me_open_x": _me(gf, 8, 24, 22, 10, 8, periodic=(False, True, False)),
        # every cell its own material or vacuum, damping, and a work area smaller than the grid
        "scattered": _scattered(gf, 8, 16, 15, [damped, D.ggg(), D.yig(1e-2, magnetoelastic=True)], 3, magnetostatics=False),
        "fe_and_fm": _scattered(gf, 6, 12, 9, [D.pto(), D.yig(1e-2, magnetoelastic=True)], 4),
        "island": _fe(gf, 12, 14, 10, nx_work=7, ny_work=8),
        "afm": _me(gf, 6, 14, 12, 6, 6, materials=[D.ggg(), afm], magnetostatics=False),
        "flexo": _fe(gf, 6, 12, 10, materials=[flexo], flexo=True),
        "no_backaction": _me(gf, 6, 14, 12, 6, 6, elasto_back=False),
        "no_maxwell": _me(gf, 6, 14, 12, 6, 6, em=False, magnetostatics=False, materials=[D.ggg(), yig]),
    }


ELASTIC = ["fe_uniform", "fe_small", "fe_two_planes", "fe_wide", "fe_open_xy", "fe_periodic_z", "me_film", "me_open_x", "scattered",
           "fe_and_fm", "island", "afm", "flexo", "no_backaction", "no_maxwell"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ELASTIC)
def test_column_march_equals_the_general_tile(gf, name, precision):
    d = _moving(_elastic_decks(gf)[name], 17)
    g = dataclasses.replace(d, Tg2c=np.eye(3))
    _same(_run(gf, d, precision), _run(gf, g, precision), TOL[precision])


# Isotropic stiffness, electrostriction and Landau coefficients: the physics
# does not know the crystal frame, so a rotated one (strain, eigenstrain,
# stiffness and polarisation go through the frame rotations, the stress through
# the general tile) gives the run of the unrotated one.  The rotations add a few
# roundings to each term, no cancellation: the tolerances above hold.
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rotated_frame_of_an_isotropic_film_changes_nothing(gf, precision):
    D = gf.decks
    film = dataclasses.replace(D.pto(), c44=0.5 * (2.3e11 - 1.0e11), Q44=0.089 + 0.026, a11=7e7, a12=1.4e8,
                               a111=2.6e8, a112=7.8e8, a123=1.56e9)
    substrate = dataclasses.replace(D.ggg(), c44=0.5 * (2.86e11 - 1.16e11))
    d = _moving(_fe(gf, 6, 15, 14, materials=[substrate, film], layers=[(4, 1), (8, 2), (2, 0)]), 47)
    a = _run(gf, d, precision)
    assert all(np.linalg.norm(a[f]) > 0.0 for f in ("p", "q", "u", "v", "Ex", "Hz"))
    _same(_run(gf, dataclasses.replace(d, Tg2c=D.rotation(30.0, 20.0)), precision), a, TOL[precision])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_engine_of_fewer_materials_leaves_the_others_their_tile(gf, precision):
    """The tile's shared-memory limit belongs to the process, not to the engine
    created last (ny < nz: the general tile)."""
    one = _moving(_fe(gf, 4, 8, 16), 53)
    many = dataclasses.replace(one, materials=one.materials * 12)
    want = _run(gf, one, precision, 1)
    with gf.Engine.from_params(many, device=0, precision=precision) as e:
        with gf.Engine.from_params(one, device=0, precision=precision):
            e.advance(1)
            got = e.download("u")
    assert np.linalg.norm(got - want["u"]) <= TOL[precision] * np.linalg.norm(want["u"])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(1, 5, 5), (9, 21, 13), (12, 33, 32)])
@pytest.mark.parametrize("elastic", [True, False])
def test_tdgl_of_one_material_equals_two_alike(gf, shape, elastic, precision):
    d = _fe(gf, *shape)
    if not elastic:
        d = dataclasses.replace(d, elastic=False, elasto_back=False, elasto_on=False)
    d = _moving(d, 31)
    g = dataclasses.replace(d, materials=[d.materials[0]] * 2)
    g.struct = np.random.default_rng(37).integers(1, 3, shape).astype(np.uint8)
    _same(_run(gf, d, precision), _run(gf, g, precision), TOL[precision])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["fe_z", "fe_x_type1", "fe_y_type6", "open", "periodic_z", "fm_sources", "both", "vacuum_film", "one_cell"])
def test_yee_update_equals_the_general_one(gf, name, precision):
    D = gf.decks
    if name == "fm_sources":
        d = _me(gf, 6, 9, 12, 5, 4)
    elif name == "both":
        d = _scattered(gf, 6, 8, 7, [D.pto(), D.yig(1e-2)], 5, em_fromM=True, em_back_M=True)
    elif name == "vacuum_film":
        d = _fe(gf, 5, 8, 8, layers=[(3, 0), (3, 1), (2, 0)])
    elif name == "one_cell":
        d = _fe(gf, 1, 1, 5, elastic=False, elasto_back=False, elasto_on=False)
    else:
        d = _fe(gf, 6, 11, 9)
        d.jf_lo, d.jf_hi = (1, 0, 2), (4, 8, 5)
        if name == "fe_x_type1":
            d.jf_comp, d.jf_type, d.jf_freq = "x", 1, 1e15
        elif name == "fe_y_type6":
            d.jf_comp, d.jf_type, d.jf_freq, d.jf_sigma = "y", 6, 1e15, 2e-17
        elif name == "open":
            d.periodic = (False, False, False)
        elif name == "periodic_z":
            d = dataclasses.replace(d, ny=9, jf_hi=(4, 8, 8), jf_lo=(0, 0, 7), periodic=(True, True, True), elastic=False,
                                    elasto_back=False, elasto_on=False)
            d.p0 = d.q0 = None
    d = _moving(d, 19)
    # a material with a Drude pole that no cell has: no current flows
    pole = dataclasses.replace(D.ggg(), drude=((1.0, 1e15, 1e-14), (0.0, 0.0, 1.0), (0.0, 0.0, 1.0)))
    g = dataclasses.replace(d, materials=list(d.materials) + [pole])
    _same(_run(gf, d, precision), _run(gf, g, precision), TOL[precision])


# Differences that are zero before any rounding, so every term of them has to be
# formed such that equal ones cancel exactly: 0 and no other value.
@pytest.mark.parametrize("general", [False, True])
def test_curl_of_a_gradient_is_zero(gf, general):
    """E = grad(3 y z): dE_z/dy = dE_y/dz in every cell, so no H grows (FP64)."""
    nx, ny, nz = 4, 24, 24
    d = _fe(gf, nx, ny, nz, elastic=False, elasto_back=False, elasto_on=False, em_fromP=False, em_back_P=False, jf=False,
            materials=[gf.decks.ggg()])
    if general:
        pole = dataclasses.replace(gf.decks.ggg(), drude=((1.0, 1e15, 1e-14), (0.0, 0.0, 1.0), (0.0, 0.0, 1.0)))
        d.materials = d.materials + [pole]
    d.p0 = d.q0 = None
    with gf.Engine.from_params(d, device=0) as e:
        Ey, Ez = e.download("Ey"), e.download("Ez")
        Ey[:] = 3.0 * np.arange(nz + 1)
        Ez[:] = 3.0 * np.arange(ny + 1)[:, None]
        e.upload("Ey", Ey)
        e.upload("Ez", Ez)
        e.advance(1)
        # the ramps break at the ends, one cell further in per stage
        for f in ("Hx", "Hy", "Hz"):
            assert not np.any(e.download(f)[:, 6:-6, 6:-6]), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("layers", [[(12, 1)], [(4, 2), (6, 1), (2, 0)]])
@pytest.mark.parametrize("rotated", [False, True])
def test_laterally_uniform_stress_has_no_lateral_force(gf, layers, rotated, precision):
    D = gf.decks
    d = _fe(gf, 5, 14, 12, em=False, em_fromP=False, em_back_P=False, jf=False, materials=[D.pto(), D.ggg()], layers=layers)
    if rotated:
        d = dataclasses.replace(d, Tg2c=np.eye(3))     # the general tile
    # a polarisation whose shear eigenstrains vanish and normal ones do not
    d.p0 = np.zeros((3, 5, 14, 12))
    d.p0[2] = 0.31 * (d.material_cell() == 1)
    d.q0 = np.zeros_like(d.p0)
    with gf.Engine.from_params(d, device=0, precision=precision) as e:
        e.advance(3)
        f, u = e.download("force_store"), e.download("u")
    assert np.any(f[2])
    assert not np.any(f[:2]) and not np.any(u[:2])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_magnetic_materials_that_no_cell_has(gf, precision):
    """They change nothing (their kernels' boxes are empty)."""
    D = gf.decks
    d = _moving(_fe(gf, 6, 12, 10), 61)
    want = _run(gf, d, precision)
    got = _run(gf, dataclasses.replace(d, materials=d.materials + [D.yig(0.02), D.afm_uniaxial(0.01)]), precision)
    assert not np.any(got.pop("m")) and not np.any(got.pop("m_afm1"))
    _same(got, want, TOL[precision])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(6, 12, 10), (64, 64, 32)])
def test_liao_boundary_waits_for_the_strain_of_the_first_stage(gf, shape, precision):
    """The first step from an uploaded u, whose k = 0 plane the boundary replaces:
    the branches of a stage give what its kernels give one after another."""
    d = _moving(_fe(gf, *shape, abc_1D=False), 67)
    out = []
    for profiled in (False, True):
        with gf.Engine.from_params(d, device=0, precision=precision) as e:
            e.profile_steps(2) if profiled else e.advance(2)
            out.append([e.download(f) for f in ("p", "q", "u", "v", "Ex")])
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_opposite_sublattices_have_no_moment(gf):
    D = gf.decks
    d = D.preset_fm_demag(nx=6, ny=5, nz=4, steps=5)
    d.materials, d.m0, d.Hext_table = [D.afm_uniaxial(0.02)], None, None
    m = _unit(np.random.default_rng(59), (6, 5, 4))
    d.afm0 = np.concatenate([m, -m])
    for kw in ({}, {"mag_1D": True}, {"demag_factor": True, "demag_fac": (0.1, 0.2, 0.7)}):
        for precision in ("fp64", "mixed"):
            with gf.Engine.from_params(dataclasses.replace(d, **kw), device=0, precision=precision) as e:
                assert not np.any(e.download("Hstat")), (kw, precision)


def test_a_moment_along_its_field_stays(gf):
    """m and H along the diagonal of the film plane (FP64): no torque."""
    D = gf.decks
    d = D.preset_fm_demag(nx=4, ny=6, nz=3, steps=5)
    d.magnetostatics, d.Hext_table, d.Hext_stat = False, None, (81234.5, 81234.5, 0.0)
    d.materials = [dataclasses.replace(D.yig(0.02), K1=0.0)]
    d.m0 = np.zeros((3, 4, 6, 3))
    d.m0[:2] = np.sqrt(0.5)
    with gf.Engine.from_params(d, device=0) as e:
        e.advance(3)
        assert np.array_equal(e.download("m"), d.m0)


# sides with the transforms' radices 8, 4, 2, 3, 5 and their products, odd
# ones, a single plane, row or layer, (49, 22, 250) three that cuFFT keeps, and
# one whose x blocks take 8 columns with a remainder
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(8, 6, 4), (5, 3, 2), (64, 16, 8), (30, 18, 10), (24, 45, 9), (128, 5, 3), (4, 4, 1), (1, 16, 6),
                                   (20, 1, 5), (90, 2, 15), (49, 6, 4), (6, 22, 4), (250, 3, 2), (6, 135, 27)])
def test_stage_convolution_matches_the_restatement(gf, shape, precision):
    from oracle import restate_fm
    nx, ny, nz = shape
    d = gf.decks.preset_fm_demag(nx=nx, ny=ny, nz=nz, steps=10)
    d.m0 = _unit(np.random.default_rng(23), shape)
    with gf.Engine.from_params(d, device=0, precision=precision) as e:
        got = [e.download("Hstat")]
        e.advance(1)
        got.append(e.download("Hstat"))
        m1 = e.download("m")
    Nk = restate_fm.demag_spectra(nx, ny, nz, d.dx, d.dy, d.dz)
    for H, m in zip(got, (d.m0, m1)):
        ref = restate_fm.h_static(Nk, d.materials[0].Ms * m, d.dx, d.dy, d.dz)
        # FP64: rounding of the tables' far field (small differences of large
        # terms) between two libms; FP32: log2(n) roundings of 6e-8
        assert np.linalg.norm(H - ref) <= {"fp64": 1e-9, "mixed": 3e-6}[precision] * np.linalg.norm(ref)


def test_stage_convolution_covers_only_magnetic_cells(gf):
    """A film over a non-magnetic substrate: the source is Ms m in the film."""
    from oracle import restate_fm
    d = gf.decks.preset_fm_demag(nx=12, ny=10, nz=8, steps=10)
    d.materials = [gf.decks.ggg(), gf.decks.yig(1e-2)]
    d.layers = [(3, 1), (4, 2), (1, 0)]
    mag = d.material_cell() == 2
    d.m0 = _unit(np.random.default_rng(29), (12, 10, 8)) * mag
    Nk = restate_fm.demag_spectra(12, 10, 8, d.dx, d.dy, d.dz)
    ref = restate_fm.h_static(Nk, d.materials[1].Ms * d.m0, d.dx, d.dy, d.dz)
    for precision, tol in (("fp64", 1e-9), ("mixed", 3e-6)):
        with gf.Engine.from_params(d, device=0, precision=precision) as e:
            H = e.download("Hstat")
        assert np.linalg.norm(H - ref) <= tol * np.linalg.norm(ref)


def test_adjoint_of_a_layered_film_matches_finite_differences(gf, tmp_path):
    """The transposed elastic march with several materials and vacuum."""
    from test_gpu_adjoint import MU0, _grads
    steps, nw = 60, 4
    D = gf.decks
    d = D.preset_fm_demag(nx=6, ny=12, nz=11, steps=steps)
    d.Hext_table = None
    d.Hext_stat = (0.0, 0.0, 1.0 / MU0)
    film = D.yig(0.02, magnetoelastic=True)
    film.lam100 *= 1000.0
    film.lam111 *= 1000.0
    d.materials = [film, dataclasses.replace(D.ggg(), c44=1.3e11, stiff_damping=2e-13, mass_damping=1e9)]
    d.layers = [(4, 2), (5, 1), (2, 0)]
    mc = d.material_cell()
    d.m0 = D.tilt_m0((6, 12, 11), 31, mc == 1, 10.0)
    d.elastic, d.elasto_back, d.elasto_on = True, True, True
    D.write_deck(d, str(tmp_path))
    alpha0 = 0.02 * (1.0 + 0.1 * np.random.default_rng(5).random(d.n)) * (mc.ravel() == 1)
    tt = (np.arange(nw) + 0.5) / nw
    wave0 = (1e-2 / MU0) * np.sin(2 * np.pi * tt)
    gw, ga, (fd_w, v, fd_a) = _grads(gf, tmp_path, d, steps, nw, wave0, alpha0, True)
    assert np.max(np.abs(gw - fd_w)) <= 1e-4 * np.max(np.abs(fd_w))
    assert abs(float(ga @ v) - fd_a) <= 1e-4 * abs(fd_a)
    gw32, ga32, _ = _grads(gf, tmp_path, d, steps, nw, wave0, alpha0, False, precision="mixed")
    assert np.max(np.abs(gw32 - gw)) <= 1e-3 * np.max(np.abs(gw))
    assert np.max(np.abs(ga32 - ga)) <= 1e-3 * np.max(np.abs(ga))


def test_stage_convolution_of_the_widest_blocks(gf):
    """x blocks of 16 columns with a remainder (FP32) against cuFFT, which the
    FP64 form keeps for planes of this size."""
    shape = (50, 216, 32)
    d = gf.decks.preset_fm_demag(nx=shape[0], ny=shape[1], nz=shape[2], steps=10)
    d.m0 = _unit(np.random.default_rng(43), shape)
    H = {}
    for precision in ("fp64", "mixed"):
        with gf.Engine.from_params(d, device=0, precision=precision) as e:
            H[precision] = e.download("Hstat")
    assert np.linalg.norm(H["mixed"] - H["fp64"]) <= 3e-6 * np.linalg.norm(H["fp64"])


# x of four passes, which the engine leaves to cuFFT and the adjoint takes by
# its own transforms
@pytest.mark.parametrize("shape", [(81, 6, 6), (250, 8, 5)])
def test_adjoint_transforms_match_the_engine(gf, shape):
    D = gf.decks
    d = D.preset_fm_demag(nx=shape[0], ny=shape[1], nz=shape[2], steps=6)
    d.Hext_table = None
    d.Hext_stat = (0.0, 0.0, 1.0 / D.MU0)
    d.m0 = D.tilt_m0(shape, 41, d.material_cell(), 20.0)
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-6)):
        with gf.Engine.from_params(d, device=0, precision=precision) as e:
            with gf.Adjoint(e, n_wave=4, checkpoint_every=3) as a:
                a.forward(6)
                m = a.final_m()
            e.advance(6)
            assert np.max(np.abs(m - e.download("m"))) <= tol
