"""The tau integral's exponentials and its walk over the spin-conserving
elements."""
import numpy
import pytest

from kelvin_gb300 import quadrature, systems
from kelvin_gb300.cc_utils import DeviceSolver
from kelvin_gb300.quadrature import ft_quad
from oracle import ft_ccsd as oft
from oracle import ft_utils
from oracle import quadrature as oq

pytestmark = pytest.mark.gpu


def test_exponential_range(ctx):
    """One weight per element: T[1] = G[1,0] exp(-delta d) tbar[0].  Arguments
    over the table's range, at its edges (|x| = 700, where the library function
    takes over), large ones that overflow or vanish, zero, and n ln2/128 (the
    largest remainders).  Tolerance: one unit in the last place for each of the
    two exponentials and half for each of the two products."""
    x = numpy.concatenate((numpy.linspace(-720.0, 720.0, 4001),
                           numpy.arange(-64, 65) * numpy.log(2.0) / 128.0,
                           [700.0, -700.0, numpy.nextafter(700.0, 0.0), 0.0, -0.0, 800.0, -800.0]))
    n = x.shape[0]
    ti, g, G = quadrature.ft_quad(2, 1.0, "lin")
    t = numpy.zeros((2, 1, n))
    t[0] = 1.0
    out = quadrature.int_tbar1(2, t, ti, -x.reshape(1, n), G)
    with numpy.errstate(over="ignore"):
        ref = 0.5 * numpy.exp(x)
    fin = numpy.isfinite(ref)
    assert numpy.array_equal(numpy.isfinite(out[1, 0]), fin)
    assert (abs(out[1, 0][fin] - ref[fin]) <= 3.0 * 2.0 ** -52 * ref[fin] + 5e-324).all()


@pytest.mark.parametrize("quad,ng,tol", [("lin", 2, 1e-13), ("lin", 3, 1e-13), ("lin", 5, 1e-13),
                                         ("lin", 8, 1e-13), ("lin", 17, 1e-13), ("mid", 9, 1e-13),
                                         ("ln", 6, 1e-13), ("gl", 7, 1e-12), ("gl", 8, 1e-12)])
def test_int_tbar_rectangular(ctx, quad, ng, tol):
    """Rows with shared coefficients (and the ones before them), the mapped
    grid, dense grids with and without a middle node; nv != no."""
    rng = numpy.random.default_rng(ng)
    nv, no = 5, 3
    ti, g, G = ft_quad(ng, 2.0, quad)
    D = rng.standard_normal((nv, nv, no, no)) * 2.0
    t = rng.standard_normal((ng, nv, nv, no, no))
    full = quad == "gl"
    ref = oq.int_tbar2(ng, t, ti, D, G, full=full)
    out = quadrature.int_tbar2(ng, t, ti, D, G, full=full)
    assert abs(out - ref).max() <= tol * max(1.0, abs(ref).max())


# alpha halves of one, several and partial units of 32 elements per quadrant,
# and of several assembly tiles (h > 64 would need 130 spin orbitals: the tile
# arithmetic is the same for every quadrant)
@pytest.mark.parametrize("pw,quad", [(1, "lin"), (3, "gl"), (6, "lin"), (11, "gl")])
def test_spin_blocked_step_vs_oracle(ctx, pw, quad):
    s = systems.ueg_recipe(1.0 if pw == 1 else 2, 2.0, pw, 0.5)
    beta, ng = 1.0 / s.T, 5
    en = s.g_energies_tot()
    ti, g, G = ft_quad(ng, beta, quad)
    sv = DeviceSolver.from_system(ctx, en, s.g_fock_tot(), s.g_aint_tot(), beta, s.mu, ti, g, G)
    try:
        sv.full = quad == "gl"
        assert sv.spin_blocks() == pw
        sv.guess(1)
        x1, x2 = sv.amplitudes()
        E, _ = sv.step(0.3)
        T1, T2 = sv.amplitudes()
    finally:
        sv.close()
    F, I = oft.ft_integrals(s.g_fock_tot(), s.g_aint_tot(), en, beta, s.mu)
    D1, D2 = ft_utils.D1(en, en), ft_utils.D2(en, en)
    r1, r2 = oft.ccsd_stanton(F, I, x1, x2, D1, D2, ti, ng, G, full=quad == "gl")
    assert abs(T1 - (0.3 * x1 + 0.7 * r1)).max() <= 1e-12 * max(1.0, abs(r1).max())
    assert abs(T2 - (0.3 * x2 + 0.7 * r2)).max() <= 1e-12 * max(1.0, abs(r2).max())
    assert abs(E - oft.ft_cc_energy(T1, T2, F.ov, I.oovv, g, beta)) <= 1e-12


# The symmetric T1 T1 half (rows a < b, a = b, a > b in one tile, a tile that
# spans three values of a), rectangular extents, one tile and several waves of
# them, T1's share on more and fewer blocks than elements; both Q terms.
@pytest.mark.parametrize("nv,no,ng", [(1, 1, 1), (1, 40, 3), (11, 2, 4), (13, 7, 20), (34, 33, 5),
                                      (60, 21, 2)])
@pytest.mark.parametrize("qterm", [True, False])
def test_energy_rectangular(ctx, nv, no, ng, qterm):
    from kelvin_gb300 import ft_cc_energy
    rng = numpy.random.default_rng(nv + no)
    T1 = rng.standard_normal((ng, nv, no))
    T2 = rng.standard_normal((ng, nv, nv, no, no))
    f, eri = rng.standard_normal((no, nv)), rng.standard_normal((no, no, nv, nv))
    g = rng.random(ng)
    E = ft_cc_energy.ft_cc_energy(T1, T2, f, eri, g, 2.0, qterm, ctx=ctx)
    ref = oft.ft_cc_energy(T1, T2, f, eri, g, 2.0, qterm)
    # both sums lie within a roundoff per term of the sum of magnitudes
    mag = oft.ft_cc_energy(abs(T1), abs(T2), abs(f), abs(eri), g, 2.0, qterm)
    assert abs(E - ref) <= 4.0 * 2.0 ** -53 * (ng + 4) * mag + 1e-15 * mag


@pytest.mark.parametrize("shift", [0.0, 8e-16, -8e-16])
def test_dense_integral_on_a_grid_off_by_last_places(ctx, shift):
    """Nodes that are symmetric about the centre only to 8e-16 of the range, and
    a large beta |d|: exp((t_x - t_y) d) keeps their actual distances.  One
    sweep from zero amplitudes with a Fock matrix alone integrates a constant;
    its values at two nodes are compared by their ratio.  Tolerance at a node:
    half a unit of the arguments (at most beta |d| / 2) of two exponentials, four
    units for these and the products, 1e-14 for the compensated FP32 sum."""
    E, ng = 80.0, 8
    ti, g, G = ft_quad(ng, 1.0, "gl")
    ti = ti.copy()
    ti[1] += shift
    fock = numpy.array([[0.0, 0.01, 0.0, 0.0], [0.01, E, 0.0, 0.0],
                        [0.0, 0.0, 0.0, 0.01], [0.0, 0.0, 0.01, E]])
    en = numpy.array([0.0, E, 0.0, E])
    sv = DeviceSolver.from_system(ctx, en, fock, numpy.zeros((4,) * 4), 1.0, -60.0, ti, g, G)
    try:
        sv.full = True
        sv.guess(0)
        sv.step(0.0)
        T1, _ = sv.amplitudes()
    finally:
        sv.close()
    t = ti.astype(numpy.longdouble)
    for a, i, d in ((0, 1, -E), (1, 0, E)):
        w = G * numpy.exp((t[None, :] - t[:, None]) * d)
        ref, size = w.sum(1), abs(w).sum(1)
        tol = (1e-14 + (E + 8) * 2.0 ** -53) * size / abs(ref)
        for y in range(ng):
            r = numpy.longdouble(T1[y, a, i]) / T1[3, a, i] * ref[3] / ref[y]
            assert abs(r - 1) <= tol[y] + tol[3]


def test_exponentials_are_as_accurate_as_the_library_function(ctx):
    """Step factors are powers of one exponential, so its last bit counts.  The
    same single weight as above, here against 64 bits: a nearly correctly
    rounded value, half a unit in the last place and a fiftieth."""
    rng = numpy.random.default_rng(8)
    x = numpy.concatenate((rng.uniform(-3.0, 3.0, 40000), rng.uniform(-600.0, 600.0, 20000),
                           rng.uniform(-0.02, 0.02, 5000)))
    n = x.shape[0]
    ti, g, G = quadrature.ft_quad(2, 1.0, "lin")
    t = numpy.zeros((2, 1, n))
    t[0] = 1.0
    out = quadrature.int_tbar1(2, t, ti, -x.reshape(1, n), G)[1, 0]
    ref = numpy.exp(x.astype(numpy.longdouble)) / 2
    ulp = numpy.spacing(ref.astype(float))
    assert (abs(out - ref) <= 0.52 * ulp).all()
