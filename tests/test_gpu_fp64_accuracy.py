"""FP64 mode: the force of single pairs against extended precision.

Isolated pairs along x at distances whose squares are exact in FP64, so that
what is measured is the evaluation of the force law alone.  With u = 2^-53 (a
rounding), the bounds follow from the operations of pair64_force:
* G = E + 2 a r / sqrt(pi) e^{-a^2 r^2} by table: the fit (1e-16), the rounding
  of the leading coefficient and of the last sum (u / 2 each, G <= 1) and that
  of 1/r (r |dG/dr| <= 0.93: u): under 3.3e-16;
* the steps after it: at most 8 roundings of the pair's Coulomb term;
* LJ: 1/r enters as its 14th (8th) power, 30 (18) roundings in all;
* the stored force: half of 2^-32, the other lanes add zeros.
The A&S form as written (no table) takes E as five products and sums, an exp
(within one ulp) and a divide: 8 u in place of the table's 3.3e-16."""
import numpy as np
import pytest

from md_gpu_gb300 import MDSystem
from md_gpu_gb300.system import TERM_PAIR

pytestmark = pytest.mark.gpu

LD = np.longdouble
U = 2.0 ** -53
QFAC = np.float32(1389.35427611722)


def _pairs(rc, rmin, seed):
    """Atoms 2 k and 2 k + 1, r_k apart along x, pairs more than 2 rc apart."""
    rng = np.random.default_rng(seed)
    a, m = 40.0, 12
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    c = (g - (m - 1) / 2.0) * a
    r = np.floor(rng.uniform(rmin, rc, len(c)) * 2.0 ** 22) * 2.0 ** -22   # 26 bits: r^2 is exact
    pos = np.empty((2 * len(c), 3))
    pos[0::2] = c
    pos[1::2] = c
    pos[1::2, 0] += r
    return np.float32(a * m), pos, r


def _system(rc, pos, box, q, lj1, lj2, lkspace, alpha, reacf):
    n = len(pos)
    return MDSystem.from_arrays(
        box=np.full(3, box, np.float32), itype=np.zeros(n, np.int32), charge=np.tile(np.float32([q, -q]), n // 2),
        pos=pos.astype(np.float32), vel=np.zeros((n, 3), np.float32), type_mass=np.float32([2e5]),
        lj1=np.float32([[lj1]]), lj2=np.float32([[lj2]]), lkspace=lkspace, rcutsq=float(np.float32(rc * rc)),
        reacf=reacf, alfa=alpha, skin=1.0, nmaxlist=64, dt=1.0, integrator=1)


def _G(alpha, r):
    """The A&S form, constants as the library holds them, in the type of r."""
    T = type(r[0])
    A = [T(np.float32(a)) for a in (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)]
    al, p = T(np.float32(alpha)), T(np.float32(0.3275911))
    spi = T(2.0 / np.sqrt(np.pi) * float(np.float32(alpha)))
    xa = al * r
    t = 1 / (1 + p * xa)
    ex = np.exp(-xa * xa)
    poly = ((((A[4] * t + A[3]) * t + A[2]) * t + A[1]) * t + A[0]) * t
    return poly * ex + spi * r * ex


def _forces(sim, pos, energy):
    sim.set_precision(64)
    sim.set_positions(pos)
    sim.compute_forces(TERM_PAIR, energy=energy)
    f = sim.forces()[:, :3]
    assert np.abs(f[:, 1:]).max() == 0.0 and np.array_equal(f[0::2], -f[1::2])
    return f[1::2, 0]


# a rc from 0.5 to 3.5 (16 to 128 pieces), the real-space Ewald form, and one without a table
@pytest.mark.parametrize("lkspace,alpha,rc", [(1, 0.05, 10.0), (1, 0.1, 12.0), (1, 0.2, 12.0), (1, 0.24, 10.0),
                                              (2, 0.309, 10.0), (1, 0.35, 10.0), (1, 1.2, 10.0)])
@pytest.mark.parametrize("energy", [False, True])
def test_coulomb_of_single_pairs(lkspace, alpha, rc, energy):
    q = 2048.0
    box, pos, r = _pairs(rc, 2.5, 7)
    with _system(rc, pos, box, q, 0.0, 0.0, lkspace, alpha, 0.0) as sim:
        f = _forces(sim, pos, energy)
    r = r.astype(LD)
    w = LD(0)
    if lkspace == 1:
        rcl = LD(np.sqrt(np.float64(np.float32(rc * rc))))
        w = _G(alpha, rcl.reshape(1))[0] / rcl
    qq = LD(QFAC) * LD(q) * LD(q)
    G = _G(alpha, r)
    fc = -qq * (G / r - w) / (r * r) * r      # attraction: towards the partner
    err = np.abs(f.astype(LD) - fc) * r / qq * r
    bound = (3.3e-16 if alpha <= 0.35 else 8 * U) + 8 * U * np.abs(G - w * r) + 2.0 ** -33 * (r * r / qq)
    assert (err <= bound).all(), f"{float((err / bound).max()):.2f} of the bound, {float(err.max()):.1e}"


@pytest.mark.parametrize("energy", [False, True])
def test_lj_and_reaction_field_of_single_pairs(energy):
    rc, reacf = 10.0, float(np.float32(0.9e-3))
    for q, lj1, lj2 in ((0.0, 4.0e8, 1.0e5), (2048.0, 0.0, 0.0)):
        box, pos, r = _pairs(rc, 2.5 if q else 1.0, 8)   # forces below 2^31
        with _system(rc, pos, box, q, lj1, lj2, 0, 0.0, reacf) as sim:
            f = _forces(sim, pos, energy)
        x = r.astype(LD)
        qq = LD(QFAC) * LD(q) * LD(q)
        a, b = LD(np.float32(lj1)) / x ** 13, LD(np.float32(lj2)) / x ** 7
        c1, c2 = qq / (x * x), qq * LD(reacf) * x
        ref = a - b - (c1 - c2)
        bound = U * (30 * a + 18 * b + 9 * (c1 + c2)) + 2.0 ** -33
        err = np.abs(f.astype(LD) - ref)
        assert (err <= bound).all(), f"{float((err / bound).max()):.2f} of the bound"


@pytest.mark.parametrize("lkspace,alpha", [(1, 0.2), (1, 1.2), (2, 0.309), (0, 0.0)])
@pytest.mark.parametrize("batch", [False, True])
def test_forces_do_not_depend_on_energies(lkspace, alpha, batch):
    """Bit for bit, so that a trajectory does not depend on which steps
    compute energies."""
    from md_gpu_gb300 import synth
    reps = []
    for k, n in enumerate((998, 1728)):
        a = synth.to_arrays(synth.nacl_replica(n, seed=3 + k, rc=10.0))
        a.update(lkspace=lkspace, alfa=alpha, reacf=9e-4 if lkspace == 0 else 0.0)
        reps.append(a)
    out = []
    for every in (0, 1):
        sim = MDSystem.from_batch(reps) if batch else MDSystem.from_arrays(**reps[0])
        with sim:
            sim.set_precision(64)
            sim.compute_forces(energy=bool(every))
            f = sim.forces()[:, :3]
            sim.step(12, every)
            out.append((f, sim.positions(), sim.velocities()))
    for p, q in zip(*out):
        assert np.array_equal(p, q)
