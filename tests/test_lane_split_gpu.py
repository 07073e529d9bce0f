"""GPU tests of lanes that share a quartet: the number of lanes follows the number of
shells (10, 64 and 256 are the lines of the rule), the contraction lengths (9 x 9
primitive pairs in STO-3G, 36 x 36 in 6-31G*, 64 x 64 in cc-pVTZ) and the class, so the
Fock matrix is compared with the oracle on both sides of each line, in FP64 and in the
mixed form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from quick_b200.basis import build_basis  # noqa: E402
from quick_b200.molecules import water_cluster  # noqa: E402


@pytest.mark.parametrize("bas,nw", [("STO-3G", 1), ("STO-3G", 2), ("STO-3G", 3), ("STO-3G", 13), ("6-31G*", 1),
                                    ("6-31G*", 6), ("6-31G*", 7), ("CC-PVTZ", 1)])
@pytest.mark.parametrize("bound", [0.0, 1e-5])
def test_shared_quartets_match_oracle(bas, nw, bound):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2e
    b = build_basis(water_cluster(nw, max(6.0, 3.2 * nw ** (1 / 3)), seed=nw), bas)
    rng = np.random.default_rng(nw)
    X = rng.normal(size=(b.nbasis, b.nbasis)) * 0.2
    D = X @ X.T / b.nbasis ** 0.5
    orc = O.Oracle(b)
    Y, cp = orc.schwarz()
    want, _ = orc.get2e(D, orc.density_cutoff(D), Y, cp, 1e-11, 1e-12)
    eng = Get2e(b, integral_cutoff=1e-11, prim_limit=1e-12, schwarz=(Y, cp))
    eng.set_precision(bound)
    got = eng.fock2e(torch.tensor(D, device="cuda")).cpu().numpy()
    eng.close()
    # FP64: an element sums at most n^2 Coulomb and n^2 exchange terms, twice (A + A^T),
    # each rounded to 2^-45, and FP64 sums of |G| (1e-13 relative); mixed: quartets below
    # the bound at FP32's 6e-8
    tol = 4 * b.nbasis ** 2 * 2.0 ** -45 + 1e-13 * np.abs(want).max()
    if bound:
        tol += bound * 6e-8 * b.nbasis
    assert np.abs(got - want).max() <= tol


def test_lane_split_does_not_depend_on_the_cutoff():
    """Lists built at a tighter cutoff are cut alike: the same Fock matrix bit for bit."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2e
    b = build_basis(water_cluster(3, 6.0, seed=2), "6-31G*")
    rng = np.random.default_rng(4)
    X = rng.normal(size=(b.nbasis, b.nbasis)) * 0.2
    D = torch.tensor(X @ X.T / b.nbasis ** 0.5, device="cuda")
    fresh = Get2e(b, integral_cutoff=1e-8, prim_limit=1e-9)
    want = fresh.fock2e(D)
    eng = Get2e(b, integral_cutoff=1e-12, prim_limit=1e-9)
    eng.prepare()
    eng.set_cutoffs(1e-8, 1e-9)
    assert torch.equal(eng.fock2e(D), want)
    fresh.close()
    eng.close()


def _rounded_elements(b):
    """How many rounded terms each element of the accumulator collects, every shell quartet of the basis taken: the
    two Coulomb blocks and each element of the exchange blocks once."""
    shells = []
    for s in range(b.nshell):
        for L in range(int(b.qstart[s]), int(b.qfinal[s]) + 1):
            f0 = int(b.ksumtype[s]) - 1 + int(b.qsbasis[s, L])
            shells.append(slice(f0, f0 + (L + 1) * (L + 2) // 2))
    N = np.zeros((b.nbasis, b.nbasis))
    pairs = [(x, y) for i, x in enumerate(shells) for y in shells[:i + 1]]
    for i, (x, y) in enumerate(pairs):
        for z, w in pairs[:i + 1]:
            N[x, y] += 1
            N[z, w] += 1
            for u, v in {(x.start, z.start): (x, z), (y.start, z.start): (y, z), (x.start, w.start): (x, w),
                         (y.start, w.start): (y, w)}.values():
                N[u, v] += 1
    return N


@pytest.mark.parametrize("bas,nw,seeds", [("STO-3G", 1, 24), ("STO-3G", 2, 12)])
def test_shared_quartets_round_no_more_often(bas, nw, seeds):
    """The accumulator's roundings (2^-44, uniform) of a build in which nothing is screened, against the oracle's 64-bit
    sums: no larger than independent roundings of each quartet's distinct elements."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2e
    err2 = bound2 = 0.0
    for seed in range(seeds):
        b = build_basis(water_cluster(nw, 6.0, seed=50 + seed), bas)
        rng = np.random.default_rng(seed)
        X = rng.normal(size=(b.nbasis, b.nbasis)) * 0.3
        D = X @ X.T
        orc = O.Oracle(b)
        Y, cp = orc.schwarz()
        want, _ = orc.get2e(D, orc.density_cutoff(D), Y, cp, 1e-18, 1e-20)
        eng = Get2e(b, integral_cutoff=1e-18, prim_limit=1e-20, schwarz=(Y, cp))
        got = eng.fock2e(torch.tensor(D, device="cuda")).cpu().numpy()
        eng.close()
        N = _rounded_elements(b)
        var = N + N.T + 2.0 * np.diag(np.diag(N))   # G = A + A^T: a diagonal element is doubled
        err2 += np.sum((got - want) ** 2)
        bound2 += var.sum() * 2.0 ** -88 / 12.0
    assert err2 <= bound2, (err2 ** 0.5, bound2 ** 0.5)
