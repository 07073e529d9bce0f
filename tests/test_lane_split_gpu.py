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
