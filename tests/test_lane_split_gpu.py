"""GPU tests of lanes that share a quartet: the number of lanes follows the number of
s, p, d and f shells (10, 64 and 256 are the lines of the rule; five to a water in
STO-3G, ten in 6-31G*, 22 in cc-pVTZ), the contraction lengths (9 x 9 primitive pairs in
STO-3G, 36 x 36 in 6-31G*, 64 x 64 in cc-pVTZ) and the class, so the Fock matrix is
compared with the oracle on both sides of each line, in FP64 and in the mixed form, and
bit for bit with the batched and the merged launches and with builds queued one behind
another."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from quick_b200.basis import build_basis  # noqa: E402
from quick_b200.molecules import water_cluster  # noqa: E402


def _tolerance(n, largest, bound=0.0):
    """FP64: an element collects at most n^2 Coulomb and n^2 exchange terms, twice (A + A^T), each rounded to 2^-44
    (2^-44/sqrt(12) rms): six standard deviations of their sum, twice that for the diagonal, where the two halves are
    the same numbers; and FP64 sums of |G| (1e-13 relative).  Mixed: quartets below the bound at FP32's 6e-8."""
    return 12.0 * (4.0 * n * n / 12.0) ** 0.5 * 2.0 ** -44 + 1e-13 * largest + bound * 6e-8 * n


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
    tol = _tolerance(b.nbasis, np.abs(want).max(), bound)
    assert np.abs(got - want).max() <= tol


@pytest.mark.parametrize("nw", [51, 52])
def test_shared_quartets_around_256_shells(nw):
    """Waters far apart: 255 and 260 shells, few pairs."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2e
    b = build_basis(water_cluster(nw, 60.0, seed=nw), "STO-3G")
    rng = np.random.default_rng(nw)
    X = rng.normal(size=(b.nbasis, b.nbasis)) * 0.2
    D = X @ X.T / b.nbasis ** 0.5
    orc = O.Oracle(b)
    Y, cp = orc.schwarz()
    want, _ = orc.get2e(D, orc.density_cutoff(D), Y, cp, 1e-9, 1e-10)
    eng = Get2e(b, integral_cutoff=1e-9, prim_limit=1e-10, schwarz=(Y, cp))
    got = eng.fock2e(torch.tensor(D, device="cuda")).cpu().numpy()
    eng.close()
    assert np.abs(got - want).max() <= _tolerance(b.nbasis, np.abs(want).max())


# five, 20, 65 and 260 shells, and the classes up to d and f
_TIERS = [("STO-3G", 1, 6.0), ("STO-3G", 4, 6.0), ("STO-3G", 13, 9.0), ("STO-3G", 52, 60.0), ("6-31G**", 2, 6.0),
          ("CC-PVTZ", 1, 6.0)]


def _engines(seed, tiers=_TIERS):
    from quick_b200.get2e import Get2e
    out = []
    for bas, nw, box in tiers:
        b = build_basis(water_cluster(nw, box, seed=nw), bas)
        X = np.random.default_rng(seed + nw).normal(size=(b.nbasis, b.nbasis)) * 0.2
        out.append((Get2e(b, integral_cutoff=1e-9, prim_limit=1e-10),
                    torch.tensor(X @ X.T / b.nbasis ** 0.5, device="cuda")))
    return out


@pytest.mark.parametrize("bound", [0.0, 1e-5])
def test_shared_quartets_batched_and_merged(bound):
    """Molecules whose lanes are shared differently, in one batch and by the merged s/p kernel: the same bits."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2eBatch
    engines = _engines(1)
    for e, _ in engines:
        e.set_precision(bound)
    want = [e.fock2e(D) for e, D in engines]
    bt = Get2eBatch()
    for got, ref in zip(bt.fock2e([e for e, _ in engines], [D for _, D in engines]), want):
        assert torch.equal(got, ref)
    bt.close()
    for (e, D), ref in zip(engines, want):
        e.set_merge_sp(True)
        assert torch.equal(e.fock2e(D), ref)
        e.close()


@pytest.mark.parametrize("streams", [0, 4])
def test_queued_builds_equal_waited_ones(streams):
    """A class kernel starts before the one it follows in the stream has ended, the next build's clearing of the
    accumulator and the finish of this one do not: builds of changing densities queued on one stream, single and
    batched by turns, give the bits of builds that were waited for."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.get2e import Get2eBatch
    engines = _engines(2, [t for t in _TIERS if t[1] < 13])
    for e, _ in engines:
        e.set_streams(streams)
    Ds = [[D * s for _, D in engines] for s in (1.0, -0.5, 1e-3, 2.0)]
    want = []
    for row in Ds:
        want.append([e.fock2e(D) for (e, _), D in zip(engines, row)])
        torch.cuda.synchronize()
    bt = Get2eBatch()
    got = []
    for row in Ds:
        got.append([e.fock2e(D) for (e, _), D in zip(engines, row)])
        got.append(bt.fock2e([e for e, _ in engines], row))
    torch.cuda.synchronize()
    for k, row in enumerate(got):
        for g, w in zip(row, want[k // 2]):
            assert torch.equal(g, w)
    bt.close()
    for e, _ in engines:
        e.close()


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
