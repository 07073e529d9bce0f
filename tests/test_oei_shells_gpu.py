"""GPU tests of the one-electron integrals' shell-pair kernel: the numbers of charges
where its block size and chunks change, s to f shells, against the oracle; and bases
whose components are not in QUICK's order (the function-pair kernel) against it."""
import copy
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from quick_b200.basis import build_basis  # noqa: E402
from quick_b200.molecules import water_cluster  # noqa: E402


def _charges(m):
    rng = np.random.default_rng(m + 1)
    return (rng.normal(size=(m, 3)) * 12.0, rng.normal(size=m)) if m else None


@pytest.mark.parametrize("bas,nw", [("STO-3G", 1), ("6-31G**", 3), ("CC-PVTZ", 2)])
@pytest.mark.parametrize("m", [0, 1, 33, 503, 506, 509, 515, 2100])
def test_oei_matches_oracle_at_the_lines(bas, nw, m):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.scf import oei
    b = build_basis(water_cluster(nw, 6.0, seed=nw), bas)
    ext = _charges(m)
    for got, want in zip(oei(b, ext), O.oei(b, ext)):
        # sums of at most m + 9 charges x 81 primitive pairs in another order
        assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("bas", ["6-31G*", "CC-PVTZ"])
def test_oei_takes_components_in_any_order(bas):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.scf import oei
    b = build_basis(water_cluster(2, 6.0, seed=5), bas)
    ext = _charges(40)
    p = np.random.default_rng(3).permutation(b.nbasis)
    q = copy.copy(b)
    for f in ("ncontract", "ncenter"):
        setattr(q, f, getattr(b, f)[p])
    for f in ("itype", "aexp", "dcoeff"):
        setattr(q, f, np.asfortranarray(getattr(b, f)[:, p]))
    for got, want in zip(oei(q, ext), oei(b, ext)):
        assert np.abs(got - want[np.ix_(p, p)]).max() <= 1e-12 * max(1.0, np.abs(want).max())


def test_oei_charge_beyond_the_range_adds_nothing():
    """A charge so far away that its squared distance overflows."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200.scf import oei
    b = build_basis(water_cluster(2, 6.0, seed=2), "6-31G*")
    far = (np.array([[1e155, 0.0, 0.0], [0.0, -3e160, 1e158]]), np.array([1.0, -2.0]))
    for got, want in zip(oei(b, far), oei(b, None)):
        assert np.array_equal(got, want)


_GIVE_BACK = """
import torch
from quick_b200.basis import build_basis
from quick_b200.get2e import Get2e
from quick_b200.molecules import water_cluster
from quick_b200.scf import oei
small, large = (build_basis(water_cluster(n, 24.0, seed=1), "6-31G*") for n in (1, 80))
free = lambda: torch.cuda.mem_get_info(0)[0]
eng = Get2e(small)
oei(small, None)
before = free()
oei(large, None)     # 3 n^2 doubles and more: 64 MB beside the small call's 32
kept = before - free()
eng.close()
assert kept >= 60 << 20, kept
assert before - free() <= 32 << 20, (kept, before - free())
"""


def test_oei_memory_goes_back_with_the_last_context():
    """In a process of its own: any context that lives keeps the memory."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", _GIVE_BACK], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
